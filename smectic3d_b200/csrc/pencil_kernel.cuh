// Pencil pass: the x transform, fused with the spectral time update.
//
// A CTA owns TK consecutive in-plane positions f (128 bytes of every x-plane
// row) and all N values of x.  Lanes run along f, so every global access of a
// warp is whole 128-byte row segments straight between HBM and registers: no
// staging of the tile in shared memory, which only carries the one exchange
// between the two register passes of each transform (line_fft.cuh).  A thread
// holds wavenumbers k and N - k together, so the cosine transforms pair them in
// registers.  The forward x transform completes the 3-D spectrum of the
// nonlinear term; the CNAB2 update runs in registers; the inverse x transform
// of the new psi spectrum starts from the same registers.
//
// The spectral state is W^n = C1 psihat^n - dt/2 Nhat^{n-1}, stored like the
// partials, [kx][f].  The reference update
//   psihat^{n+1} = (C1 psihat^n + dt/2 (3 Nhat^n - Nhat^{n-1})) / C2
// (periodicFFT/pf3d.cpp:476-478, cosFFT/mesabi/cosNoAdvMorph.cpp:524-525)
// becomes psihat^{n+1} = (W^n + 3 dt/2 Nhat^n) / C2 and
// W^{n+1} = C1 psihat^{n+1} - dt/2 Nhat^n: one state read and one state write.
#pragma once
#include <type_traits>

#include "line_fft.cuh"
#include "sh_common.cuh"

namespace shb {

enum PencilMode : int {
  kPencilStep = 0,
  kPencilInit = 1,
  kPencilEnergy = 2,
  kPencilStepAdv = 3,  // step that also emits extra partials: i q_x psihat and opSH psihat (periodic, advection),
                       // -q_x^2 psihat (Neumann, substrate penalty)
  kPencilInitAdv = 4,
  kPencilStokes = 5,   // Stokes velocity from the stress (periodicFFT/pf3d.cpp:433-447)
  kPencilXMul = 6,     // partial P -> partial of its spectrum times an x-line multiplier (XMul)
  kPencilSpec = 7,     // partial P -> psihat
  kPencilAdjInit = 8,  // adjoint: partial of lambda^T -> lambdahat^T, mu partial
  kPencilAdj = 9,      // adjoint step: lambdahat^n = A lambdahat^{n+1} + ghat^n, mu partial, parameter gradients
  kPencilAdjOut = 10,  // adjoint: lambdahat -> its x-inverse partial (for lambda^0 in real space)
  kPencilStepU64 = 11, // the step of FP32 fields with the CNAB2 multipliers and update in FP64
  kPencilStepGen = 12, // the step with what kPencilStep and kPencilStepEuler leave out: the energy, psihat out
  kPencilStepU64Gen = 13,  // the same for kPencilStepU64
  kPencilStepAdvGen = 14,  // the same for kPencilStepAdv
  kPencilStepSpec = 15,    // kPencilStep that keeps psihat^{n+1} in spec_out (the adjoint's recompute)
  kPencilStepEuler = 16,   // kPencilStep with IMEX Euler
};
// multiplier of kPencilXMul
enum XMulKind : int {
  kXIqx = 0,     // i q_x (periodic)
  kXNegQx2 = 1,  // -q_x^2
  kXOpSH = 2,    // alpha (|q|^2 - q0^2)^2
  kXSinDx = 3,   // Neumann: x derivative of the cosine series, as the reversed coefficients
                 // -q_{N-k} X[N-k] (0 at k = 0) whose REDFT01 is (-1)^x psi_x
};
// tiles of shared memory a pencil mode uses (the exchange, a spectrum kept
// aside, Stokes components)
__host__ __device__ constexpr int pencil_sets(int mode) {
  return mode == kPencilStokes ? 3 : ((mode == kPencilStepAdv || mode == kPencilStepAdvGen || mode == kPencilInitAdv || mode == kPencilInit) ? 2 : 1);
}

// TKV: lines per CTA (the tile), 0 = the default of 16 (FP32) or 8 (FP64)
template <typename T, int N, bool DCT, int TKV = 0>
struct PencilCfg {
  using I = LineIdx<N>;
  static constexpr int E = I::E;
  static constexpr int G = I::G;
  // 128-byte row segments; at least one warp per CTA
  static constexpr int TK_DEF = sizeof(T) == 4 || N < 32 ? 16 : 8;
  static constexpr int TK = TKV > 0 ? TKV : TK_DEF;
  static constexpr int THREADS = TK * G;
  static constexpr int FP = DCT ? N * (N / 2) : N * (N / 2 + 1);
  static constexpr int TILES = FP / TK;
  static constexpr size_t SET_BYTES = size_t(TK) * N * sizeof(cplx<T>);
  static constexpr size_t red_off(int mode) { return SET_BYTES * pencil_sets(mode); }
  // |k| shells of the spectral-power histogram (shell = rint |index vector|):
  // at most sqrt(3) N / 2 + 1 periodic, sqrt(3) (N - 1) + 1 Neumann
  static constexpr int NSHELL = DCT ? 2 * N : N;
  static constexpr size_t shell_off(int mode) { return red_off(mode) + 64 * sizeof(double); }
  static constexpr size_t smem(int mode) {
    return shell_off(mode) + (mode == kPencilEnergy ? size_t(NSHELL) * sizeof(double) : 0);
  }
  // per-CTA shared memory limit of sm_100
  static constexpr bool fits(int mode) { return smem(mode) <= size_t(227) * 1024; }
  // Threads per SM that the register budget aims at: the E values of a thread, the
  // values read ahead and the temporaries of a radix-16 butterfly, without spills.
  // FP32 at 256^3: 384 threads (168 registers, three CTAs) and 512 (128 registers,
  // 8 bytes of spills) measure the same, 63.4 and 64.3 us.  FP32, E = 16: 768
  // threads periodic (64 x 64^3: 52.8 us, with 512 55.5), 512 Neumann, whose pairing
  // spills at 80 registers (57.0 us, with 768 60.6).
  static constexpr int step_threads() {
    return sizeof(T) == 4 ? (E == 32 ? 384 : (DCT ? 512 : 768)) : (E == 32 ? 256 : 512);
  }
  static constexpr int min_blocks(int mode) {
    // the six CTAs whose shared memory fits (Neumann 256^3 shells 229 us with five, 198)
    if (mode == kPencilEnergy && sizeof(T) == 8 && E == 32) return 384 / THREADS;
    return mode != kPencilInit && mode != kPencilInitAdv && mode != kPencilEnergy && step_threads() >= THREADS
               ? step_threads() / THREADS
               : 0;
  }
  // values of W (or of the adjoint's fields) a thread reads ahead of the update
  static constexpr int WB = E < 16 ? E : (sizeof(T) == 4 && (E == 32 || DCT) ? 16 : 8);
  static_assert(FP % TK == 0, "tile must divide the plane");
  static_assert(THREADS % 32 == 0, "pencil CTA must be whole warps");
};

template <typename T>
struct PencilArgs {
  const cplx<T>* src;   // step: partial of N ; init: partial of psi   [rep][x][FP]
  const cplx<T>* src2;  // init: partial of N(psi)
  cplx<T>* w;           // state W [rep][kx][FP] (adjoint: lambdahat)
  cplx<T>* dst;         // partial of scale * psihat^{n+1}, x-inverse applied [rep][x][FP]
  cplx<T>* dst_x;       // advection: partial of scale * i q_x psihat^{n+1}
  cplx<T>* dst_sh;      // advection: partial of scale * opSH psihat^{n+1}
  cplx<T>* spec_out;     // kFlSpecOut / kPencilSpec: psihat [rep][kx][FP]
  const cplx<T>* spec_a; // adjoint: psihat^n [rep][kx][FP]
  const cplx<T>* spec_b; // adjoint: psihat^{n+1} [rep][kx][FP]
  const cplx<T>* s3[3]; // Stokes: partial stress components (forward y,z applied)
  cplx<T>* u3[3];       // Stokes: partial velocity components (may alias s3)
  double* red;          // per-CTA spectral energy partial [rep][grid.x]
  double* shell;        // kFlShell: spectral power per |k| shell [rep][NSHELL] (accumulated, FP64)
  int* nonfinite;       // set to 1 when a new coefficient is NaN/Inf
  double coef;          // adjoint: c_{n-1} of the emitted mu combination (0 on the last reverse step)
  int xmul;             // kPencilXMul: XMulKind
  const T* q;           // wavenumber table (N entries)
  const double* qd;     // the same wavenumbers in FP64
  const T* qs;          // q of every B-side slot [t][E] (canonical order for the cosine transforms)
  const double* qds;    // qd of every B-side slot [t][E]
  const cplx<T>* lt;    // line tables (LineTab)
  PointParams pp;
  int flags;
};

template <typename T, int N, bool DCT, int TKV = 0>
struct PencilOps {
  using Cfg = PencilCfg<T, N, DCT, TKV>;
  using I = LineIdx<N>;
  using F = LineFFT<T, N>;
  static constexpr int E = Cfg::E, TK = Cfg::TK, FP = Cfg::FP;
  using X = TileExchange<T, TK>;
  using Tab = ColTables<T, N>;

  // wavenumber index of B-side slot s: the cosine transforms keep the canonical
  // pair order between their post- and pre-processing
  static __device__ __forceinline__ int kx_of(int t, int s) { return DCT ? I::c_slot(t, s) : I::b_elem(t, s); }

  // line (position f of every x-plane) between global memory and the A side
  static __device__ __forceinline__ void load(cplx<T> (&v)[E], const cplx<T>* __restrict__ src, int t) {
#pragma unroll
    for (int s = 0; s < E; ++s) v[s] = src[size_t(real_pos<N, DCT>(I::a_elem(t, s))) * FP];
  }
  static __device__ __forceinline__ void store(const cplx<T> (&v)[E], cplx<T>* __restrict__ dst, int t) {
#pragma unroll
    for (int s = 0; s < E; ++s) dst[size_t(real_pos<N, DCT>(I::a_elem(t, s))) * FP] = v[s];
  }
  // forward x transform: A side -> spectrum at kx_of
  static __device__ __forceinline__ void forward(cplx<T> (&v)[E], const X& x, int t, const Tab& tw, bool first_sync) {
    F::forward(v, t, x, tw, first_sync);
    if constexpr (DCT) {
      F::canon(v, t);
      F::dct2_post(v, t, tw);
    }
  }
  // inverse x transform: spectrum at kx_of -> A side
  static __device__ __forceinline__ void inverse(cplx<T> (&v)[E], const X& x, int t, const Tab& tw, bool first_sync) {
    if constexpr (DCT) {
      F::dct3_pre(v, t, tw);
      F::uncanon(v, t);
    }
    F::inverse(v, t, x, tw, first_sync);
  }
};

// Spectral multipliers of mode (kx, ky, kz) for replica epsilon ``eps``
template <typename T>
struct Mult {
  T mq2, a_lin, c1, c2;
};
template <typename T>
__device__ __forceinline__ Mult<T> make_mult(T qx, T qy, T qz, T eps, const PointParams& pp) {
  Mult<T> m;
  m.mq2 = qx * qx + qy * qy + qz * qz;
  const T d = m.mq2 - T(pp.q0 * pp.q0);
  const T op_sh = T(pp.alpha) * d * d;
  m.a_lin = eps - op_sh;
  const T h = T(0.5 * pp.dt);
  m.c1 = T(1) + h * m.a_lin;
  m.c2 = T(1) - h * m.a_lin;
  return m;
}

// correctly rounded reciprocal
__device__ __forceinline__ float rcp_rn(float x) { return __frcp_rn(x); }
__device__ __forceinline__ double rcp_rn(double x) { return __drcp_rn(x); }

// Both parts of a complex value as two independent reals (packed FP32x2)
template <typename T>
__device__ __forceinline__ cplx<T> both(T s) { return mk<T>(s, s); }
template <typename T>
__device__ __forceinline__ cplx<T> cfma(cplx<T> a, cplx<T> b, cplx<T> c) {
  return mk<T>(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
template <typename T>
__device__ __forceinline__ cplx<T> cmul2(cplx<T> a, cplx<T> b) { return mk<T>(a.x * b.x, a.y * b.y); }
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000 && !defined(SHB_NO_F32X2)
template <>
__device__ __forceinline__ float2 cfma<float>(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pk2(a)), "l"(pk2(b)), "l"(pk2(c)));
  return upk2(r);
}
template <>
__device__ __forceinline__ float2 cmul2<float>(float2 a, float2 b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk2(a)), "l"(pk2(b)));
  return upk2(r);
}
#endif
// products that no addition may absorb (ptxas fuses a packed mul and add)
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
// Reciprocals of the step's divisors C2 = 1 -+ (a rounded product), which are 0 (then
// psi turns non-finite with any reciprocal) or at least 2^-24 in size, 2^-53 in FP64.
// FP32: the hardware approximation and one Newton-Raphson iteration r + r (1 - x r) in
// fused arithmetic; equal to __frcp_rn for every significand from 2^-24 to 2^125, above
// which the approximation is flushed to 0 (NaN at infinity; C1 is infinite there too).
// With __frcp_rn the pencil pass takes 73.5 us instead of 64.5 at Neumann 256^3.
__device__ __forceinline__ float rcp2(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return fmaf(r, fmaf(-x, r, 1.0f), r);
}
__device__ __forceinline__ float2 rcp2(float2 x) {
  float2 r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(x.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(x.y));
  const float2 e = cfma<float>(make_float2(-x.x, -x.y), r, make_float2(1.0f, 1.0f));
  return cfma<float>(r, e, r);
}
// FP64: the 20-bit approximation and two iterations (relative error 2^-80 before
// the last rounding), 2^-53 to 2^1000
__device__ __forceinline__ double rcp2(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  return fma(r, fma(-x, r, 1.0), r);
}
__device__ __forceinline__ double2 rcp2(double2 x) { return make_double2(rcp2(x.x), rcp2(x.y)); }

// The same where the divisor may overflow: 0 beyond 2^125 (2^1000), as the quotient
__device__ __forceinline__ float rcp2_or_0(float x) { return fabsf(x) > 0x1p125f ? 0.0f : rcp2(x); }
__device__ __forceinline__ double rcp2_or_0(double x) { return fabs(x) > 0x1p1000 ? 0.0 : rcp2(x); }

// One mode (Neumann: the pair kz, kz + 1 in .x, .y) of the CNAB2 update:
//   psihat^{n+1} = (W + 3dt/2 Nhat) / C2,  W' = C1 psihat^{n+1} - dt/2 Nhat
// h = dt/2, h3 = 3dt/2, qyz = q_y^2 + q_z^2 - q0^2
template <typename T, bool DCT>
__device__ __forceinline__ void cnab2_update(T qx, cplx<T> qyz, T alpha, T eps, T h, T h3, cplx<T> nh, cplx<T>& wv,
                                             cplx<T>& pn) {
  const cplx<T> d = cfma<T>(both<T>(qx), both<T>(qx), qyz);
  const cplx<T> al = cfma<T>(cmul2<T>(both<T>(-alpha), d), d, both<T>(eps));
  const cplx<T> ha = mk<T>(mul_rn(h, al.x), mul_rn(h, al.y));
  const cplx<T> c2 = csub<T>(both<T>(T(1)), ha), c1 = cadd<T>(both<T>(T(1)), ha);
  cplx<T> inv;
  if constexpr (DCT) inv = rcp2(c2);
  else inv = both<T>(rcp2(c2.x));  // one multiplier for both parts
  pn = cmul2<T>(cfma<T>(both<T>(h3), nh, wv), inv);
  wv = cfma<T>(c1, pn, cmul2<T>(both<T>(-h), nh));
}
// IMEX Euler: psihat^{n+1} = (psihat + dt Nhat) / (1 - dt aLin),  W' = psihat^{n+1}.
// Where aLin overflows the mode vanishes (with CNAB2 it is not finite anyway).
template <typename T, bool DCT>
__device__ __forceinline__ void euler_update(T qx, cplx<T> qyz, T alpha, T eps, T dt, cplx<T> nh, cplx<T>& wv,
                                             cplx<T>& pn) {
  const cplx<T> d = cfma<T>(both<T>(qx), both<T>(qx), qyz);
  const cplx<T> al = cfma<T>(cmul2<T>(both<T>(-alpha), d), d, both<T>(eps));
  const cplx<T> c2 = cfma<T>(both<T>(-dt), al, both<T>(T(1)));
  cplx<T> inv;
  if constexpr (DCT) inv = mk<T>(rcp2_or_0(c2.x), rcp2_or_0(c2.y));
  else inv = both<T>(rcp2_or_0(c2.x));
  pn = cmul2<T>(cfma<T>(both<T>(dt), nh, wv), inv);
  wv = pn;
}
// The same of FP32 fields with the per-mode multipliers and the update in FP64 from
// the FP64 wavenumbers, one rounding of each stored result.  A multiplier rounded to
// FP32 repeats the same relative error every step, which drifts a mode's amplitude
// linearly with the step count.  The products are spelled out so that every kernel
// rounds alike (a step, a traced step and the adjoint's recompute of it).
template <typename T, bool DCT>
__device__ __forceinline__ void cnab2_update64(double qx, double qyz0, double qyz1, double alpha, double eps, double h,
                                               cplx<T> nh, cplx<T>& wv, cplx<T>& pn) {
  auto one = [&](double c1, double inv, T n, T& w1, T& p1) {
    p1 = T((double(w1) + 3.0 * h * double(n)) * inv);
    w1 = T(fma(c1, double(p1), -__dmul_rn(h, double(n))));
  };
  const double e0 = qx * qx + qyz0;
  const double b0 = eps - alpha * e0 * e0;
  const double hb0 = __dmul_rn(h, b0), c10 = 1.0 + hb0, i0 = rcp2(1.0 - hb0);
  double c11 = c10, i1 = i0;
  if constexpr (DCT) {
    const double e1 = qx * qx + qyz1;
    const double b1 = eps - alpha * e1 * e1;
    const double hb1 = __dmul_rn(h, b1);
    c11 = 1.0 + hb1;
    i1 = rcp2(1.0 - hb1);
  }
  one(c10, i0, nh.x, wv.x, pn.x);
  one(c11, i1, nh.y, wv.y, pn.y);
}
template <typename T, bool DCT>
__device__ __forceinline__ void euler_update64(double qx, double qyz0, double qyz1, double alpha, double eps, double dt,
                                               cplx<T> nh, cplx<T>& wv, cplx<T>& pn) {
  const double e0 = qx * qx + qyz0, i0 = rcp2_or_0(1.0 - dt * (eps - alpha * e0 * e0));
  double i1 = i0;
  if constexpr (DCT) {
    const double e1 = qx * qx + qyz1;
    i1 = rcp2_or_0(1.0 - dt * (eps - alpha * e1 * e1));
  }
  pn = mk<T>(T((double(wv.x) + dt * double(nh.x)) * i0), T((double(wv.y) + dt * double(nh.y)) * i1));
  wv = pn;
}

// What bounds it: Neumann 256^3 FP32 moves 268 MB (41 us at the measured copy
// rate) in 55 us; 24.5 M warp instructions (45 % of the issue slots), 2.1 M
// shared-memory wavefronts; the waits are the HBM latency of the line loads and of
// W.  The 16-values-per-thread form it replaces staged tiles in shared memory and
// paired k with N - k by shuffles: 42 M instructions, 7.5 M wavefronts, 76 us.
// Step pencil pass, event to event, that form -> now: Neumann 256^3 FP32 76.3 -> 61.1,
// periodic 65.3 -> 54.8, Neumann 256^3 FP64 154 -> 143, Neumann 512^3 FP64 1716 -> 1138,
// periodic 512^3 FP32 634 -> 470, periodic 128^3 FP64 23.3 -> 16.6, 64 x 64^3 FP32 68.9
// -> 52.9 periodic, 84.0 -> 57.9 Neumann, FP64 update (kPencilStepU64) Neumann 256^3
// 95.7 -> 72.1 us.
template <typename T, int N, bool DCT, int MODE, int TKV = 0>
__global__ void __launch_bounds__(PencilCfg<T, N, DCT, TKV>::THREADS, PencilCfg<T, N, DCT, TKV>::min_blocks(MODE))
pencil_kernel(const __grid_constant__ PencilArgs<T> a) {
  using Cfg = PencilCfg<T, N, DCT, TKV>;
  using Ops = PencilOps<T, N, DCT, TKV>;
  constexpr int E = Cfg::E, TK = Cfg::TK, FP = Cfg::FP, WB = Cfg::WB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* buf = reinterpret_cast<cplx<T>*>(smem_raw);
  double* scratch = reinterpret_cast<double*>(smem_raw + Cfg::red_off(MODE));

  const int f0 = blockIdx.x * TK;
  const int rep = blockIdx.y;
  const int c = threadIdx.x % TK, t = threadIdx.x / TK;
  const int f = f0 + c;
  const typename Ops::X x{buf + c};
  const typename Ops::Tab tw(a.lt, t);
  // this thread's slots of a spectrum kept aside: conflict-free, private
  cplx<T>* aside = buf + size_t(TK) * N + threadIdx.x;
  const size_t line = size_t(rep) * N * FP + f;  // position f of plane 0 (and of kx = 0)
  const T eps = T(a.pp.eps[rep]);
  const T scale = T(a.pp.scale);

  // in-plane wavenumber indices of this line
  int ky, kz;
  if (DCT) {
    ky = f / (N / 2);
    kz = 2 * (f % (N / 2));  // the pair holds kz and kz + 1
  } else if (f < N * (N / 2)) {
    ky = f / (N / 2);
    kz = f % (N / 2);
  } else {
    ky = f - N * (N / 2);
    kz = N / 2;
  }
  const T qy = __ldg(&a.q[ky]);
  const T qz0 = __ldg(&a.q[kz]);
  const T qz1 = DCT ? __ldg(&a.q[kz + 1]) : T(0);
  const T* qs = a.qs + t * E;

  cplx<T> v[E];
  KahanSum acc;
  const bool want_energy = (a.flags & kFlEnergy) != 0;
  grid_dependency_wait();

  // W is read after the transform: bring its rows (one 128-byte segment per kx)
  // into L2 meanwhile.  Neumann 256^3 FP32: pencil pass 68.7 -> 64.3 us.
  // Not for FP64 (137 -> 142 us), nor where the fields live in L2 anyway.
  auto prefetch_w = [&] {
    if constexpr (sizeof(T) == 4 && N >= 256) {
      const cplx<T>* wt = a.w + size_t(rep) * N * FP + f0;
      for (int k = threadIdx.x; k < N; k += Cfg::THREADS)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(wt + size_t(k) * FP));
    }
  };
  if constexpr (MODE == kPencilStep || MODE == kPencilStepU64 || MODE == kPencilStepAdv || MODE == kPencilStepSpec ||
                MODE == kPencilStepEuler) {
    // One scheme and nothing else: this kernel is bound by the instructions it issues
    // and fetches, so what only some runs ask for (kPencilStepGen) stays out of it
    cplx<T>* w = a.w + line;
    Ops::load(v, a.src + line, t);
    prefetch_w();
    Ops::forward(v, x, t, tw, false);
    const T q02 = T(a.pp.q0 * a.pp.q0), alpha = T(a.pp.alpha);
    const T h = T(0.5 * a.pp.dt), h3 = T(1.5 * a.pp.dt);
    const T qyz0 = qy * qy + qz0 * qz0 - q02;
    const cplx<T> qyz = mk<T>(qyz0, DCT ? qy * qy + qz1 * qz1 - q02 : qyz0);
    double hd = 0.0, epsd = 0.0, qyz0d = 0.0, qyz1d = 0.0;
    if constexpr (MODE == kPencilStepU64) {
      hd = 0.5 * a.pp.dt;
      epsd = a.pp.eps[rep];
      const double qyd = __ldg(&a.qd[ky]), qz0d = __ldg(&a.qd[kz]);
      qyz0d = qyd * qyd + qz0d * qz0d - a.pp.q0 * a.pp.q0;
      if constexpr (DCT) {
        const double qz1d = __ldg(&a.qd[kz + 1]);
        qyz1d = qyd * qyd + qz1d * qz1d - a.pp.q0 * a.pp.q0;
      }
    }
    cplx<T> finite = mk<T>(T(0), T(0));  // stays 0 unless a new coefficient is NaN / Inf
#pragma unroll
    for (int s0 = 0; s0 < E; s0 += WB) {
      cplx<T> wreg[WB];
#pragma unroll
      for (int i = 0; i < WB; ++i) wreg[i] = w[size_t(Ops::kx_of(t, s0 + i)) * FP];
#pragma unroll
      for (int i = 0; i < WB; ++i) {
        const int s = s0 + i;
        const cplx<T> nh = v[s];
        cplx<T> wv = wreg[i];
        cplx<T> pn;
        if constexpr (MODE == kPencilStepU64) {
          const double qxd = __ldg(&a.qds[t * E + s]);
          cnab2_update64<T, DCT>(qxd, qyz0d, qyz1d, a.pp.alpha, epsd, hd, nh, wv, pn);
        } else if constexpr (MODE == kPencilStepEuler) {
          euler_update<T, DCT>(__ldg(&qs[s]), qyz, alpha, eps, T(a.pp.dt), nh, wv, pn);
        } else {
          cnab2_update<T, DCT>(__ldg(&qs[s]), qyz, alpha, eps, h, h3, nh, wv, pn);
        }
        finite = cfma<T>(pn, both<T>(T(0)), finite);
        if constexpr (MODE == kPencilStepSpec) a.spec_out[line + size_t(Ops::kx_of(t, s)) * FP] = pn;
        w[size_t(Ops::kx_of(t, s)) * FP] = wv;
        v[s] = cscale<T>(pn, scale);
      }
    }
    if (!(finite.x == T(0) && finite.y == T(0))) *a.nonfinite = 1;
  } else if constexpr (MODE == kPencilStepGen || MODE == kPencilStepU64Gen || MODE == kPencilStepAdvGen) {
    cplx<T>* w = a.w + line;
    Ops::load(v, a.src + line, t);
    prefetch_w();
    Ops::forward(v, x, t, tw, false);
    const T q02 = T(a.pp.q0 * a.pp.q0), alpha = T(a.pp.alpha);
    const T h = T(0.5 * a.pp.dt), h3 = T(1.5 * a.pp.dt), dtT = T(a.pp.dt);
    const T qyz0 = qy * qy + qz0 * qz0 - q02;
    const cplx<T> qyz = mk<T>(qyz0, DCT ? qy * qy + qz1 * qz1 - q02 : qyz0);
    // FP64 values of the FP32 update; the scalars stay kernel parameters
    const double epsd = a.pp.eps[rep];
    double qyz0d = 0.0, qyz1d = 0.0;
    if constexpr (MODE == kPencilStepU64Gen) {
      const double qyd = __ldg(&a.qd[ky]), qz0d = __ldg(&a.qd[kz]);
      qyz0d = qyd * qyd + qz0d * qz0d - a.pp.q0 * a.pp.q0;
      if constexpr (DCT) {
        const double qz1d = __ldg(&a.qd[kz + 1]);
        qyz1d = qyd * qyd + qz1d * qz1d - a.pp.q0 * a.pp.q0;
      }
    }
    cplx<T>* spec = (a.flags & kFlSpecOut) ? a.spec_out + line : nullptr;
    cplx<T> finite = mk<T>(T(0), T(0));
    // One loop per scheme, with and without the energy: branches inside one loop kept
    // the values of a thread apart.  256^3 pencil pass with the energy trace, us, before
    // -> now: FP32 Neumann 105 -> 84, periodic 74 -> 62, FP64 Neumann 188 -> 156 (IMEX
    // without it, kPencilStepEuler: 97 -> 78, 68 -> 53, 179 -> 164).
    auto update = [&](auto cnab2_, auto energy_) {
      constexpr bool CN = decltype(cnab2_)::value, EN = decltype(energy_)::value;
#pragma unroll
      for (int s0 = 0; s0 < E; s0 += WB) {
        cplx<T> wreg[WB];
#pragma unroll
        for (int i = 0; i < WB; ++i) wreg[i] = w[size_t(Ops::kx_of(t, s0 + i)) * FP];
#pragma unroll
        for (int i = 0; i < WB; ++i) {
          const int s = s0 + i;
          const int kx = Ops::kx_of(t, s);
          const T qx = __ldg(&qs[s]);
          const cplx<T> nh = v[s];
          cplx<T> wv = wreg[i], pn;
          if constexpr (MODE == kPencilStepU64Gen) {
            const double qxd = __ldg(&a.qds[t * E + s]);
            if constexpr (CN) cnab2_update64<T, DCT>(qxd, qyz0d, qyz1d, a.pp.alpha, epsd, 0.5 * a.pp.dt, nh, wv, pn);
            else euler_update64<T, DCT>(qxd, qyz0d, qyz1d, a.pp.alpha, epsd, a.pp.dt, nh, wv, pn);
          } else {
            if constexpr (CN) cnab2_update<T, DCT>(qx, qyz, alpha, eps, h, h3, nh, wv, pn);
            else euler_update<T, DCT>(qx, qyz, alpha, eps, dtT, nh, wv, pn);
          }
          if constexpr (EN) {
            const T qx2 = qx * qx;
            if constexpr (!DCT) {
              const double d = double(qx2 + qyz.x);
              const double wgt = (kz == 0 || kz == N / 2) ? 1.0 : 2.0;
              acc.add(wgt * d * d * (double(pn.x) * pn.x + double(pn.y) * pn.y));
            } else {
              const double wxy = (kx == 0 ? 0.5 : 1.0) * (ky == 0 ? 0.5 : 1.0);
              const double e0 = double(qx2 + qyz.x), e1 = double(qx2 + qyz.y);
              acc.add(wxy * ((kz == 0 ? 0.5 : 1.0) * e0 * e0 * double(pn.x) * pn.x + e1 * e1 * double(pn.y) * pn.y));
            }
          }
          finite = cfma<T>(pn, both<T>(T(0)), finite);
          if (spec) spec[size_t(kx) * FP] = pn;
          w[size_t(kx) * FP] = wv;
          v[s] = cscale<T>(pn, scale);
        }
      }
    };
    using Yes = std::true_type;
    using No = std::false_type;
    if (a.pp.scheme == kCNAB2) {
      if (want_energy) update(Yes(), Yes());
      else update(Yes(), No());
    } else {
      if (want_energy) update(No(), Yes());
      else update(No(), No());
    }
    if (!(finite.x == T(0) && finite.y == T(0))) *a.nonfinite = 1;
  } else if constexpr (MODE == kPencilEnergy) {
    // gradient part of the energy of the current state from its partial P,
    // and (kFlShell) its spectral power per |k| shell
    double* hist = reinterpret_cast<double*>(smem_raw + Cfg::shell_off(MODE));
    const bool want_shell = (a.flags & kFlShell) != 0;
    if (want_shell)
      for (int i = threadIdx.x; i < Cfg::NSHELL; i += Cfg::THREADS) hist[i] = 0.0;
    Ops::load(v, a.src + line, t);
    __syncthreads();
    Ops::forward(v, x, t, tw, false);
    // P = IDFT_x(scale psihat): its forward x transform is N scale psihat
    // (REDFT10 after REDFT01: 2N scale psihat)
    const double inv = 1.0 / (a.pp.scale * (DCT ? 2 * N : N));
    // The spectrum goes through this thread's slots of the exchange tile, so that the
    // loops stay rolled: their FP64 code for 32 values would fill the instruction
    // cache.  Periodic: k and N - k, which share |q| and the shell, are added up first.
    // 256^3, whole calls, us, before -> now: energy FP32 Neumann 181 -> 133, FP64 278 ->
    // 234 periodic; dominant wavenumber FP64 periodic 208 -> 112.
    if constexpr (!DCT) Ops::F::canon(v, t);
    constexpr int NV = DCT ? E : E / 2;  // terms of a thread
    cplx<T>* own = buf + threadIdx.x;
    __syncthreads();
#pragma unroll
    for (int s = 0; s < E; ++s) own[s * Cfg::THREADS] = v[s];
    // f(kx, power of kz, power of kz + 1) of term s; periodic: the whole pair's power
    // as the first, and k = 0 and N / 2, which have no mirror, as two terms
    auto term = [&](int s, auto f) {
      const cplx<T> u = own[s * Cfg::THREADS];
      const double px = double(u.x) * inv, py = double(u.y) * inv;
      if constexpr (DCT) {
        f(Ops::kx_of(t, s), px * px, py * py);
      } else {
        const cplx<T> m = own[(E - 1 - s) * Cfg::THREADS];
        const double mx = double(m.x) * inv, my = double(m.y) * inv;
        const double pu = px * px + py * py, pm = mx * mx + my * my;
        const int k = LineIdx<N>::c_elem(t, s);
        const bool self = s == 0 && t == 0;
        f(k < N / 2 ? k : N - k, self ? pu : pu + pm, 0.0);
        if (s == 0) f(N / 2, self ? pm : 0.0, 0.0);
      }
    };
    const double wy = ky == 0 ? 0.5 : 1.0, wz = kz == 0 ? 0.5 : 1.0;
    const double wgt = (kz == 0 || kz == N / 2) ? 1.0 : 2.0;  // periodic: kz also stands for its conjugate
    if (want_energy) {
      const double q02 = double(a.pp.q0) * a.pp.q0;
#pragma unroll 1
      for (int s = 0; s < NV; ++s)
        term(s, [&](int kx, double p0, double p1) {
          const T qx = __ldg(&a.q[kx]);
          const double d0 = q02 - double(qx * qx + qy * qy + qz0 * qz0);
          if constexpr (!DCT) {
            acc.add(wgt * d0 * d0 * p0);
          } else {
            const double d1 = q02 - double(qx * qx + qy * qy + qz1 * qz1);
            acc.add((kx == 0 ? 0.5 : 1.0) * wy * (wz * d0 * d0 * p0 + d1 * d1 * p1));
          }
        });
    }
    if (want_shell) {
      // shell = rint |(ix, iy, iz)|: signed indices (Nyquist +N/2) on the periodic
      // grid.  |.|^2 is below 2^20 and never within 1/4 of (k + 1/2)^2, so FP32 rounds
      // to the same shell.
      auto shell = [](int r2) { return __float2int_rn(__fsqrt_rn(float(r2))); };
      // |k| is monotonic along the lanes of one ky row (or half the kz = N/2 column), so
      // those of one shell are neighbours: the first adds their sum, instead of all of
      // them meeting at one shared-memory word
      constexpr int W = TK < N / 2 ? TK : N / 2;  // a tile of 16^3 holds two rows
      const int cw = c % W;
      auto deposit = [&](int sh, double pw) {
#pragma unroll
        for (int o = 1; o < W; o <<= 1) {
          const int so = __shfl_down_sync(0xffffffffu, sh, o, W);
          const double po = __shfl_down_sync(0xffffffffu, pw, o, W);
          if (cw + o < W && so == sh) pw += po;
        }
        const int left = __shfl_up_sync(0xffffffffu, sh, 1, W);
        if (cw == 0 || left != sh) atomicAdd(&hist[sh], pw);
      };
      const int iy = DCT || ky <= N / 2 ? ky : ky - N;
#pragma unroll 2
      for (int s = 0; s < NV; ++s)
        term(s, [&](int kx, double p0, double p1) {
          const int r2 = kx * kx + iy * iy;
          if constexpr (!DCT) {
            deposit(shell(r2 + kz * kz), wgt * p0);
          } else {
            const double wxy = (kx == 0 ? 0.5 : 1.0) * wy;
            deposit(shell(r2 + kz * kz), wxy * wz * p0);
            deposit(shell(r2 + (kz + 1) * (kz + 1)), wxy * p1);
          }
        });
    }
    if (want_shell) {
      __syncthreads();
      for (int i = threadIdx.x; i < Cfg::NSHELL; i += Cfg::THREADS)
        if (hist[i] != 0.0) atomicAdd(&a.shell[size_t(rep) * Cfg::NSHELL + i], hist[i]);
    }
  } else if constexpr (MODE == kPencilSpec) {
    Ops::load(v, a.src + line, t);
    Ops::forward(v, x, t, tw, false);
    // P = IDFT_x(scale psihat): its forward x transform is N scale psihat
    const T inv = T(1.0 / (a.pp.scale * N));
#pragma unroll
    for (int s = 0; s < E; ++s) a.spec_out[line + size_t(Ops::kx_of(t, s)) * FP] = cscale<T>(v[s], inv);
  } else if constexpr (MODE == kPencilAdjInit || MODE == kPencilAdj) {
    if constexpr (!DCT) {
      // Discrete adjoint of CNAB2 (reverse of psi^{n+1} = A psi^n + B (c_n N^n - N^{n-1}), c_0 = 2,
      // c_n = 3):
      //   lambdahat^n = A lambdahat^{n+1} + ghat^n,  mu^n = B lambda^n,
      //   g^{n-1} = N'(psi^{n-1}) (c_{n-1} mu^n - mu^{n+1}).
      // The output partial is that combination, scale B (coef lambdahat^n - lambdahat^{n+1}),
      // so the plane pass of step n-1 reads one field.  The parameter gradients
      //   dL/dtheta = sum_n <lambda^{n+1}, dt/2 (psihat^n + psihat^{n+1}) / C2 da/dtheta>
      // are regrouped by psihat^m: step n adds <lambda^{n+1} + [n >= 1] lambda^n, D psihat^n>, and
      // the first reverse step (spec_b set) also <lambda^{n+1}, D psihat^{n+1}>.
      Ops::load(v, a.src + line, t);
      Ops::forward(v, x, t, tw, false);
      cplx<T>* w = a.w + line;
      const T q02 = T(a.pp.q0 * a.pp.q0), alpha = T(a.pp.alpha), h = T(0.5 * a.pp.dt);
      const T qyz = qy * qy + qz0 * qz0;
      const double wgt = ((kz == 0 || kz == N / 2) ? 1.0 : 2.0) / (double(N) * N * N);
      const double dadq0 = 4.0 * a.pp.alpha * a.pp.q0;
      const T coef = T(a.coef);
      const bool lam_n = a.coef != 0.0;  // n >= 1
      // a thread's E terms are summed plainly (FP64); the per-CTA and
      // per-step totals are combined in a fixed order
      double ge = 0.0, gq = 0.0;
      constexpr int AB = WB / 2;
#pragma unroll
      for (int s0 = 0; s0 < E; s0 += AB) {
        cplx<T> lreg[AB], preg[AB];
        if constexpr (MODE == kPencilAdj) {
#pragma unroll
          for (int i = 0; i < AB; ++i) {
            const size_t k = size_t(Ops::kx_of(t, s0 + i)) * FP;
            lreg[i] = w[k];
            preg[i] = a.spec_a[line + k];
          }
        }
#pragma unroll
        for (int i = 0; i < AB; ++i) {
          const int s = s0 + i;
          const size_t k = size_t(Ops::kx_of(t, s)) * FP;
          const T qx = __ldg(&qs[s]);
          const T mq2 = qx * qx + qyz;
          const T d = mq2 - q02;
          const T al = eps - alpha * d * d;
          const T inv2 = rcp_rn(T(1) - h * al);
          const T am = (T(1) + h * al) * inv2, bm = h * inv2;
          cplx<T> lam = v[s];
          cplx<T> lnext = mk<T>(T(0), T(0));
          if constexpr (MODE == kPencilAdj) {
            const cplx<T> l1 = lreg[i];
            lam = mk<T>(am * l1.x + lam.x, am * l1.y + lam.y);
            const cplx<T> pa = preg[i];
            const double wx = double(l1.x) + (lam_n ? double(lam.x) : 0.0);
            const double wy = double(l1.y) + (lam_n ? double(lam.y) : 0.0);
            double dot = wx * double(pa.x) + wy * double(pa.y);
            if (a.spec_b) {
              const cplx<T> pb = a.spec_b[line + k];
              dot += double(l1.x) * double(pb.x) + double(l1.y) * double(pb.y);
            }
            const double inner = wgt * double(bm) * dot;  // bm = dt/2 / C2
            ge += inner;
            gq += inner * double(d);
            lnext = l1;
          }
          w[k] = lam;
          v[s] = cscale<T>(mk<T>(coef * lam.x - lnext.x, coef * lam.y - lnext.y), scale * bm);
        }
      }
      if constexpr (MODE == kPencilAdj) {
        // each CTA accumulates into its own slot over the reverse sweep (fixed order)
        const double te = block_sum(ge, scratch);
        const double tq = block_sum(gq, scratch);
        if (threadIdx.x == 0) {
          double* o = a.red + (size_t(rep) * gridDim.x + blockIdx.x) * 2;
          o[0] += te;
          o[1] += tq * dadq0;
        }
      }
    }
  } else if constexpr (MODE == kPencilAdjOut) {
#pragma unroll
    for (int s = 0; s < E; ++s) v[s] = cscale<T>(a.w[line + size_t(Ops::kx_of(t, s)) * FP], scale);
  } else if constexpr (MODE == kPencilXMul) {
    Ops::load(v, a.src + line, t);
    Ops::forward(v, x, t, tw, false);
    // P is the x-inverse of (scale X); its forward x transform is N scale X
    // (2N scale X for REDFT10 after REDFT01): multiply by m(q) / N (/ 2N)
    const T invn = T(1) / T(DCT ? 2 * N : N);
    const T q02 = T(a.pp.q0 * a.pp.q0), alpha = T(a.pp.alpha);
    if (DCT && a.xmul == kXSinDx) {
      // RODFT01(X)[x] = (-1)^x REDFT01(X reversed)[x] (the sine series of
      // d/dx): slot kx takes -q_{N-kx} times coefficient N - kx, the mirror of
      // kx; the plane pass applies (-1)^x
      using I = LineIdx<N>;
#pragma unroll
      for (int r = 0; r < E / 2; ++r) {
        const int k = I::c_elem(t, r), m = E - 1 - r;
        const bool self = r == 0 && t == 0;  // the pair (0, N/2): each its own mirror
        const cplx<T> lo = v[r], hi = v[m];
        const T wk = k == 0 ? T(0) : -__ldg(&a.q[N - k]) * invn;
        const T wm = self ? -__ldg(&a.q[N / 2]) * invn : -__ldg(&a.q[k]) * invn;
        v[r] = cscale<T>(hi, wk);
        v[m] = self ? cscale<T>(hi, wm) : cscale<T>(lo, wm);
      }
    } else {
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const T qx = __ldg(&qs[s]);
        const cplx<T> val = v[s];
        if (a.xmul == kXIqx) {
          v[s] = mk<T>(-qx * invn * val.y, qx * invn * val.x);
        } else if (a.xmul == kXNegQx2) {
          v[s] = cscale<T>(val, -qx * qx * invn);
        } else {
          const T d0 = qx * qx + qy * qy + qz0 * qz0 - q02;
          const T d1 = DCT ? qx * qx + qy * qy + qz1 * qz1 - q02 : d0;
          v[s] = mk<T>(alpha * d0 * d0 * invn * val.x, alpha * d1 * d1 * invn * val.y);
        }
      }
    }
  } else if constexpr (MODE == kPencilStokes) {
    // The three stress components go forward one after the other, the second and the
    // third on their way into shared memory meanwhile; there the finished spectra
    // take the place of the lines (every thread reads and writes its own slots only).
    // The projector runs in registers, and the three velocity components go back.  1 / |q|^2
    // is the correctly rounded one: |q|^2 goes with dx^-2 and may be subnormal, where
    // rcp2 has no value, and the pass waits for memory either way (256^3 FP32 step 819 us
    // with rcp2, 821 with rcp_rn; Neumann 1004, 1006; FP64 1882, 1905).
    cplx<T>* keep[2] = {aside, aside + size_t(TK) * N};
    constexpr int TH = Cfg::THREADS;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const cplx<T>* src = a.s3[m + 1] + line;
#pragma unroll
      for (int s = 0; s < E; ++s)
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(keep[m] + s * TH)),
                     "l"(src + size_t(real_pos<N, DCT>(LineIdx<N>::a_elem(t, s))) * FP), "n"(int(sizeof(cplx<T>)))
                     : "memory");
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    Ops::load(v, a.s3[0] + line, t);
    Ops::forward(v, x, t, tw, false);
#pragma unroll 1
    for (int m = 0; m < 2; ++m) {
      if (m == 0) asm volatile("cp.async.wait_group 1;" ::: "memory");
      else asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const cplx<T> u = keep[m][s * TH];
        keep[m][s * TH] = v[s];
        v[s] = u;
      }
      Ops::forward(v, x, t, tw, true);
    }
    const T ce = T(1.0 / a.pp.eta_rho);
    if constexpr (DCT) {
      // Neumann box: the stress came in as the cosine-transform partial of
      // (-1)^(x+y+z) S, whose REDFT10 at index k is the RODFT10 of S at index
      // N-1-k (cosFFT/comet/morphSurfK.cpp:390-418 uses RODFT10/01).  So the
      // sine-wavenumber projector u = CM1 (S - CM2 (Vs . S)) of morphSurfK.cpp:
      // 862-882, Vs(m) = pi (m+1)/L, reads Vs = pi (N-k)/L at index k; the
      // inverse REDFT01 then yields (-1)^(x+y+z) u, unsigned by the plane pass.
      const T q1 = __ldg(&a.q[1]);  // pi / L
      const T sy = T(N - ky) * q1, sz0 = T(N - kz) * q1, sz1 = T(N - kz - 1) * q1;
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const T sx = T(N - Ops::kx_of(t, s)) * q1;
        const cplx<T> px = keep[0][s * TH], py = keep[1][s * TH], pz = v[s];
        // .x holds kz, .y holds kz + 1
        const T m0 = sx * sx + sy * sy + sz0 * sz0, m1 = sx * sx + sy * sy + sz1 * sz1;
        const T i0 = rcp_rn(m0), i1 = rcp_rn(m1);
        const T c0 = scale * ce * i0, c1 = scale * ce * i1;
        const T d0 = sx * px.x + sy * py.x + sz0 * pz.x;
        const T d1 = sx * px.y + sy * py.y + sz1 * pz.y;
        keep[0][s * TH] = mk<T>(c0 * (px.x - sx * i0 * d0), c1 * (px.y - sx * i1 * d1));
        keep[1][s * TH] = mk<T>(c0 * (py.x - sy * i0 * d0), c1 * (py.y - sy * i1 * d1));
        v[s] = mk<T>(c0 * (pz.x - sz0 * i0 * d0), c1 * (pz.y - sz1 * i1 * d1));
      }
    } else {
      // S -> u = scale CM1 (S - CM2 (q.S)),  CM1 = 1/(rho eta |q|^2), CM2 = q/|q|^2, both 0 at q = 0
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const T qx = __ldg(&qs[s]);
        const T mq2 = qx * qx + qy * qy + qz0 * qz0;
        const cplx<T> sx = keep[0][s * TH], sy = keep[1][s * TH], sz = v[s];
        cplx<T> ux = mk<T>(T(0), T(0)), uy = ux, uz = ux;
        if (mq2 != T(0)) {
          const T inv = rcp_rn(mq2);
          const T cm1 = scale * ce * inv;
          const cplx<T> dot = mk<T>(qx * sx.x + qy * sy.x + qz0 * sz.x, qx * sx.y + qy * sy.y + qz0 * sz.y);
          ux = mk<T>(cm1 * (sx.x - qx * inv * dot.x), cm1 * (sx.y - qx * inv * dot.y));
          uy = mk<T>(cm1 * (sy.x - qy * inv * dot.x), cm1 * (sy.y - qy * inv * dot.y));
          uz = mk<T>(cm1 * (sz.x - qz0 * inv * dot.x), cm1 * (sz.y - qz0 * inv * dot.y));
        }
        keep[0][s * TH] = ux;
        keep[1][s * TH] = uy;
        v[s] = uz;
      }
    }
#pragma unroll 1
    for (int comp = 2; comp >= 0; --comp) {
      if (comp < 2) {
#pragma unroll
        for (int s = 0; s < E; ++s) v[s] = keep[comp][s * TH];
      }
      Ops::inverse(v, x, t, tw, true);
      Ops::store(v, a.u3[comp] + line, t);
    }
  } else {  // kPencilInit(Adv): W^0 from psi^0 and N(psi^0); P^0 from psi^0
    constexpr int TH = Cfg::THREADS;
    Ops::load(v, a.src2 + line, t);
    Ops::forward(v, x, t, tw, false);
#pragma unroll
    for (int s = 0; s < E; ++s) aside[s * TH] = v[s];
    Ops::load(v, a.src + line, t);
    Ops::forward(v, x, t, tw, true);
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const T qx = __ldg(&qs[s]);
      const cplx<T> ph = v[s], nh = aside[s * TH];
      cplx<T> wv;
      const Mult<T> m0 = make_mult<T>(qx, qy, qz0, eps, a.pp);
      const Mult<T> m1 = DCT ? make_mult<T>(qx, qy, qz1, eps, a.pp) : m0;
      if (a.pp.scheme == kCNAB2) {
        wv.x = m0.c1 * ph.x - T(0.5 * a.pp.dt) * nh.x;
        wv.y = m1.c1 * ph.y - T(0.5 * a.pp.dt) * nh.y;
      } else {
        wv = ph;
      }
      a.w[line + size_t(Ops::kx_of(t, s)) * FP] = wv;
      v[s] = cscale<T>(ph, scale);
    }
  }

  if constexpr (MODE == kPencilStep || MODE == kPencilStepSpec || MODE == kPencilStepEuler || MODE == kPencilStepGen ||
                MODE == kPencilStepU64 ||
                MODE == kPencilStepU64Gen || MODE == kPencilInit || MODE == kPencilXMul ||
                MODE == kPencilAdjInit || MODE == kPencilAdj || MODE == kPencilAdjOut) {
    Ops::inverse(v, x, t, tw, MODE != kPencilAdjOut);
    Ops::store(v, a.dst + line, t);
  } else if constexpr (MODE == kPencilStepAdv || MODE == kPencilStepAdvGen || MODE == kPencilInitAdv) {
    // v = scale psihat^{n+1}; emit its partial, one inverse x transform each, and
    //   periodic: those of i q_x v and opSH v (periodicFFT/pf3d.cpp:404-407)
    //   Neumann, where asked: those of -q_x^2 v (the x half of the substrate's
    //   in-plane Laplacian) and of opSH v (L psi of the Stokes stress,
    //   cosFFT/comet/morphSurfK.cpp:686-696)
    constexpr int TH = Cfg::THREADS;
    const T q02 = T(a.pp.q0 * a.pp.q0), alpha = T(a.pp.alpha);
#pragma unroll
    for (int s = 0; s < E; ++s) aside[s * TH] = v[s];
    cplx<T>* outs[3] = {a.dst, a.dst_x, a.dst_sh};
#pragma unroll 1
    for (int o = 0; o < 3; ++o) {
      if (!outs[o]) continue;  // uniform over the grid
      if (o > 0) {
#pragma unroll
        for (int s = 0; s < E; ++s) {
          const cplx<T> val = aside[s * TH];
          const T qx = __ldg(&qs[s]);
          if (o == 1) {
            v[s] = DCT ? cscale<T>(val, -qx * qx) : mk<T>(-qx * val.y, qx * val.x);
          } else {  // Neumann: the pair holds kz and kz + 1
            const T d0 = qx * qx + qy * qy + qz0 * qz0 - q02;
            const T d1 = DCT ? qx * qx + qy * qy + qz1 * qz1 - q02 : d0;
            v[s] = mk<T>(alpha * d0 * d0 * val.x, alpha * d1 * d1 * val.y);
          }
        }
      }
      Ops::inverse(v, x, t, tw, true);
      Ops::store(v, outs[o] + line, t);
    }
  }

  if (want_energy && (MODE == kPencilStepGen || MODE == kPencilStepU64Gen || MODE == kPencilStepAdvGen ||
                      MODE == kPencilEnergy)) {
    const double tot = block_sum(acc.s, scratch);
    if (threadIdx.x == 0) a.red[size_t(rep) * gridDim.x + blockIdx.x] = tot;
  }
}

// src[rep][r][c] -> dst[rep][c - c0][r] of complex values, the columns c0 <= c <
// c0 + 16 gridDim.x: the checkpoint file keeps W as [f][kx], the device as [kx][f]
template <typename T>
__global__ void transpose_kernel(const cplx<T>* __restrict__ src, cplx<T>* __restrict__ dst, int rows, int cols,
                                 int c0) {
  __shared__ cplx<T> tile[16][17];
  const int c = blockIdx.x * 16 + threadIdx.x, r = blockIdx.y * 16 + threadIdx.y;
  tile[threadIdx.y][threadIdx.x] = src[(size_t(blockIdx.z) * rows + r) * cols + c0 + c];
  __syncthreads();
  const int c2 = blockIdx.x * 16 + threadIdx.y, r2 = blockIdx.y * 16 + threadIdx.x;
  dst[(size_t(blockIdx.z) * gridDim.x * 16 + c2) * rows + r2] = tile[threadIdx.x][threadIdx.y];
}

}  // namespace shb
