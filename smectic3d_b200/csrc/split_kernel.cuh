// The plane pass of large planes as three one-axis passes.
//
// A 256 x 256 or larger plane does not fit one SM, and a cluster that shares it
// moves 7/8 of two fields between SMs per pass (3.3 TB/s of bulk copies, 2.6 with
// clusters of 16).  Here each axis is a pass of its own over a slab of planes:
//
//   ycol_kernel (inverse)   partial spectra [x][ky][c] -> slab
//   zrow_kernel             slab in place: inverse z, the real-space work, forward z
//   ycol_kernel (forward)   slab -> partial spectra [x][ky][c]
//
// The slab is small enough to live in the 126 MB L2, so HBM still sees each field
// once; it holds row pairs (plane_stages.cuh).
#pragma once
#include "plane_stages.cuh"

namespace shb {

// threads per SM the register budgets aim at (as PencilCfg::step_threads)
template <typename T, int N>
__host__ __device__ constexpr int split_threads() {
  return sizeof(T) == 4 ? 512 : 256;
}

template <typename T, int N, bool DCT>
struct YcolCfg {
  using I = LineIdx<N>;
  static constexpr int E = I::E, G = I::G;
  static constexpr int TK = sizeof(T) == 4 ? 16 : 8;  // 128-byte row segments
  static constexpr int THREADS = TK * G;
  static constexpr int TILES = N / 2 / TK;
  static constexpr int FP = DCT ? N * (N / 2) : N * (N / 2 + 1);
  static constexpr int SP = N * (N / 2);  // slab plane
  static constexpr size_t SMEM = size_t(TK) * N * sizeof(cplx<T>);
  static constexpr int MIN_BLOCKS = split_threads<T, N>() / THREADS;
};

constexpr int kSplitComps = 4;  // fields one launch takes (blockIdx.y)
template <typename T>
struct YcolArgs {
  const cplx<T>* src[kSplitComps];  // inverse: partial spectra of the slab's first plane; forward: the slab
  cplx<T>* dst[kSplitComps];        // inverse: the slab; forward: partial spectra of the slab's first plane
  const cplx<T>* lt;                // line tables
  const T* q;                       // wavenumbers (only for iqy)
  int iqy;                          // inverse: the field that is multiplied by i q_y on the way (-1: none)
};

// y transform of TK columns of one plane.  blockIdx.x = plane * TILES + tile,
// blockIdx.y = field.
// Bound by the latency of its loads at 16 warps per SM (issue slots 46 % busy,
// shared-memory pipe 15 %): Neumann 256^3 FP32 24 us for 134 MB, of which one
// field is in L2.  16 columns keep every access whole 128-byte segments while four
// CTAs of 32 KB fit an SM.
template <typename T, int N, bool DCT, bool INV, bool IQY = false>
__global__ void __launch_bounds__(YcolCfg<T, N, DCT>::THREADS, YcolCfg<T, N, DCT>::MIN_BLOCKS)
ycol_kernel(const __grid_constant__ YcolArgs<T> a) {
  using Cfg = YcolCfg<T, N, DCT>;
  using S = PlaneStages<T, N, DCT>;
  constexpr int E = Cfg::E, TK = Cfg::TK;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int c = threadIdx.x % TK, t = threadIdx.x / TK;
  const int tile = blockIdx.x % Cfg::TILES, plane = blockIdx.x / Cfg::TILES;
  const int col = tile * TK + c;
  const TileExchange<T, TK> x{reinterpret_cast<cplx<T>*>(smem_raw) + c};
  const ColTables<T, N> tw(a.lt, t);
  const bool packed = !DCT && tile == 0 && c == 0;  // the kz = 0 column carries kz = N/2 too
  cplx<T> v[E];
  grid_dependency_wait();
  const int f = blockIdx.y;
  if constexpr (INV) {
    const cplx<T>* src = a.src[f] + size_t(plane) * Cfg::FP;
#pragma unroll
    for (int s = 0; s < E; ++s) v[s] = src[S::ky_of(t, s) * (N / 2) + col];
    if constexpr (IQY) {
      const bool on = f == a.iqy;
      if (on) {
#pragma unroll
        for (int s = 0; s < E; ++s) {
          const T q = __ldg(&a.q[S::ky_of(t, s)]);
          v[s] = mk<T>(-q * v[s].y, q * v[s].x);
        }
      }
      S::col_inverse(v, t, x, tw, false, packed, [&](int ky) {
        const cplx<T> n = src[N * (N / 2) + ky];
        const T q = __ldg(&a.q[ky]);
        return on ? mk<T>(-q * n.y, q * n.x) : n;
      });
    } else {
      S::col_inverse(v, t, x, tw, false, packed, [&](int ky) { return src[N * (N / 2) + ky]; });
    }
    S::to_pairs(v, t, a.dst[f] + size_t(plane) * Cfg::SP + 2 * col, N);
  } else {
    S::from_pairs(v, t, a.src[f] + size_t(plane) * Cfg::SP + 2 * col, N);
    cplx<T>* dst = a.dst[f] + size_t(plane) * Cfg::FP;
    S::col_forward(v, t, x, tw, false, packed, [&](int ky, cplx<T> z) { dst[N * (N / 2) + ky] = z; });
#pragma unroll
    for (int s = 0; s < E; ++s) dst[S::ky_of(t, s) * (N / 2) + col] = v[s];
  }
}

template <typename T, int N, bool DCT>
struct ZrowCfg {
  using I = LineIdx<N>;
  static constexpr int E = I::E, G = I::G;
  static constexpr int THREADS = sizeof(T) == 4 ? 128 : 64;
  static constexpr int LINES = THREADS / G;  // row pairs per CTA
  static constexpr int BLOCKS = N / 2 / LINES;  // CTAs per plane
  static constexpr int SP = N * (N / 2);
  // padded line; the + 8 puts the two lines of a half-warp on different banks
  static constexpr int LS = warp_line<N>() + 8;
  static constexpr size_t RED_OFF = size_t(LINES) * LS * sizeof(cplx<T>);
  static constexpr size_t KEEP_OFF = RED_OFF + 16 * sizeof(double);  // one value per slot and thread kept aside
  static constexpr size_t smem(int mode) {
    return KEEP_OFF + (mode == 3 || mode == 5 ? size_t(E) * THREADS * sizeof(cplx<T>) : 0);
  }
  // CTAs per SM the register budget aims at.  FP32: four (128 registers); three
  // where they spill, the Neumann step (256^3 step 135.4 -> 131.9 us) and the passes
  // over several fields, whose shared memory holds three.
  static constexpr int min_blocks(int mode) {
    if (mode == 1 || (sizeof(T) == 8 && mode > 1)) return 0;  // kZrowGen: as many registers as it takes
    return sizeof(T) == 4 && (DCT || mode > 1) ? 3 : split_threads<T, N>() / THREADS;
  }
};

enum ZrowMode : int {
  kZrowStep = 0,    // N(psi) alone
  kZrowGen = 1,     // also the penalties, psi out and the monitors (PassFlags)
  kZrowReal = 2,    // slab[f] -> real_to[f] (field 0 with the monitors and psi out), no way back
  kZrowStress = 3,  // periodic advection: psi, L psi, grad psi to real space and (L psi) d_c psi forward
  kZrowMul = 4,     // real_in[f] real_in[3] (signed for the sine transform) forward -> slab[f]
  kZrowAdvN = 5,    // N(real_in[3]) - sum_c u_c real_in[c], the velocity from slab[c]; forward -> slab[0]
  kZrowInit = 6,    // real psi (FP64) forward -> slab[0], N(psi) forward -> slab[1]
};

template <typename T>
struct ZrowArgs {
  cplx<T>* slab[kSplitComps];
  const cplx<T>* lt;
  PointParams pp;
  const T* real_in[kSplitComps];
  T* real_to[kSplitComps];
  const T* q;
  int sign_axes;          // axis_sign of the real-space factors
  // kZrowGen, kZrowReal, kZrowStress
  int flags, plane0;      // first plane of the slab, rep * N + x
  const double* psi_in;   // kZrowInit
  double* psi_out;
  const double* psi_old;
  double* red;            // per-CTA partial sums [plane][BLOCKS][3]
  T* real_out;
  const T* wall;          // substrate penalty (PlaneArgs)
  const T* lperp;
  int kwall;
};

// The three passes against the clustered kernel: Neumann 256^3 FP32 113 -> 80 us,
// periodic 94 -> 71, Neumann 256^3 FP64 262 -> 183, 512^3 FP64 5408 -> 1578.  The z
// pass is the longest (36 us Neumann 256^3 FP32): two transforms and the pointwise
// work, 19.7 M warp instructions, issue slots 55 % busy.
//
// z transforms of LINES row pairs around the real-space work.  G consecutive
// lanes own a line and exchange inside their warp: no block barrier, every warp
// runs on its own.  blockIdx.x = plane * BLOCKS + block.
template <typename T, int N, bool DCT, int MODE>
__global__ void __launch_bounds__(ZrowCfg<T, N, DCT>::THREADS,
                                  ZrowCfg<T, N, DCT>::min_blocks(MODE))
zrow_kernel(const __grid_constant__ ZrowArgs<T> a) {
  using Cfg = ZrowCfg<T, N, DCT>;
  using S = PlaneStages<T, N, DCT>;
  constexpr int E = Cfg::E, G = Cfg::G;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int line = threadIdx.x / G, t = threadIdx.x % G;
  cplx<T>* L = reinterpret_cast<cplx<T>*>(smem_raw) + line * Cfg::LS;
  const WarpExchange<T> x{L};
  const RowTables<T, N> tw(a.lt, t);
  const int plane = blockIdx.x / Cfg::BLOCKS;
  const int p = (blockIdx.x % Cfg::BLOCKS) * Cfg::LINES + line;
  const size_t row_off = size_t(plane) * Cfg::SP + p * N;
  const int gp = a.plane0 + plane;  // rep * N + x
  const int ya = real_pos<N, DCT>(p), yb = real_pos<N, DCT>(p + N / 2);
  const size_t ra = (size_t(gp) * N + ya) * N, rb = (size_t(gp) * N + yb) * N;
  cplx<T> v[E];
  grid_dependency_wait();
  auto monitor = [&] {
    if (a.flags & (kFlPsiOut | kFlL1 | kFlEnergy))
      S::monitor_line(v, t, x, a.flags, a.pp, gp / N, ra, rb, a.psi_old, a.psi_out,
                      a.red + (size_t(gp) * Cfg::BLOCKS + blockIdx.x % Cfg::BLOCKS) * 3,
                      reinterpret_cast<double*>(smem_raw + Cfg::RED_OFF));
  };
  cplx<T>* keep = reinterpret_cast<cplx<T>*>(smem_raw + Cfg::KEEP_OFF) + threadIdx.x;
  if constexpr (MODE == kZrowStep || MODE == kZrowGen) {
    cplx<T>* row = a.slab[0] + row_off;
    S::row_inverse(v, t, row, x, tw, false, typename S::Plain());
    if constexpr (MODE == kZrowGen) {
      monitor();
      if (a.flags & kFlRealOut) S::real_store(v, t, a.real_out, ra, rb);
    }
    if (MODE == kZrowGen && (a.pp.w_mid != 0.0 || a.kwall > 0))
      S::nonlin_penalties(v, t, x, a.pp, a.wall, a.lperp, a.kwall, ra, rb);
    else
      S::nonlin(v, a.pp);
    S::row_forward(v, t, row, x, tw, true, [] {}, typename S::Plain());
  } else if constexpr (MODE == kZrowReal) {
    const int f = blockIdx.y;
    S::row_inverse(v, t, a.slab[f] + row_off, x, tw, false, typename S::Plain());
    if (f == 0) monitor();
    if (a.real_to[f]) S::real_store(v, t, a.real_to[f], ra, rb);
  } else if constexpr (MODE == kZrowInit) {
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int z = S::z_of(t, s);
      v[s] = mk<T>(T(a.psi_in[ra + z]), T(a.psi_in[rb + z]));
    }
    if (blockIdx.y == 1) S::nonlin_penalties(v, t, x, a.pp, a.wall, a.lperp, a.kwall, ra, rb);
    S::row_forward(v, t, a.slab[blockIdx.y] + row_off, x, tw, true, [] {}, typename S::Plain());
  } else if constexpr (MODE == kZrowMul) {
    // stress component S_c = (L psi) d_c psi of the Neumann Stokes solve
    // (cosFFT/comet/morphSurfK.cpp:760-770), signed for the sine transform
    const int f = blockIdx.y;
    const T *f0 = a.real_in[3], *f1 = a.real_in[f];
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int z = S::z_of(t, s);
      const T sa = axis_sign<T>(a.sign_axes, gp % N, ya, z), sb = axis_sign<T>(a.sign_axes, gp % N, yb, z);
      v[s] = mk<T>(sa * f0[ra + z] * f1[ra + z], sb * f0[rb + z] * f1[rb + z]);
    }
    S::row_forward(v, t, a.slab[f] + row_off, x, tw, false, [] {}, typename S::Plain());
  } else if constexpr (MODE == kZrowStress && !DCT) {
    // slabs: psi, d_x psi, d_y psi, L psi.  L psi stays aside in shared memory while
    // each gradient component is inverted, written out and sent forward as the
    // stress S_c = (L psi) d_c psi (periodicFFT/pf3d.cpp:404-429); d_z psi is i q_z
    // times psi's own rows.  The stress components replace slabs 1, 2 and 0.  One
    // loop body for all five inverses: with three copies of the transform the warps
    // waited for instructions (2.5 of 8 cycles per issue).
#pragma unroll 1
    for (int i = 0; i < 5; ++i) {  // L psi, psi, d_x, d_y, d_z
      cplx<T>* row = a.slab[i == 0 ? 3 : (i == 2 || i == 3 ? i - 1 : 0)] + row_off;
      S::row_inverse(v, t, row, x, tw, true, typename S::Dz{i == 4 ? a.q : nullptr});
      if (i == 0) {
#pragma unroll
        for (int s = 0; s < E; ++s) keep[s * Cfg::THREADS] = v[s];
        continue;
      }
      if (i == 1) monitor();
      S::real_store(v, t, a.real_to[i == 1 ? 3 : i - 2], ra, rb);
      if (i == 1) continue;
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const cplx<T> l = keep[s * Cfg::THREADS];
        v[s] = mk<T>(v[s].x * l.x, v[s].y * l.y);
      }
      S::row_forward(v, t, row, x, tw, true, [] {}, typename S::Plain());
    }
  } else if constexpr (MODE == kZrowAdvN) {
    // N = beta psi^3 - gamma psi^5 (+ pinning) - u . grad psi (periodicFFT/pf3d.cpp:455-467)
#pragma unroll
    for (int s = 0; s < E; ++s) keep[s * Cfg::THREADS] = mk<T>(T(0), T(0));
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
      S::row_inverse(v, t, a.slab[c] + row_off, x, tw, c > 0, typename S::Plain());
      const T* d = a.real_in[c];
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const int z = S::z_of(t, s);
        // Neumann: the partials carry (-1)^(x+y+z) u
        const T sa = axis_sign<T>(a.sign_axes, gp % N, ya, z), sb = axis_sign<T>(a.sign_axes, gp % N, yb, z);
        const cplx<T> o = keep[s * Cfg::THREADS];
        keep[s * Cfg::THREADS] = mk<T>(fma(sa * v[s].x, d[ra + z], o.x), fma(sb * v[s].y, d[rb + z], o.y));
      }
    }
    const T beta = T(a.pp.beta), gamma = T(a.pp.gamma);
    const T cpen = T(2.0 * a.pp.w_mid * a.pp.inv_dz2);
    const T* ps = a.real_in[3];
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int z = S::z_of(t, s);
      const size_t ia = ra + z, ib = rb + z;
      const T pa = ps[ia], pb = ps[ib];
      T oa = nonlin_eval<T>(pa, beta, gamma, a.pp.nonlin);
      T ob = nonlin_eval<T>(pb, beta, gamma, a.pp.nonlin);
      if (a.pp.w_mid != 0.0 && z == N / 2) {
        oa += cpen * (ps[ia - 1] - T(2) * pa + ps[ia + 1]);
        ob += cpen * (ps[ib - 1] - T(2) * pb + ps[ib + 1]);
      }
      const cplx<T> acc = keep[s * Cfg::THREADS];
      v[s] = mk<T>(oa - acc.x, ob - acc.y);
    }
    S::row_forward(v, t, a.slab[0] + row_off, x, tw, true, [] {}, typename S::Plain());
  }
}

}  // namespace shb
