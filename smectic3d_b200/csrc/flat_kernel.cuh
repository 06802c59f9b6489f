// Plane pass of a plane that fits one SM (32^2 to 128^2): one CTA per x-plane.
//
// The modes and their arguments are those of plane_kernel.cuh; the transforms run
// in the lane-per-line form of line_fft.cuh.  In the column stage lanes are
// columns, so a warp reads and writes whole rows of the plane straight from and to
// global memory; in the row stage the G lanes of a row pair are neighbours and
// exchange inside their warp.  One buffer serves the column exchange, the row pairs
// and the row exchanges (a row pair is its own scratch), so shared memory holds the
// plane once.  Rows are packed two by two (2 p, 2 p + 1) as in plane_kernel.cuh, one
// after the other in the pair, so psi and the gradients of FP32 (and periodic FP64)
// runs are bit for bit those of that kernel.  Pairs of rows p and p + N / 2, which a
// periodic column holds in one thread and can store as 16 bytes, round every step
// otherwise and gain nothing: 64 x 64^3 FP32 step 95.8 us, 93.2 with neighbours;
// 128^3 FP64 27.7, 26.4; 128^3 FP32 15.1, 15.4.
#pragma once
#include "plane_stages.cuh"

namespace shb {

template <typename T, int N, bool DCT>
struct FlatCfg {
  using I = LineIdx<N>;
  static constexpr int E = I::E, G = I::G;
  static constexpr int THREADS = (N / 2) * G;
  static constexpr int FP = DCT ? N * (N / 2) : N * (N / 2 + 1);
  // padded row pair: room for the warp exchange, and the lines of a half-warp on
  // different banks (G = 4: four lines, a stride of 4 mod 16; G = 8: two, 8 mod 16)
  static constexpr int LS = (warp_line<N>() + 15) / 16 * 16 + (G == 4 ? 4 : 8);
  static constexpr size_t ROWS = size_t(N / 2) * LS, COLS = size_t(N) * (N / 2);
  static constexpr size_t PK_OFF = (ROWS > COLS ? ROWS : COLS) * sizeof(cplx<T>);
  // the packed kz = 0 / N/2 column of the periodic box
  static constexpr size_t RED_OFF = PK_OFF + (DCT ? 0 : size_t(N) * sizeof(cplx<T>));
  static constexpr size_t SMEM = RED_OFF + 16 * sizeof(double);
  static constexpr bool ok = N >= 32 && N <= 128 && THREADS % 32 == 0 && THREADS <= 512 && SMEM <= size_t(227) * 1024;
  // register budget of the step: 768 threads per SM in FP32 (80 registers), 512 in FP64
  static constexpr int STEP_THREADS = sizeof(T) == 4 ? 768 : 512;
  static constexpr int MIN_BLOCKS = THREADS <= STEP_THREADS ? STEP_THREADS / THREADS : 1;
};

// What bounds it: 64 x 64^3 FP32 the shared-memory pipe (79 % busy, 12 moves of the
// plane; 51 us for 134 MB), 128^3 FP64 its barriers and the one CTA of 16 warps that
// an SM holds (22 us).  The step's plane pass, event to event, plane_kernel -> now:
// 64 x 64^3 FP32 periodic 84.1 -> 52.0 us, Neumann 98.5 -> 56.9; periodic 128^3 FP32
// 20.5 -> 14.3, FP64 26.5 -> 22.2.
template <typename T, int N, bool DCT, int MODE>
__global__ void __launch_bounds__(FlatCfg<T, N, DCT>::THREADS,
                                  MODE == kPlaneStepLean || MODE == kPlaneStepHist || MODE == kPlaneAdj
                                      ? FlatCfg<T, N, DCT>::MIN_BLOCKS
                                      : 1)
flat_kernel(const __grid_constant__ PlaneLaunch<T> pl) {
  const PlaneArgs<T>& a = pl.c[plane_multi(MODE) ? blockIdx.z : 0];
  using Cfg = FlatCfg<T, N, DCT>;
  using S = PlaneStages<T, N, DCT>;
  using Ops = PlaneOps<T, N, 1, DCT>;
  using Access = typename S::Planar;
  constexpr int E = Cfg::E, G = Cfg::G, LS = Cfg::LS, NC = N / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T>* buf = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* pk = reinterpret_cast<cplx<T>*>(smem_raw + Cfg::PK_OFF);
  double* scratch = reinterpret_cast<double*>(smem_raw + Cfg::RED_OFF);
  // column stage
  const int c = threadIdx.x % NC, ct = threadIdx.x / NC;
  const TileExchange<T, NC> cx{buf + c};
  const ColTables<T, N> ctw(a.lt, ct);
  // row stage
  const int p = threadIdx.x / G, rt = threadIdx.x % G;
  cplx<T>* row = buf + p * LS;
  const WarpExchange<T> rx{row};
  const RowTables<T, N> rtw(a.lt, rt);
  const int x = blockIdx.x, rep = blockIdx.y;
  const size_t plane_off = (size_t(rep) * N + x) * Cfg::FP;
  const int ya = 2 * p, yb = 2 * p + 1;
  const size_t ra = ((size_t(rep) * N + x) * N + ya) * N, rb = ((size_t(rep) * N + x) * N + yb) * N;
  cplx<T> v[E];
  grid_dependency_wait();

  // partial spectrum (times ``mult``; plus plane2 times mult2) -> row pairs in buf;
  // ``busy``: other threads may still be using buf
  auto columns_in = [&](const cplx<T>* __restrict__ plane, int mult, const cplx<T>* __restrict__ plane2, int mult2,
                        bool busy) {
    constexpr bool MULT = MODE == kPlaneInvReal || MODE == kPlaneInvMulFwd;
    auto value = [&](int ky, int kz) -> cplx<T> {
      const size_t off = kz == N / 2 && !DCT ? size_t(N * NC + ky) : size_t(ky) * NC + kz;
      if constexpr (MULT) {
        const size_t o1 = mult == kMulSinDy ? size_t((N - ky) & (N - 1)) * NC + kz : off;  // reversed rows for d/dy
        cplx<T> u = Ops::apply_mult(plane[o1], mult, a.q, ky, kz);
        if (plane2) u = cadd<T>(u, Ops::apply_mult(plane2[off], mult2, a.q, ky, kz));
        return u;
      } else {
        return plane[off];
      }
    };
#pragma unroll
    for (int s = 0; s < E; ++s) v[s] = value(S::ky_of(ct, s), c);
    if constexpr (!DCT) {
      // Hermitian projection in ky of the kz = 0 and kz = N/2 columns (the real part
      // FFTW's c2r keeps on those planes), packed as F0 + i FN, one ky per thread
      if (threadIdx.x < N) {
        const int ky = threadIdx.x, km = (N - ky) & (N - 1);
        const cplx<T> a0 = value(ky, 0), a1 = value(km, 0), b0 = value(ky, N / 2), b1 = value(km, N / 2);
        const T f0x = T(0.5) * (a0.x + a1.x), f0y = T(0.5) * (a0.y - a1.y);
        const T fnx = T(0.5) * (b0.x + b1.x), fny = T(0.5) * (b0.y - b1.y);
        pk[ky] = mk<T>(f0x - fny, f0y + fnx);
      }
      __syncthreads();
      busy = false;
      if (c == 0) {
#pragma unroll
        for (int s = 0; s < E; ++s) v[s] = pk[S::ky_of(ct, s)];
      }
    }
    S::col_inverse(v, ct, cx, ctw, busy, false, [](int) { return cplx<T>(); });
    __syncthreads();  // every line has left the exchange
    S::to_planar(v, ct, buf, c, LS);
    __syncthreads();
  };
  // rows on the A side -> partial spectrum
  auto rows_out = [&](cplx<T>* __restrict__ plane, bool busy) {
    S::row_forward(v, rt, row, rx, rtw, busy, [&] { rx.sync(); }, Access());
    __syncthreads();
    S::from_planar(v, ct, buf, c, LS);
    S::col_forward(v, ct, cx, ctw, true, false, [](int, cplx<T>) {});
    if (DCT || c > 0) {
#pragma unroll
      for (int s = 0; s < E; ++s) plane[S::ky_of(ct, s) * NC + c] = v[s];
    } else {
#pragma unroll
      for (int s = 0; s < E; ++s) pk[S::ky_of(ct, s)] = v[s];
    }
    if constexpr (!DCT) {
      __syncthreads();
      if (threadIdx.x < N) {  // unpack F0 + i FN, one ky per thread
        const int ky = threadIdx.x;
        const cplx<T> z = pk[ky], zm = pk[(N - ky) & (N - 1)];
        plane[ky * NC] = mk<T>(T(0.5) * (z.x + zm.x), T(0.5) * (z.y - zm.y));
        plane[N * NC + ky] = mk<T>(T(0.5) * (z.y + zm.y), T(0.5) * (zm.x - z.x));
      }
    }
  };
  auto rows_in = [&] {
    if constexpr (MODE == kPlaneInvReal && DCT) {
      S::row_inverse(v, rt, row, rx, rtw, true, typename S::SinDz{a.sin_dz ? a.q : nullptr});
    } else {
      S::row_inverse(v, rt, row, rx, rtw, true, Access());
    }
  };

  if constexpr (MODE == kPlaneStepLean || MODE == kPlaneStepHist) {
    columns_in(a.src + plane_off, kMulNone, nullptr, kMulNone, false);
    rows_in();
    if constexpr (MODE == kPlaneStepHist) S::real_store(v, rt, a.real_out, ra, rb);
    S::nonlin(v, a.pp);
    rows_out(a.dst + plane_off, true);
  } else if constexpr (MODE == kPlaneStep || MODE == kPlaneGetPsi || MODE == kPlaneInvReal || MODE == kPlaneAdj ||
                       MODE == kPlaneInvMulFwd) {
    columns_in(a.src + plane_off, a.mult, a.src2 ? a.src2 + plane_off : nullptr, a.mult2, false);
    rows_in();
    if constexpr (MODE == kPlaneInvReal) {
      if (a.sign_axes) {  // the sine transforms' real-space signs
#pragma unroll
        for (int s = 0; s < E; ++s) {
          const int z = S::z_of(rt, s);
          v[s] = mk<T>(axis_sign<T>(a.sign_axes, x, ya, z) * v[s].x, axis_sign<T>(a.sign_axes, x, yb, z) * v[s].y);
        }
      }
    }
    if (a.flags & (kFlPsiOut | kFlL1 | kFlEnergy))
      S::monitor(v, rt, a.flags, a.pp, rep, ra, rb, a.psi_old, a.psi_out,
                 a.red + (size_t(rep) * gridDim.x + blockIdx.x) * 3, scratch);
    if (MODE == kPlaneInvReal && a.real_zn > 0) {
      // only the planes z < real_zn, compact
      const int zn = a.real_zn;
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const int z = S::z_of(rt, s);
        if (z < zn) {
          a.real_out[(ra / N) * zn + z] = v[s].x;
          a.real_out[(rb / N) * zn + z] = v[s].y;
        }
      }
    } else if (MODE == kPlaneInvReal || MODE == kPlaneInvMulFwd || (MODE == kPlaneStep && (a.flags & kFlRealOut))) {
      S::real_store(v, rt, a.real_out, ra, rb);
    }
    if constexpr (MODE == kPlaneAdj) {
      // g^n = N'(psi^n) (c_n mu^{n+1} - mu^{n+2}); v holds the bracket (its
      // partial is what the pencil pass of step n+1 emitted)
      const T beta = T(a.pp.beta), gamma = T(a.pp.gamma);
      const T* psi = a.real_in[1];
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const int z = S::z_of(rt, s);
        v[s] = mk<T>(nonlin_deriv<T>(psi[ra + z], beta, gamma, a.pp.nonlin) * v[s].x,
                     nonlin_deriv<T>(psi[rb + z], beta, gamma, a.pp.nonlin) * v[s].y);
      }
    }
    if constexpr (MODE == kPlaneInvMulFwd) {
      // stress component S_c = (L psi) d_c psi (periodicFFT/pf3d.cpp:417-429), formed
      // from the derivative just written and sent forward in the same pass
      const T* f = a.real_in[0];
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const int z = S::z_of(rt, s);
        v[s] = mk<T>(v[s].x * f[ra + z], v[s].y * f[rb + z]);
      }
    }
    if constexpr (MODE == kPlaneStep) S::nonlin_penalties(v, rt, rx, a.pp, a.wall, a.lperp, a.kwall, ra, rb);
    if constexpr (MODE == kPlaneStep || MODE == kPlaneAdj || MODE == kPlaneInvMulFwd) rows_out(a.dst + plane_off, true);
  } else if constexpr (MODE == kPlaneAdvN) {
    // N = beta psi^3 - gamma psi^5 (+ pinning) - u . grad psi (periodicFFT/pf3d.cpp:455-467):
    // the velocity components come in as partials and are inverted here one
    // after the other, u_c d_c psi accumulating in registers
    cplx<T> acc[E];
#pragma unroll
    for (int s = 0; s < E; ++s) acc[s] = mk<T>(T(0), T(0));
#pragma unroll 1
    for (int comp = 0; comp < 3; ++comp) {
      columns_in(a.src3[comp] + plane_off, kMulNone, nullptr, kMulNone, comp > 0);
      rows_in();
      const T* d = a.real_in[1 + comp];
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const int z = S::z_of(rt, s);
        // Neumann: the partials carry (-1)^(x+y+z) u
        const T sa = axis_sign<T>(a.sign_axes, x, ya, z), sb = axis_sign<T>(a.sign_axes, x, yb, z);
        acc[s].x = fma(sa * v[s].x, d[ra + z], acc[s].x);
        acc[s].y = fma(sb * v[s].y, d[rb + z], acc[s].y);
      }
    }
    const T beta = T(a.pp.beta), gamma = T(a.pp.gamma);
    const T cpen = T(2.0 * a.pp.w_mid * a.pp.inv_dz2);
    const T* ps = a.real_in[0];
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int z = S::z_of(rt, s);
      const size_t ia = ra + z, ib = rb + z;
      const T pa = ps[ia], pb = ps[ib];
      T oa = nonlin_eval<T>(pa, beta, gamma, a.pp.nonlin);
      T ob = nonlin_eval<T>(pb, beta, gamma, a.pp.nonlin);
      if (a.pp.w_mid != 0.0 && z == N / 2) {
        oa += cpen * (ps[ia - 1] - T(2) * pa + ps[ia + 1]);
        ob += cpen * (ps[ib - 1] - T(2) * pb + ps[ib + 1]);
      }
      v[s] = mk<T>(oa - acc[s].x, ob - acc[s].y);
    }
    rows_out(a.dst + plane_off, true);
  } else if constexpr (MODE == kPlaneMulFwd) {
    // stress component S_c = (L psi) d_c psi of the Neumann Stokes solve
    // (cosFFT/comet/morphSurfK.cpp:760-770), signed for the sine transform
    const T* f0 = a.real_in[0];
    const T* f1 = a.real_in[1];
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int z = S::z_of(rt, s);
      const T sa = axis_sign<T>(a.sign_axes, x, ya, z), sb = axis_sign<T>(a.sign_axes, x, yb, z);
      v[s] = mk<T>(sa * f0[ra + z] * f1[ra + z], sb * f0[rb + z] * f1[rb + z]);
    }
    rows_out(a.dst + plane_off, false);
  } else {  // kPlaneInit: real psi -> partial spectra of psi (dst2) and N(psi) (dst)
    const T beta = T(a.pp.beta), gamma = T(a.pp.gamma);
    const T cw = T(2.0 * a.pp.w_mid * a.pp.inv_dz2);
#pragma unroll 1
    for (int field = 0; field < 2; ++field) {
      if (field > 0) __syncthreads();
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const int z = S::z_of(rt, s);
        T pa = T(a.psi_in[ra + z]), pb = T(a.psi_in[rb + z]);
        if (field == 1) {
          T na = nonlin_eval<T>(pa, beta, gamma, a.pp.nonlin);
          T nb = nonlin_eval<T>(pb, beta, gamma, a.pp.nonlin);
          if (a.pp.w_mid != 0.0 && z == N / 2) {
            na += cw * (T(a.psi_in[ra + z - 1]) - T(2) * pa + T(a.psi_in[ra + z + 1]));
            nb += cw * (T(a.psi_in[rb + z - 1]) - T(2) * pb + T(a.psi_in[rb + z + 1]));
          }
          if (z < a.kwall) {  // substrate penalty of psi^0
            na += a.wall[z] * a.lperp[(ra / N) * a.kwall + z];
            nb += a.wall[z] * a.lperp[(rb / N) * a.kwall + z];
          }
          pa = na;
          pb = nb;
        }
        v[s] = mk<T>(pa, pb);
      }
      rows_out((field == 0 ? a.dst2 : a.dst) + plane_off, false);
    }
  }
}

}  // namespace shb
