// Column (y) and row (z) stages of one x-plane in registers (line_fft.cuh), shared
// by the one-CTA plane pass (flat_kernel.cuh) and the split passes
// (split_kernel.cuh).
//
// Between the stages a plane is kept as row pairs, which is what the z stage packs
// into one complex line.  In the split passes' slab:
//   [p][2 c + h], p < N/2, rows real_pos(p) and real_pos(p + N/2)
//   periodic: h = 0, 1: kz = c of either row (kz = 0 carries F0 + i FN)
//   Neumann : z = 2 c + h, as (first row, second row)
// A column thread ends with both rows of a pair in registers, so a pair of columns
// moves as one 16-byte access (32 in FP64).  The one-CTA pass keeps rows 2 p and
// 2 p + 1, one after the other (Planar).
#pragma once
#include "line_fft.cuh"
#include "plane_kernel.cuh"

namespace shb {

// two consecutive complex values
__device__ __forceinline__ void ld2(const float2* p, float2& a, float2& b) { ld_pair(p, a, b); }
__device__ __forceinline__ void st2(float2* p, float2 a, float2 b) { st_pair(p, a, b); }
__device__ __forceinline__ void ld2(const double2* p, double2& a, double2& b) {
  a = p[0];
  b = p[1];
}
__device__ __forceinline__ void st2(double2* p, double2 a, double2 b) {
  p[0] = a;
  p[1] = b;
}

template <typename T, int N, bool DCT>
struct PlaneStages {
  using I = LineIdx<N>;
  using F = LineFFT<T, N>;
  static constexpr int E = I::E, RA = I::RA, NA = I::NA;

  // wavenumber of B-side slot s between a column's pre- / post-processing and memory
  static __device__ __forceinline__ int ky_of(int t, int s) { return DCT ? I::c_slot(t, s) : I::b_elem(t, s); }

  // ---- column stage, inverse: v at ky_of -> A side.  ``packed``: this is the
  // periodic kz = 0 column, nyq(ky) reads the kz = N/2 column
  template <class X, class Tab, class Nyq>
  static __device__ __forceinline__ void col_inverse(cplx<T> (&v)[E], int t, const X& x, const Tab& tw, bool first_sync,
                                                     bool packed, Nyq nyq) {
    if constexpr (DCT) {
      F::dct3_pre(v, t, tw);
      F::uncanon(v, t);
    } else if (packed) {
      // Hermitian projection in ky of the kz = 0 and kz = N/2 columns (the real part
      // FFTW's c2r keeps on those planes), packed as F0 + i FN
      F::canon(v, t);
#pragma unroll
      for (int s = 0; s < E / 2; ++s) {
        cplx<T>&lo = v[s], &hi = v[E - 1 - s];
        const cplx<T> nl = nyq(I::c_elem(t, s)), nh = nyq(I::c_mirror(t, s));
        if (s == 0 && t == 0) {  // ky = 0 and ky = N/2 are their own mirrors
          lo = mk<T>(lo.x, nl.x);
          hi = mk<T>(hi.x, nh.x);
        } else {
          const T f0x = T(0.5) * (lo.x + hi.x), f0y = T(0.5) * (lo.y - hi.y);
          const T fnx = T(0.5) * (nl.x + nh.x), fny = T(0.5) * (nl.y - nh.y);
          lo = mk<T>(f0x - fny, f0y + fnx);
          hi = mk<T>(f0x + fny, fnx - f0y);
        }
      }
      F::uncanon(v, t);
    }
    F::inverse(v, t, x, tw, first_sync);
  }
  // A side -> row pairs; dst = pair 0, column 0 of this thread's column pair, rows
  // ``ld`` elements apart
  static __device__ __forceinline__ void to_pairs(const cplx<T> (&v)[E], int t, cplx<T>* dst, int ld) {
#pragma unroll
    for (int g = 0; g < NA; ++g)
#pragma unroll
      for (int r = 0; r < RA / 2; ++r) {
        const cplx<T> p = v[g * RA + r], q = v[g * RA + r + RA / 2];
        cplx<T>* d = dst + I::a_elem(t, g * RA + r) * ld;
        if constexpr (DCT) st2(d, mk<T>(p.x, q.x), mk<T>(p.y, q.y));
        else st2(d, p, q);
      }
  }
  static __device__ __forceinline__ void from_pairs(cplx<T> (&v)[E], int t, const cplx<T>* src, int ld) {
#pragma unroll
    for (int g = 0; g < NA; ++g)
#pragma unroll
      for (int r = 0; r < RA / 2; ++r) {
        cplx<T> p, q;
        ld2(src + I::a_elem(t, g * RA + r) * ld, p, q);
        v[g * RA + r] = DCT ? mk<T>(p.x, q.x) : p;
        v[g * RA + r + RA / 2] = DCT ? mk<T>(p.y, q.y) : q;
      }
  }
  // ---- column stage, forward: A side -> v at ky_of.  ``packed``: st_nyq(ky, value)
  // stores the kz = N/2 column
  template <class X, class Tab, class Nyq>
  static __device__ __forceinline__ void col_forward(cplx<T> (&v)[E], int t, const X& x, const Tab& tw, bool first_sync,
                                                     bool packed, Nyq st_nyq) {
    F::forward(v, t, x, tw, first_sync);
    if constexpr (DCT) {
      F::canon(v, t);
      F::dct2_post(v, t, tw);
    } else if (packed) {
      // unpack F0 + i FN
      F::canon(v, t);
#pragma unroll
      for (int s = 0; s < E / 2; ++s) {
        cplx<T>&lo = v[s], &hi = v[E - 1 - s];
        cplx<T> nl, nh;
        if (s == 0 && t == 0) {
          nl = mk<T>(lo.y, T(0));
          nh = mk<T>(hi.y, T(0));
          lo = mk<T>(lo.x, T(0));
          hi = mk<T>(hi.x, T(0));
        } else {
          const cplx<T> z = lo, zm = hi;
          lo = mk<T>(T(0.5) * (z.x + zm.x), T(0.5) * (z.y - zm.y));
          hi = conjg<T>(lo);
          nl = mk<T>(T(0.5) * (z.y + zm.y), T(0.5) * (zm.x - z.x));
          nh = conjg<T>(nl);
        }
        st_nyq(I::c_elem(t, s), nl);
        st_nyq(I::c_mirror(t, s), nh);
      }
      F::uncanon(v, t);
    }
  }

  // ---- row stage: a row pair -> psi of the two rows on the A side.  ``mul`` reads
  // the pair's kz = k, in its layout and times its spectral multiplier
  template <class X, class Tab, class Mul>
  static __device__ __forceinline__ void row_inverse(cplx<T> (&v)[E], int t, const cplx<T>* row, const X& x,
                                                     const Tab& tw, bool first_sync, Mul mul) {
    if constexpr (DCT) {
#pragma unroll
      for (int s = 0; s < E; ++s) v[s] = mul(I::c_slot(t, s), row);
      F::dct3_pre(v, t, tw);
    } else {
      // Z = X_a + i X_b with Hermitian extension; kz = 0 holds (X[0], X[N/2])
#pragma unroll
      for (int s = 0; s < E / 2; ++s) {
        const int k = I::c_low(s) ? I::c_elem(t, s) : N - I::c_elem(t, s);  // < N/2
        cplx<T> A, B;
        mul.load(k, row, A, B);
        cplx<T> zk = mk<T>(A.x - B.y, A.y + B.x), zm = mk<T>(A.x + B.y, B.x - A.y);
        if (s == 0 && t == 0) {
          zk = mk<T>(A.x, B.x);
          zm = mk<T>(A.y, B.y);
        }
        v[s] = I::c_low(s) ? zk : zm;
        v[E - 1 - s] = I::c_low(s) ? zm : zk;
      }
    }
    F::uncanon(v, t);
    F::inverse(v, t, x, tw, first_sync);
  }
  // real rows on the A side -> their spectra, stored to the row pair; ``ready``
  // runs before the first store (the exchange may overlay the row)
  template <class X, class Tab, class Sync, class Put>
  static __device__ __forceinline__ void row_forward(cplx<T> (&v)[E], int t, cplx<T>* row, const X& x, const Tab& tw,
                                                     bool first_sync, Sync ready, Put put) {
    F::forward(v, t, x, tw, first_sync);
    F::canon(v, t);
    ready();
    if constexpr (DCT) {
      F::dct2_post(v, t, tw);
#pragma unroll
      for (int s = 0; s < E; ++s) put(I::c_slot(t, s), row, v[s]);
    } else {
      // split Z into the half spectra of the two rows
#pragma unroll
      for (int s = 0; s < E / 2; ++s) {
        const int k = I::c_low(s) ? I::c_elem(t, s) : N - I::c_elem(t, s);  // < N/2
        const cplx<T> z = I::c_low(s) ? v[s] : v[E - 1 - s], zm = I::c_low(s) ? v[E - 1 - s] : v[s];
        cplx<T> A = mk<T>(T(0.5) * (z.x + zm.x), T(0.5) * (z.y - zm.y));
        cplx<T> B = mk<T>(T(0.5) * (z.y + zm.y), T(0.5) * (zm.x - z.x));
        if (s == 0 && t == 0) {
          A = mk<T>(z.x, zm.x);
          B = mk<T>(z.y, zm.y);
        }
        put.store(k, row, A, B);
      }
    }
  }
  // row access of the split passes: no multiplier, (first row, second row) interleaved
  struct Plain {
    __device__ __forceinline__ cplx<T> operator()(int k, const cplx<T>* row) const { return row[k]; }
    __device__ __forceinline__ void operator()(int k, cplx<T>* row, cplx<T> z) const { row[k] = z; }
    __device__ __forceinline__ void load(int k, const cplx<T>* row, cplx<T>& A, cplx<T>& B) const {
      ld2(row + 2 * k, A, B);
    }
    __device__ __forceinline__ void store(int k, cplx<T>* row, cplx<T> A, cplx<T> B) const { st2(row + 2 * k, A, B); }
  };
  // d/dz of a periodic row when q is given: i q_z
  struct Dz {
    const T* q;
    __device__ __forceinline__ void load(int k, const cplx<T>* row, cplx<T>& A, cplx<T>& B) const {
      ld2(row + 2 * k, A, B);
      if (q) {
        // the kz = 0 slot holds the kz = 0 and N/2 columns, whose z derivatives vanish
        const T qz = k != 0 ? __ldg(&q[k]) : T(0);
        A = mk<T>(-qz * A.y, qz * A.x);
        B = mk<T>(-qz * B.y, qz * B.x);
      }
    }
  };
  // rows one after the other: N values (Neumann) or N / 2 complex values (periodic)
  // of the first row, then the second
  struct Planar {
    __device__ __forceinline__ cplx<T> operator()(int k, const cplx<T>* row) const {
      const T* f = reinterpret_cast<const T*>(row);
      return mk<T>(f[k], f[N + k]);
    }
    __device__ __forceinline__ void operator()(int k, cplx<T>* row, cplx<T> z) const {
      T* f = reinterpret_cast<T*>(row);
      f[k] = z.x;
      f[N + k] = z.y;
    }
    __device__ __forceinline__ void load(int k, const cplx<T>* row, cplx<T>& A, cplx<T>& B) const {
      A = row[k];
      B = row[N / 2 + k];
    }
    __device__ __forceinline__ void store(int k, cplx<T>* row, cplx<T> A, cplx<T> B) const {
      row[k] = A;
      row[N / 2 + k] = B;
    }
  };
  // the sine series of d/dz when q is given: coefficient k is -q_{N-k} times
  // coefficient N - k, 0 at k = 0
  struct SinDz {
    const T* q;
    __device__ __forceinline__ cplx<T> operator()(int k, const cplx<T>* row) const {
      if (!q) return Planar()(k, row);
      return k == 0 ? mk<T>(T(0), T(0)) : cscale<T>(Planar()(N - k, row), -__ldg(&q[N - k]));
    }
  };
  // A side <-> rows one after the other, row pair (2 p, 2 p + 1) at p ld; ``pairs`` =
  // pair 0, ``c`` = column (Neumann: column pair)
  static __device__ __forceinline__ cplx<T>* planar_at(cplx<T>* pairs, int t, int s, int c, int ld) {
    const int y = real_pos<N, DCT>(I::a_elem(t, s));
    return pairs + (y >> 1) * ld + (y & 1) * (N / 2) + c;
  }
  static __device__ __forceinline__ void to_planar(const cplx<T> (&v)[E], int t, cplx<T>* pairs, int c, int ld) {
#pragma unroll
    for (int s = 0; s < E; ++s) *planar_at(pairs, t, s, c, ld) = v[s];
  }
  static __device__ __forceinline__ void from_planar(cplx<T> (&v)[E], int t, cplx<T>* pairs, int c, int ld) {
#pragma unroll
    for (int s = 0; s < E; ++s) v[s] = *planar_at(pairs, t, s, c, ld);
  }

  // ---- real space: v holds psi of rows ra, rb (element offsets of their z = 0 in a
  // real field) on entry, N(psi) on exit
  static __device__ __forceinline__ int z_of(int t, int s) { return real_pos<N, DCT>(I::a_elem(t, s)); }

  // the monitors and outputs of PassFlags; o receives this CTA's three sums
  static __device__ __forceinline__ void monitor(const cplx<T> (&v)[E], int t, int flags, const PointParams& pp, int rep,
                                                 size_t ra, size_t rb, const double* psi_old, double* psi_out, double* o,
                                                 double* scratch) {
    KahanSum s0, s1, s2;
    const double eps = pp.eps[rep];
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int z = z_of(t, s);
      const double pa = double(v[s].x), pb = double(v[s].y);
      if (flags & kFlL1) {  // read before a possibly aliased write
        s0.add(fabs(pa - psi_old[ra + z]) + fabs(pb - psi_old[rb + z]));
        s1.add(fabs(pa) + fabs(pb));
      }
      if (flags & kFlPsiOut) {
        psi_out[ra + z] = pa;
        psi_out[rb + z] = pb;
      }
      if (flags & kFlEnergy) {
        s2.add(local_density(pa, eps, pp.beta, pp.gamma, pp.nonlin) +
               local_density(pb, eps, pp.beta, pp.gamma, pp.nonlin));
      }
    }
    if (flags & (kFlL1 | kFlEnergy)) {
      const double t0 = block_sum(s0.s, scratch);
      const double t1 = block_sum(s1.s, scratch);
      const double t2 = block_sum(s2.s, scratch);
      if (threadIdx.x == 0) {
        o[0] = t0;
        o[1] = t1;
        o[2] = t2;
      }
    }
  }
  // The same through the line ``x``, for the 32 values per thread of the split passes:
  // the lanes of a row pair hold consecutive z and the loops stay rolled.  Unrolled over
  // the registers, the FP64 code of the sums outgrew the instruction cache, and a store
  // between two reads of one array kept the reads apart.  256^3 plane pass, us, before ->
  // now: energy trace, FP32 Neumann 226 -> 113, periodic 144 -> 89, FP64 Neumann 374 ->
  // 218; L1 monitor every step, 268 -> 146, 1693 -> 135, 428 -> 269.
  template <class X>
  static __device__ __forceinline__ void monitor_line(const cplx<T> (&v)[E], int t, const X& x, int flags,
                                                      const PointParams& pp, int rep, size_t ra, size_t rb,
                                                      const double* psi_old, double* psi_out, double* o,
                                                      double* scratch) {
    x.sync();
#pragma unroll
    for (int s = 0; s < E; ++s) x.template store<16>(z_of(t, s), v[s]);
    x.sync();
    KahanSum s0, s1, s2;
    if (flags & kFlL1) {  // all of it before a possibly aliased write
#pragma unroll 4
      for (int z = t; z < N; z += I::G) {
        const cplx<T> q = x.template load<16>(z);
        const double pa = double(q.x), pb = double(q.y);
        s0.add(fabs(pa - psi_old[ra + z]) + fabs(pb - psi_old[rb + z]));
        s1.add(fabs(pa) + fabs(pb));
      }
    }
    if (flags & kFlPsiOut) {
#pragma unroll 4
      for (int z = t; z < N; z += I::G) {
        const cplx<T> q = x.template load<16>(z);
        psi_out[ra + z] = double(q.x);
        psi_out[rb + z] = double(q.y);
      }
    }
    if (flags & kFlEnergy) {
      const double eps = pp.eps[rep];
#pragma unroll 2
      for (int z = t; z < N; z += I::G) {
        const cplx<T> q = x.template load<16>(z);
        s2.add(local_density(double(q.x), eps, pp.beta, pp.gamma, pp.nonlin) +
               local_density(double(q.y), eps, pp.beta, pp.gamma, pp.nonlin));
      }
    }
    if (flags & (kFlL1 | kFlEnergy)) {
      const double t0 = block_sum(s0.s, scratch);
      const double t1 = block_sum(s1.s, scratch);
      const double t2 = block_sum(s2.s, scratch);
      if (threadIdx.x == 0) {
        o[0] = t0;
        o[1] = t1;
        o[2] = t2;
      }
    }
  }
  static __device__ __forceinline__ void real_store(const cplx<T> (&v)[E], int t, T* out, size_t ra, size_t rb) {
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int z = z_of(t, s);
      out[ra + z] = v[s].x;
      out[rb + z] = v[s].y;
    }
  }
  static __device__ __forceinline__ void nonlin(cplx<T> (&v)[E], const PointParams& pp) {
    const T beta = T(pp.beta), gamma = T(pp.gamma);
    if (pp.nonlin == kQuintic) {
#pragma unroll
      for (int s = 0; s < E; ++s)
        v[s] = mk<T>(nonlin_eval<T>(v[s].x, beta, gamma, kQuintic), nonlin_eval<T>(v[s].y, beta, gamma, kQuintic));
    } else {
#pragma unroll
      for (int s = 0; s < E; ++s)
        v[s] = mk<T>(nonlin_eval<T>(v[s].x, beta, gamma, kQuadCubic), nonlin_eval<T>(v[s].y, beta, gamma, kQuadCubic));
    }
  }
  // with the pinning penalty on the plane z = N/2 (periodicFFT/pf3dMorph.cpp:456-467,
  // its neighbours come through the line ``x``) and the substrate penalty on the
  // planes z < kwall (cosFFT/comet/cosNoAdvMorph.cpp:591-623)
  template <class X>
  static __device__ __forceinline__ void nonlin_penalties(cplx<T> (&v)[E], int t, const X& x, const PointParams& pp,
                                                          const T* wall, const T* lperp, int kwall, size_t ra, size_t rb) {
    const T beta = T(pp.beta), gamma = T(pp.gamma);
    if (pp.w_mid != 0.0) {
      x.sync();
#pragma unroll
      for (int s = 0; s < E; ++s) x.template store<16>(z_of(t, s), v[s]);
      x.sync();
    }
    const T* lpa = kwall > 0 ? lperp + (ra / N) * kwall : nullptr;
    const T* lpb = kwall > 0 ? lperp + (rb / N) * kwall : nullptr;
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int z = z_of(t, s);
      const cplx<T> q = v[s];
      cplx<T> o = mk<T>(nonlin_eval<T>(q.x, beta, gamma, pp.nonlin), nonlin_eval<T>(q.y, beta, gamma, pp.nonlin));
      if (pp.w_mid != 0.0 && z == N / 2) {
        const cplx<T> lo = x.template load<16>(z - 1), hi = x.template load<16>(z + 1);
        const T cw = T(2.0 * pp.w_mid * pp.inv_dz2);
        o.x += cw * (lo.x - T(2) * q.x + hi.x);
        o.y += cw * (lo.y - T(2) * q.y + hi.y);
      }
      if (z < kwall) {
        const T w = wall[z];
        o.x += w * lpa[z];
        o.y += w * lpb[z];
      }
      v[s] = o;
    }
  }
};

}  // namespace shb
