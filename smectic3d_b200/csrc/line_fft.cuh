// Two-pass line transforms for sm_100a: N = RA x RB, one exchange of the line.
//
// A group of G threads owns a line of N complex points, E = N / G values per
// thread in registers.  Both directions go through the same two register layouts:
//
//   A side (real space):  slot a RA + r holds element  jA + RB r,  jA = t + G a
//   B side (wavenumbers): slot b RB + r holds element  jB + RA r,  jB = jb(t, b)
//
// forward: DFT_RA on the A side, exchange, twiddle, DFT_RB -> B side
// inverse: DFT_RB on the B side, exchange, twiddle, DFT_RA -> A side
//
// The B-side butterflies of a thread come in mirrored pairs (j and RA - j), so
// element k and its mirror N - k sit in the same thread: REDFT10 / REDFT01, the
// Hermitian split of two packed real lines and the kz = 0, N/2 columns need
// neither shuffles nor a round trip through shared memory (with 16 values per
// thread and one butterfly, each of those cost two shuffles and two selects per
// value, as much as the transform itself).  Slot s mirrors into slot E - 1 - s,
// except in thread 0, whose first and last butterfly (0 and RA / 2) are their own
// mirrors: canon() moves thread 0's values so that the rule holds there too, which
// costs RB selects instead of a second code path.
//
// FP32 results are bit for bit those of the former one-butterfly form at every
// size but 512 (same radices, same order of the roundings); a cheaper form of the
// REDFT10 pair is used in FP64.
//
// The exchange is a caller-supplied object with sync / store / load.
#pragma once
#include "fft_engine.cuh"

namespace shb {

template <int N> struct LinePlan;
template <> struct LinePlan<16>  { static constexpr int RA = 4,  RB = 4; };
template <> struct LinePlan<32>  { static constexpr int RA = 8,  RB = 4; };
template <> struct LinePlan<64>  { static constexpr int RA = 16, RB = 4; };
template <> struct LinePlan<128> { static constexpr int RA = 16, RB = 8; };
template <> struct LinePlan<256> { static constexpr int RA = 16, RB = 16; };
template <> struct LinePlan<512> { static constexpr int RA = 32, RB = 16; };

// Device tables of one transform length (complex entries), built on the host:
//   colB [t][E]   forward twiddles w^{jB r} in B-side slot order
//   colA [t][E]   inverse twiddles w^{-jA r} in A-side slot order
//   colD [t][E/2] quarter-wave exp(-i pi k / 2N) of the canonical slots s < E / 2
//   rowB, rowA, rowD  the same, [slot][t]
// The [t][slot] order is for kernels whose lanes share t (one vector load
// serves the warp), the [slot][t] order for lanes with consecutive t.
template <int N>
struct LineTab {
  static constexpr int colB = 0, colA = N, colD = 2 * N, rowB = 2 * N + N / 2, rowA = rowB + N, rowD = rowA + N;
  static constexpr int total = rowD + N / 2;
};

template <int N>
struct LineIdx {
  static constexpr int RA = LinePlan<N>::RA, RB = LinePlan<N>::RB;
  static constexpr int E = RA > 2 * RB ? RA : 2 * RB, G = N / E;
  static constexpr int NA = E / RA, NB = E / RB;  // butterflies per thread on either side
  static_assert((NB == 2 && G == RA / 2) || (NB == 4 && G == RA / 4), "line plan");
  static __host__ __device__ __forceinline__ int ja(int t, int a) { return t + G * a; }
  static __host__ __device__ __forceinline__ int jb(int t, int b) {
    if (b == 0) return t;
    if (b == NB - 1) return t == 0 ? RA / 2 : RA - t;
    return b == 1 ? (t == 0 ? RA / 4 : RA / 2 - t) : (t == 0 ? RA / 2 + RA / 4 : RA / 2 + t);
  }
  // element of A-side slot s
  static __host__ __device__ __forceinline__ int a_elem(int t, int s) { return ja(t, s / RA) + RB * (s % RA); }
  // element of B-side slot s, butterfly order
  static __host__ __device__ __forceinline__ int b_elem(int t, int s) { return jb(t, s / RB) + RA * (s % RB); }
  // element of canonical slot s < E / 2, and of its mirror slot E - 1 - s
  static __host__ __device__ __forceinline__ int c_elem(int t, int s) {
    if (s >= RB) return b_elem(t, s);
    return RA * s + ((t == 0 && s >= RB / 2) ? RA / 2 : t);
  }
  static __host__ __device__ __forceinline__ int c_mirror(int t, int s) {
    return (s == 0 && t == 0) ? N / 2 : N - c_elem(t, s);
  }
  // element of any canonical slot
  static __host__ __device__ __forceinline__ int c_slot(int t, int s) {
    return s < E / 2 ? c_elem(t, s) : c_mirror(t, E - 1 - s);
  }
  // whether c_elem(t, s) < N / 2 (else its mirror is)
  static __host__ __device__ constexpr bool c_low(int s) { return s % RB < RB / 2; }
};

template <typename T, int N, class Vec>
void host_line_tables(Vec& out) {
  using I = LineIdx<N>;
  using L = LineTab<N>;
  const long double pi = 3.141592653589793238462643383279502884L;
  out.resize(L::total);
  auto w = [&](long double ang) {
    cplx<T> c;
    c.x = T(cosl(ang));
    c.y = T(sinl(ang));
    return c;
  };
  for (int t = 0; t < I::G; ++t) {
    for (int s = 0; s < I::E; ++s) {
      const cplx<T> b = w(-2.0L * pi * (long double)(I::jb(t, s / I::RB) * (s % I::RB)) / N);
      const cplx<T> a = w(2.0L * pi * (long double)(I::ja(t, s / I::RA) * (s % I::RA)) / N);
      out[L::colB + t * I::E + s] = b;
      out[L::rowB + s * I::G + t] = b;
      out[L::colA + t * I::E + s] = a;
      out[L::rowA + s * I::G + t] = a;
    }
    for (int s = 0; s < I::E / 2; ++s) {
      const cplx<T> d = w(-pi * I::c_elem(t, s) / (2.0L * N));
      out[L::colD + t * (I::E / 2) + s] = d;
      out[L::rowD + s * I::G + t] = d;
    }
  }
}

// Twiddle readers.  get2(s, a, b) reads slots s and s + 1 (s even).
template <typename T>
struct ColTab {
  const cplx<T>* p;  // table + t * (entries per thread)
  __device__ __forceinline__ void get2(int s, cplx<T>& a, cplx<T>& b) const {
    if constexpr (sizeof(T) == 4) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(p + s));
      a = mk<T>(v.x, v.y);
      b = mk<T>(v.z, v.w);
    } else {
      a = __ldg(p + s);
      b = __ldg(p + s + 1);
    }
  }
};
template <typename T, int G>
struct RowTab {
  const cplx<T>* p;  // table + t
  __device__ __forceinline__ void get2(int s, cplx<T>& a, cplx<T>& b) const {
    a = __ldg(p + s * G);
    b = __ldg(p + (s + 1) * G);
  }
};
// the three tables of a thread, column (lanes share t) or row (consecutive t) order
template <typename T, int N>
struct ColTables {
  ColTab<T> b, a, d;
  __device__ __forceinline__ ColTables(const cplx<T>* tab, int t)
      : b{tab + LineTab<N>::colB + t * LineIdx<N>::E},
        a{tab + LineTab<N>::colA + t * LineIdx<N>::E},
        d{tab + LineTab<N>::colD + t * (LineIdx<N>::E / 2)} {}
};
template <typename T, int N>
struct RowTables {
  RowTab<T, LineIdx<N>::G> b, a, d;
  __device__ __forceinline__ RowTables(const cplx<T>* tab, int t)
      : b{tab + LineTab<N>::rowB + t}, a{tab + LineTab<N>::rowA + t}, d{tab + LineTab<N>::rowD + t} {}
};

// Exchange of a tile of TK lines whose lanes are the lines: element p of line c
// at p TK + c, so that a warp reads and writes whole rows without conflicts.
template <typename T, int TK>
struct TileExchange {
  cplx<T>* base;  // tile + c
  __device__ __forceinline__ void sync() const { __syncthreads(); }
  template <int R>
  __device__ __forceinline__ void store(int p, cplx<T> v) const { base[p * TK] = v; }
  template <int R>
  __device__ __forceinline__ cplx<T> load(int p) const { return base[p * TK]; }
};
// Exchange inside a warp: the G threads of a line are consecutive lanes.  Every R
// elements, R the radix that stores them, are followed by one slot of padding: the
// stores of neighbouring threads are R + 1 apart and their loads consecutive, which
// with the line strides of the kernels is free of bank conflicts both ways (a fixed
// 16 made the inverse stores of the 64-point lines four-way).
template <typename T>
struct WarpExchange {
  cplx<T>* line;
  __device__ __forceinline__ void sync() const { __syncwarp(); }
  template <int R>
  __device__ __forceinline__ void store(int p, cplx<T> v) const { line[p + p / R] = v; }
  template <int R>
  __device__ __forceinline__ cplx<T> load(int p) const { return line[p + p / R]; }
};
// slots of such a line
template <int N>
__host__ __device__ constexpr int warp_line() { return N + N / LinePlan<N>::RB; }

template <typename T, int N>
struct LineFFT {
  using I = LineIdx<N>;
  static constexpr int RA = I::RA, RB = I::RB, E = I::E, NA = I::NA, NB = I::NB;

  // A side -> B side (butterfly order).  ``first_sync``: the exchange buffer may
  // still be read by other threads.
  template <class X, class Tab>
  static __device__ __forceinline__ void forward(cplx<T> (&v)[E], int t, const X& x, const Tab& tw, bool first_sync) {
#pragma unroll
    for (int a = 0; a < NA; ++a) DFT<T, RA, -1>::run(&v[a * RA]);
    if (first_sync) x.sync();
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
      for (int q = 0; q < RA; ++q) x.template store<RA>(I::ja(t, a) * RA + q, v[a * RA + q]);
    x.sync();
#pragma unroll
    for (int s = 0; s < E; ++s) v[s] = x.template load<RA>(I::b_elem(t, s));
#pragma unroll
    for (int s = 0; s < E; s += 2) {
      cplx<T> w0, w1;
      tw.b.get2(s, w0, w1);
      if (s % RB != 0) v[s] = cmul<T>(v[s], w0);
      v[s + 1] = cmul<T>(v[s + 1], w1);
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) DFT<T, RB, -1>::run(&v[b * RB]);
  }

  // B side (butterfly order) -> A side
  template <class X, class Tab>
  static __device__ __forceinline__ void inverse(cplx<T> (&v)[E], int t, const X& x, const Tab& tw, bool first_sync) {
#pragma unroll
    for (int b = 0; b < NB; ++b) DFT<T, RB, +1>::run(&v[b * RB]);
    if (first_sync) x.sync();
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int q = 0; q < RB; ++q) x.template store<RB>(I::jb(t, b) * RB + q, v[b * RB + q]);
    x.sync();
#pragma unroll
    for (int s = 0; s < E; ++s) v[s] = x.template load<RB>(I::a_elem(t, s));
#pragma unroll
    for (int s = 0; s < E; s += 2) {
      cplx<T> w0, w1;
      tw.a.get2(s, w0, w1);
      if (s % RA != 0) v[s] = cmul<T>(v[s], w0);
      v[s + 1] = cmul<T>(v[s + 1], w1);
    }
#pragma unroll
    for (int a = 0; a < NA; ++a) DFT<T, RA, +1>::run(&v[a * RA]);
  }

  static __device__ __forceinline__ cplx<T> sel(bool c, cplx<T> a, cplx<T> b) {
    return mk<T>(c ? a.x : b.x, c ? a.y : b.y);
  }
  // butterfly order -> canonical order (slot s mirrors into slot E - 1 - s): only
  // thread 0 moves anything, between its first and last butterfly
  static __device__ __forceinline__ void canon(cplx<T> (&v)[E], int t) {
    const bool z = t == 0;
    constexpr int LB = E - RB;  // first slot of the last butterfly
    cplx<T> lo[RB / 2];         // first butterfly, upper half
#pragma unroll
    for (int r = RB / 2; r < RB; ++r) {
      lo[r - RB / 2] = v[r];
      v[r] = sel(z, v[LB + r], v[r]);
    }
    // mirror of slot r < RB / 2: thread 0 element RA (RB - r) of butterfly 0 (r > 0), RA RB / 2 (r = 0)
#pragma unroll
    for (int r = 0; r < RB / 2; ++r) {
      const int src = r == 0 ? RB / 2 : RB - r;
      v[E - 1 - r] = sel(z, lo[src - RB / 2], v[E - 1 - r]);
    }
  }
  static __device__ __forceinline__ void uncanon(cplx<T> (&v)[E], int t) {
    const bool z = t == 0;
    cplx<T> hi[RB / 2];  // canonical mirrors of slots r < RB / 2
#pragma unroll
    for (int r = 0; r < RB / 2; ++r) {
      hi[r] = v[E - 1 - r];
      v[E - 1 - r] = sel(z, v[RB - 1 - r], hi[r]);  // thread 0: butterfly RA/2 slot RB - 1 - r
    }
#pragma unroll
    for (int r = RB / 2; r < RB; ++r) {
      const int m = r == RB / 2 ? 0 : RB - r;
      v[r] = sel(z, hi[m], v[r]);
    }
  }

  // REDFT10 post-processing of V = FFT of the permuted line, canonical order:
  //   X[k] = w V[k] + conj(w) V[N-k],  w = exp(-i pi k / 2N),  V[N] = V[0]
  // In FP64 the mirror takes the same two products: X[N-k] = i (w V[k] - conj(w) V[N-k]).
  template <class Tab>
  static __device__ __forceinline__ void dct2_post(cplx<T> (&v)[E], int t, const Tab& tw) {
    const T h = T(0.70710678118654752440);
#pragma unroll
    for (int s = 0; s < E / 2; s += 2) {
      cplx<T> w2[2];
      tw.d.get2(s, w2[0], w2[1]);
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const cplx<T> a = v[s + g], b = v[E - 1 - s - g], w = w2[g];
        if (s + g == 0 || sizeof(T) == 4) {
          // k = 0 and N/2 (thread 0, slot 0) are their own mirrors
          const bool self = s + g == 0 && t == 0;
          const cplx<T> pa = s + g == 0 ? sel(self, a, b) : b, pb = s + g == 0 ? sel(self, b, a) : a;
          cplx<T> m = mk<T>(-w.y, -w.x);  // exp(-i pi (N - k) / 2N)
          if (s + g == 0) m = sel(self, mk<T>(h, -h), m);
          v[s + g] = cadd<T>(cmul<T>(a, w), cmul<T>(pa, conjg<T>(w)));
          v[E - 1 - s - g] = cadd<T>(cmul<T>(b, m), cmul<T>(pb, conjg<T>(m)));
        } else {
          const cplx<T> p = cmul<T>(a, w), q = cmul<T>(b, conjg<T>(w));
          const cplx<T> d = csub<T>(p, q);
          v[s + g] = cadd<T>(p, q);
          v[E - 1 - s - g] = mk<T>(-d.y, d.x);
        }
      }
    }
  }
  // REDFT01 pre-processing, canonical order:
  //   V[k] = conj(w) (X[k] - i X[N-k]),  X[N] = 0
  template <class Tab>
  static __device__ __forceinline__ void dct3_pre(cplx<T> (&v)[E], int t, const Tab& tw) {
    const T h = T(0.70710678118654752440);
#pragma unroll
    for (int s = 0; s < E / 2; s += 2) {
      cplx<T> w2[2];
      tw.d.get2(s, w2[0], w2[1]);
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const cplx<T> a = v[s + g], b = v[E - 1 - s - g], w = w2[g];
        cplx<T> pa = b, pb = a, m = mk<T>(-w.y, -w.x);
        if (s + g == 0) {  // thread 0: k = 0 has no mirror, k = N/2 is its own
          const bool self = t == 0;
          pa = sel(self, mk<T>(T(0), T(0)), b);
          pb = sel(self, b, a);
          m = sel(self, mk<T>(h, -h), m);
        }
        v[s + g] = cmul<T>(mk<T>(a.x + pa.y, a.y - pa.x), conjg<T>(w));
        v[E - 1 - s - g] = cmul<T>(mk<T>(b.x + pb.y, b.y - pb.x), conjg<T>(m));
      }
    }
  }
};

// position on the real axis of element n of the FFT: natural, or the Makhoul
// even / odd permutation of the cosine transforms
template <int N, bool DCT>
__host__ __device__ __forceinline__ int real_pos(int n) {
  if (!DCT) return n;
  return n < N / 2 ? 2 * n : 2 * (N - 1 - n) + 1;
}

}  // namespace shb
