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

template <typename T>
struct YcolArgs {
  const cplx<T>* src;  // inverse: partial spectra of the slab's first plane; forward: the slab
  cplx<T>* dst;        // inverse: the slab; forward: partial spectra of the slab's first plane
  const cplx<T>* lt;   // line tables
};

// y transform of TK columns of one plane.  blockIdx.x = plane * TILES + tile.
// Bound by the memory it streams (two fields per pass); 16 columns keep every
// access whole 128-byte segments while four CTAs of 32 KB fit an SM.
template <typename T, int N, bool DCT, bool INV>
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
  if constexpr (INV) {
    const cplx<T>* src = a.src + size_t(plane) * Cfg::FP;
#pragma unroll
    for (int s = 0; s < E; ++s) v[s] = src[S::ky_of(t, s) * (N / 2) + col];
    S::col_inverse(v, t, x, tw, false, packed, [&](int ky) { return src[N * (N / 2) + ky]; });
    S::to_pairs(v, t, a.dst + size_t(plane) * Cfg::SP + 2 * col, N);
  } else {
    S::from_pairs(v, t, a.src + size_t(plane) * Cfg::SP + 2 * col, N);
    cplx<T>* dst = a.dst + size_t(plane) * Cfg::FP;
    S::col_forward(v, t, x, tw, false, packed, [&](int ky, cplx<T> z) { dst[N * (N / 2) + ky] = z; });
#pragma unroll
    for (int s = 0; s < E; ++s) dst[S::ky_of(t, s) * (N / 2) + col] = v[s];
  }
}

template <typename T, int N, bool DCT>
struct ZrowCfg {
  using I = LineIdx<N>;
  static constexpr int E = I::E, G = I::G;
  static constexpr int THREADS = 128;
  static constexpr int LINES = THREADS / G;  // row pairs per CTA
  static constexpr int BLOCKS = N / 2 / LINES;  // CTAs per plane
  static constexpr int SP = N * (N / 2);
  // padded line; the + 8 puts the two lines of a half-warp on different banks
  static constexpr int LS = N + N / 16 + 8;
  static constexpr size_t RED_OFF = size_t(LINES) * LS * sizeof(cplx<T>);
  static constexpr size_t SMEM = RED_OFF + 16 * sizeof(double);
  static constexpr int MIN_BLOCKS = split_threads<T, N>() / THREADS;
};

// kZrowStep: N(psi) alone.  kZrowGen: also the penalties, psi out and the
// monitors (PassFlags).
enum ZrowMode : int { kZrowStep = 0, kZrowGen = 1 };

template <typename T>
struct ZrowArgs {
  cplx<T>* slab;
  const cplx<T>* lt;
  PointParams pp;
  // kZrowGen
  int flags, plane0;      // first plane of the slab, rep * N + x
  double* psi_out;
  const double* psi_old;
  double* red;            // per-CTA partial sums [plane][BLOCKS][3]
  T* real_out;
  const T* wall;          // substrate penalty (PlaneArgs)
  const T* lperp;
  int kwall;
};

// z transforms of LINES row pairs around the real-space work.  G consecutive
// lanes own a line and exchange inside their warp: no block barrier, every warp
// runs on its own.  blockIdx.x = plane * BLOCKS + block.
template <typename T, int N, bool DCT, int MODE>
__global__ void __launch_bounds__(ZrowCfg<T, N, DCT>::THREADS, MODE == kZrowStep ? ZrowCfg<T, N, DCT>::MIN_BLOCKS : 0)
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
  cplx<T>* row = a.slab + size_t(plane) * Cfg::SP + p * N;
  cplx<T> v[E];
  grid_dependency_wait();
  S::row_inverse(v, t, row, x, tw, false, typename S::Plain());
  if constexpr (MODE == kZrowGen) {
    const int gp = a.plane0 + plane;
    const size_t ra = (size_t(gp) * N + real_pos<N, DCT>(p)) * N;
    const size_t rb = (size_t(gp) * N + real_pos<N, DCT>(p + N / 2)) * N;
    if (a.flags & (kFlPsiOut | kFlL1 | kFlEnergy))
      S::monitor(v, t, a.flags, a.pp, gp / N, ra, rb, a.psi_old, a.psi_out,
                 a.red + (size_t(gp) * Cfg::BLOCKS + blockIdx.x % Cfg::BLOCKS) * 3,
                 reinterpret_cast<double*>(smem_raw + Cfg::RED_OFF));
    if (a.flags & kFlRealOut) S::real_store(v, t, a.real_out, ra, rb);
    S::nonlin_penalties(v, t, x, a.pp, a.wall, a.lperp, a.kwall, ra, rb);
  } else {
    S::nonlin(v, a.pp);
  }
  S::row_forward(v, t, row, x, tw, true, [] {}, typename S::Plain());
}

}  // namespace shb
