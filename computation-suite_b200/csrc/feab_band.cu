// Direct solve of the reduced SPD system: banded tile Cholesky on the GPU.
//
// Replaces FESystem._sparse_lu_solve (fea_engine/src/fea_engine/solver.py:1681-1724), the SuperLU
// factorisation behind solve_static(method=None).  K_ff is SPD, so the factorisation without
// pivoting is its Cholesky factor L (U = D L^T with U_ii = L_ii^2), and the reference's
// singularity test on SuperLU's pivots (min |U_ii| < tol max |U_ii|) is made on the pivots L_ii^2.
//
// The caller renumbers the rows (a bandwidth-reducing order) so that every nonzero lies within
// `bandwidth` of the diagonal.  The lower band is kept as 64 x 64 tiles: block row I holds the
// tiles of block columns I - bands .. I, tile (I, d) being block column I - d.  The fill of a
// Cholesky factor stays inside the band, so the factorisation is a tile algorithm over block columns
// J = 0 .. n_tiles - 1: the diagonal tile is factored and its factor inverted (Linv_JJ, kept beside
// the band), and the tiles below it are L_IJ = (A_IJ - sum_K L_IK L_JK^T) Linv_JJ^T, products of 64 x
// 64 tiles on the FP64 tensor path (mma.sync).  It runs as one kernel (k_band_factor).
// The solves walk the block rows forward (L y = b) and backward (L^T x = y) with the inverted diagonal
// factors, in one kernel of one cluster (k_band_solve).
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include "feab_common.cuh"

namespace feab {
namespace {

constexpr int kT = FEAB_BAND_TILE;       // tile edge
constexpr int kTile = kT * kT;           // doubles per tile

__host__ __device__ inline size_t tile_index(int I, int d, int bands) {
  return ((size_t)I * (size_t)(bands + 1) + (size_t)d) * (size_t)kTile;
}

// ---------------------------------------------------------------- bandwidth and assembly
// One warp per CSR row: the largest |iperm[row] - iperm[col]|; an iperm entry outside [0, n)
// sets bad.
__global__ void k_band_width(const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ col_idx, int32_t n,
                             const int32_t* __restrict__ iperm, int32_t* width, int32_t* bad) {
  const int lane = threadIdx.x & 31;
  const int row = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
  if (row >= n) return;
  const int i = __ldg(iperm + row);
  int w = 0;
  bool ok = i >= 0 && i < n;
  for (int e = __ldg(row_ptr + row) + lane; e < __ldg(row_ptr + row + 1); e += 32) {
    const int c = __ldg(col_idx + e);
    const int j = (c >= 0 && c < n) ? __ldg(iperm + c) : -1;
    if (j < 0 || j >= n) ok = false;
    else w = max(w, abs(i - j));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) w = max(w, __shfl_xor_sync(FEAB_FULL_MASK, w, o));
  const bool all_ok = __all_sync(FEAB_FULL_MASK, ok);
  if (lane == 0) {
    atomicMax(width, w);
    if (!all_ok) atomicExch(bad, 1);
  }
}

// One warp per CSR row: the row's lower entries (new row >= new column) into their tiles; an
// entry outside the band sets bad.
__global__ void k_band_scatter(const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ col_idx,
                               const double* __restrict__ vals, int32_t n, const int32_t* __restrict__ iperm,
                               int bands, double* __restrict__ tiles, int32_t* bad) {
  const int lane = threadIdx.x & 31;
  const int row = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
  if (row >= n) return;
  const int i = __ldg(iperm + row), I = i / kT;
  for (int e = __ldg(row_ptr + row) + lane; e < __ldg(row_ptr + row + 1); e += 32) {
    const int c = __ldg(col_idx + e);
    const int j = (c >= 0 && c < n) ? __ldg(iperm + c) : -1;
    if (i < 0 || i >= n || j < 0 || j >= n) {  // not a permutation of the rows: skip, report
      atomicExch(bad, 1);
      continue;
    }
    if (j > i) continue;
    const int d = I - j / kT;
    if (d > bands) {
      atomicExch(bad, 1);
      continue;
    }
    tiles[tile_index(I, d, bands) + (size_t)(i % kT) * kT + (j % kT)] = __ldg(vals + e);
  }
}

// Rows n .. 64 n_tiles - 1 are identity rows.
__global__ void k_band_pad(int32_t n, int n_tiles, int bands, double* __restrict__ tiles) {
  const int r = n + blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n_tiles * kT) return;
  tiles[tile_index(r / kT, 0, bands) + (size_t)(r % kT) * kT + (r % kT)] = 1.0;
}

// ---------------------------------------------------------------- factorisation
// The 256-byte header of the band storage.
struct BandState {
  unsigned long long piv_min, piv_max;  // bit patterns of positive doubles (order-preserving)
  int32_t status;
  int32_t bad;                          // assembly: an entry outside the band
  int32_t next_task, abort_flag;        // factorisation
  int32_t solve_error;                  // of solves without an error flag of their own
};
static_assert(sizeof(BandState) <= FEAB_BAND_HEADER_BYTES, "band header");
static_assert(offsetof(BandState, solve_error) == FEAB_BAND_ERROR_BYTE, "band header");

// The factorisation is one cooperative kernel, so that a block column costs what its dependences
// cost and not three launches.  CTA 0 walks the diagonal (the chain): for block row J it forms
// L_{J,J-1} = C_{J,J-1} Linv_{J-1}^T, takes it from the diagonal tile, factors that tile and inverts
// the factor.  The other CTAs (workers) draw tasks, each one tile of the band brought up to date
// left-looking, in one go: C_IJ = A_IJ - sum_K L_IK L_JK^T, and for tiles at least two below the
// diagonal L_IJ = C_IJ Linv_J^T.  The two tiles of a row that the chain needs next are left as C
// (without the last term, which the chain adds).  Progress is published per block row: progress[I]
// = K + 1 once L_IK is stored (a row's tiles finish in order of K), prepared[I] counts the two
// tiles left for the chain.  Tasks are drawn in an order in which each depends only on tasks before
// it and on the chain, and all CTAs run at once, so every wait ends; each is bounded all the same
// and a CTA whose wait runs out makes all leave with an error.
//
// What bounds it: the chain, as long as the workers keep up (b (b + 1) / 2 tile products per block
// column over 147 SMs), else the FP64 tensor path.  Of the chain's 14.5 us per block column the 64
// pivots take 6.5 (a reciprocal square root, a product and a difference, 16 cycles each, one after
// the other), the two products 3.2, the inverse 2.7.  Measured, three launches per block column ->
// one kernel: 64x16x16 elements (867 block columns, 28 bands) 74.2 -> 12.6 ms, 96x24x24 (2,813, 59
// bands, bound by the workers at 22 TFLOP/s) 335 -> 118 ms (45.7 with the nodes in layers, 31 bands), 33x9x8 (140, 9 bands) 10.6 -> 2.0 ms.

struct BandWork {
  double* tiles;
  double* inv;
  BandState* st;
  int32_t* progress;   // n_tiles
  int32_t* prepared;   // n_tiles
  int32_t* next_task;
  int32_t* abort_flag;
  int32_t n, n_tiles, bands;
};

constexpr int kBandThreads = 256;
constexpr int kMmaLd = kT + 4;                 // row stride of a staged tile: no bank conflicts between fragments
constexpr int kStage = kT * kMmaLd;            // doubles of a staged tile
constexpr size_t kFactorSmem = 6 * kStage * sizeof(double);   // of the chain; the workers use four stages
constexpr int kBandSpinLimit = 1 << 22;        // polls before a wait gives up (seconds)

__device__ __forceinline__ void dmma884(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

__device__ __forceinline__ int32_t ld_relaxed(const int32_t* p) {
  int32_t v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(int32_t* p, int32_t v) {
  asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// All threads, after their stores: `where` becomes `value` (0: it is counted up) once the stores are
// visible to every CTA.  One thread of warp 1 waits for that (a thousand cycles); the others go on.
__device__ __forceinline__ void publish(int32_t* where, int32_t value) {
  __syncthreads();
  if (threadIdx.x == 32) {
    fence_gpu();
    if (value) st_relaxed(where, value);
    else atomicAdd(where, 1);
  }
}

// One thread: waits until *p >= want.  False (and every CTA told) when that takes too long.
__device__ __forceinline__ bool wait_for(const int32_t* p, int32_t want, int32_t* abort_flag) {
  for (int spin = 0; ld_relaxed(p) < want; ++spin) {
    if (spin >= kBandSpinLimit) atomicExch(abort_flag, 1);
    if ((spin & 255) == 255 && ld_relaxed(abort_flag)) return false;
  }
  fence_gpu();
  return true;
}

// Asynchronous copy of a tile into its padded stage (all threads; commit and wait are the caller's).
__device__ __forceinline__ void stage_tile(double* dst, const double* src) {
  for (int q = threadIdx.x; q < kTile / 2; q += kBandThreads) {
    const int row = q / (kT / 2), k2 = q % (kT / 2);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst + row * kMmaLd + 2 * k2)),
                 "l"(src + 2 * (size_t)q)
                 : "memory");
  }
}
__device__ __forceinline__ void stage_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void stage_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// acc += A B^T of two staged 64 x 64 tiles, on the FP64 tensor path: warp w owns rows 16 (w / 2) .. + 15
// and 32 columns as 2 x 4 accumulators; the column half changes sides at warp 4, so that each
// scheduler (warps w and w + 4) has one warp of either half.  TRI: B is lower triangular, columns k
// past the output column are zero and left out.  LOWER: only blocks on or below the diagonal.  Fragments (m8n8k4): A
// row-major 8 x 4, lane l holds (l / 4, l % 4); B column-major 4 x 8, lane l holds (l % 4, l / 4); C
// 8 x 8, lane l holds (l / 4, 2 (l % 4) + i).
typedef double TileAcc[2][4][2];

__device__ __forceinline__ void tile_zero(TileAcc& acc) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
}

__device__ __forceinline__ int tile_row0() { return 16 * (threadIdx.x >> 6); }
__device__ __forceinline__ int tile_col0() { return 32 * (((threadIdx.x >> 5) ^ (threadIdx.x >> 7)) & 1); }

template <bool TRI, bool LOWER>
__device__ __forceinline__ void tile_mma(const double* As, const double* Bs, TileAcc& acc) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, row0 = tile_row0(), col0 = tile_col0();
  if (LOWER && col0 > row0 + 15) return;
  const double* Ar = As + (row0 + g) * kMmaLd + t;
  const double* Br = Bs + (col0 + g) * kMmaLd + t;
  const int kend = TRI ? col0 + 32 : kT;
#pragma unroll 4
  for (int k0 = 0; k0 < kend; k0 += 4) {
    const double a0 = Ar[k0], a1 = Ar[8 * kMmaLd + k0];
    double b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = Br[8 * j * kMmaLd + k0];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (TRI && k0 >= col0 + 8 * j + 8) continue;
      if (!LOWER || col0 + 8 * j <= row0) dmma884(acc[0][j], a0, b[j]);
      if (!LOWER || col0 + 8 * j <= row0 + 8) dmma884(acc[1][j], a1, b[j]);
    }
  }
}

// The accumulators' places in a tile of row stride ld: fn(offset of two adjacent columns, i, j).
template <typename F>
__device__ __forceinline__ void tile_each(int ld, F fn) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) fn((tile_row0() + 8 * i + g) * ld + tile_col0() + 8 * j + 2 * t, i, j);
}

// C -= L L^T on the blocks on or below the diagonal: warp w < 4 block row w, warp w >= 4 block row
// 11 - w, so that each scheduler has nine blocks.  NB: blocks of the block row.
template <int NB>
__device__ __forceinline__ void syrk_row(const double* Ls, double* C) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double acc[NB][2];
#pragma unroll
  for (int j = 0; j < NB; ++j) acc[j][0] = acc[j][1] = 0.0;
  const double* Ar = Ls + (8 * (NB - 1) + g) * kMmaLd + t;
  const double* Br = Ls + g * kMmaLd + t;
#pragma unroll 4
  for (int k0 = 0; k0 < kT; k0 += 4) {
    const double a = Ar[k0];
    double b[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) b[j] = Br[8 * j * kMmaLd + k0];
#pragma unroll
    for (int j = 0; j < NB; ++j) dmma884(acc[j], a, b[j]);
  }
#pragma unroll
  for (int j = 0; j < NB; ++j) {
    double2* c = reinterpret_cast<double2*>(C + (8 * (NB - 1) + g) * kMmaLd + 8 * j + 2 * t);
    double2 v = *c;
    v.x -= acc[j][0];
    v.y -= acc[j][1];
    *c = v;
  }
}

__device__ __forceinline__ void tile_syrk(const double* Ls, double* C) {
  switch (threadIdx.x >> 5) {
    case 0: syrk_row<1>(Ls, C); break;
    case 1: syrk_row<2>(Ls, C); break;
    case 2: syrk_row<3>(Ls, C); break;
    case 3: syrk_row<4>(Ls, C); break;
    case 4: syrk_row<8>(Ls, C); break;
    case 5: syrk_row<7>(Ls, C); break;
    case 6: syrk_row<6>(Ls, C); break;
    default: syrk_row<5>(Ls, C); break;
  }
}

// C B^T of an 8 x 8 block: rows at A, columns' rows at B, eight columns of k; one warp.
__device__ __forceinline__ void mma8(double (&c)[2], const double* A, const double* B, int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int k0 = 0; k0 < 8; k0 += 4) dmma884(c, A[g * kMmaLd + k0 + t], B[g * kMmaLd + k0 + t]);
}

// Cholesky of the staged tile C (lower part), L in its place with zeros above the diagonal, and the
// inverse of L in X (W: scratch).  Panels of 8 columns: warp 0 factors a panel in registers, a lane
// per two rows, every lane carrying the 8 x 8 diagonal block along so that no pivot crosses lanes,
// while the other warps apply the panel before it to the columns behind.  pivot[] takes the pivots; one
// that is not > 0 counts as 1.  The inverse is put together from the inverses of the 8 x 8 diagonal
// blocks, doubling the block: X_21 = -X_22 (L_21 X_11).  after_panels() runs between the two parts.
struct TileScratch {
  double pivot[kT];
  double rsq[kT];   // pivot^(-1/2)
};

// One doubling: off-diagonal squares of H x H blocks.
template <int H>
__device__ __forceinline__ void inverse_double(const double* C, double* X, double* W) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  constexpr int kBlocks = 4 / H * H * H;                 // 8 x 8 output blocks of a pass: 4, 8, 16
  constexpr int kPer = (kBlocks + 7) / 8;                // of one warp
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
    double c[kPer][2];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      c[u][0] = c[u][1] = 0.0;
      const int q = warp + 8 * u;
      if (q < kBlocks) {
        const int pr = q / (H * H), bi = (q % (H * H)) / H, bj = q % H;
        const int r0 = 8 * (2 * H * pr + H), c0 = 8 * 2 * H * pr;   // first row of block 2, first column of block 1
        const double* A = (pass == 0 ? C + (r0 + 8 * bi) * kMmaLd + c0 : X + (r0 + 8 * bi) * kMmaLd + r0) + g * kMmaLd + t;
        const double* B = (pass == 0 ? X + c0 * kMmaLd + c0 : W + r0 * kMmaLd + c0) + 8 * bj + t * kMmaLd + g;
        double a[2 * H], b[2 * H];
#pragma unroll
        for (int k = 0; k < 2 * H; ++k) {
          a[k] = A[4 * k];
          b[k] = B[4 * k * kMmaLd];
        }
#pragma unroll
        for (int k = 0; k < 2 * H; ++k) dmma884(c[u], a[k], b[k]);
      }
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int q = warp + 8 * u;
      if (q < kBlocks) {
        const int pr = q / (H * H), bi = (q % (H * H)) / H, bj = q % H;
        const int r0 = 8 * (2 * H * pr + H), c0 = 8 * 2 * H * pr;
        double2* out = reinterpret_cast<double2*>((pass == 0 ? W : X) + (r0 + 8 * bi + g) * kMmaLd + c0 + 8 * bj + 2 * t);
        *out = pass == 0 ? make_double2(c[u][0], c[u][1]) : make_double2(-c[u][0], -c[u][1]);
      }
    }
    __syncthreads();
  }
}

// last_panel() runs in warp 7 beside the last panel.
template <typename P, typename F>
__device__ __forceinline__ void tile_cholesky(double* C, double* X, double* W, TileScratch& sc, P last_panel,
                                              F after_panels) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
#pragma unroll 1   // the body is long: eight copies would not stay in the instruction cache
  for (int p = 0; p < 8; ++p) {
    const int base = 8 * p;
    if (p > 0) {
      // column block p takes panel p - 1 first: warp w the block in block row p + w
      if (p + warp < 8) {
        double c[2] = {0.0, 0.0};
        double2* d = reinterpret_cast<double2*>(C + (8 * (p + warp) + g) * kMmaLd + base + 2 * t);
        double2 v = *d;
        mma8(c, C + 8 * (p + warp) * kMmaLd + base - 8, C + base * kMmaLd + base - 8, lane);
        v.x -= c[0];
        v.y -= c[1];
        *d = v;
      }
      __syncthreads();
    }
    if (warp == 0) {
      double d[8][8], a1[8], a2[8];
      const int r1 = base + lane, r2 = base + 32 + lane;
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int k = 0; k <= i; k += 2) {
          const double2 u = *reinterpret_cast<const double2*>(C + (base + i) * kMmaLd + base + k);
          d[i][k] = u.x;
          d[i][k + 1] = u.y;
        }
#pragma unroll
      for (int k = 0; k < 8; k += 2) {
        const double2 u = r1 < kT ? *reinterpret_cast<const double2*>(C + r1 * kMmaLd + base + k) : make_double2(0.0, 0.0);
        const double2 w = r2 < kT ? *reinterpret_cast<const double2*>(C + r2 * kMmaLd + base + k) : make_double2(0.0, 0.0);
        a1[k] = u.x;
        a1[k + 1] = u.y;
        a2[k] = w.x;
        a2[k + 1] = w.y;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const double pj = d[j][j];
        const double pv = pj > 0.0 ? pj : 1.0;
        const double rs = rsqrt(pv);
        if (lane == 0) {
          sc.pivot[base + j] = pj;
          sc.rsq[base + j] = rs;
        }
#pragma unroll
        for (int i = j + 1; i < 8; ++i) d[i][j] *= rs;
        a1[j] = lane > j ? a1[j] * rs : (lane == j ? pv * rs : 0.0);
        a2[j] *= rs;
#pragma unroll
        for (int k = j + 1; k < 8; ++k) {
#pragma unroll
          for (int i = k; i < 8; ++i) d[i][k] -= d[i][j] * d[k][j];
          a1[k] -= a1[j] * d[k][j];
          a2[k] -= a2[j] * d[k][j];
        }
      }
#pragma unroll
      for (int k = 0; k < 8; k += 2) {
        if (r1 < kT) *reinterpret_cast<double2*>(C + r1 * kMmaLd + base + k) = make_double2(a1[k], a1[k + 1]);
        if (r2 < kT) *reinterpret_cast<double2*>(C + r2 * kMmaLd + base + k) = make_double2(a2[k], a2[k + 1]);
      }
    } else {
      if (p > 0) {
        // panel p - 1 on the columns behind block p: the blocks (i, k), p < k <= i < 8
        const int m = 7 - p;
        for (int q = warp - 1; q < m * (m + 1) / 2; q += 7) {
          int i = 0;
          while ((i + 1) * (i + 2) / 2 <= q) ++i;
          const int k = q - i * (i + 1) / 2, bi = 8 * (p + 1 + i), bk = 8 * (p + 1 + k);
          double c[2] = {0.0, 0.0};
          mma8(c, C + bi * kMmaLd + base - 8, C + bk * kMmaLd + base - 8, lane);
          double2* d = reinterpret_cast<double2*>(C + (bi + g) * kMmaLd + bk + 2 * t);
          double2 v = *d;
          v.x -= c[0];
          v.y -= c[1];
          *d = v;
        }
      }
      if (p == 7 && warp == 7) last_panel();
      // zeros above the diagonal of the inverse: block row p's columns right of the diagonal block
      const int w = kT - base - 8;
      for (int q = tid - 32; q < 8 * w; q += kBandThreads - 32) X[(base + q / w) * kMmaLd + base + 8 + q % w] = 0.0;
    }
    __syncthreads();
  }
  after_panels();
  // zeros above the diagonal blocks of L
  for (int q = tid; q < kTile; q += kBandThreads) {
    const int r = q / kT, c = q % kT;
    if ((c >> 3) > (r >> 3)) C[r * kMmaLd + c] = 0.0;
  }
  // 8 x 8 diagonal inverses: warp w block w, lane c < 8 its column c, by forward substitution
  if (lane < 8) {
    const double* Lb = C + 8 * warp * kMmaLd + 8 * warp;
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      double s = i == lane ? 1.0 : 0.0;
#pragma unroll
      for (int k = 0; k < i; ++k) s -= Lb[i * kMmaLd + k] * x[k];
      x[i] = i < lane ? 0.0 : s * sc.rsq[8 * warp + i];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) X[(8 * warp + i) * kMmaLd + 8 * warp + lane] = x[i];
  }
  __syncthreads();
  inverse_double<1>(C, X, W);
  inverse_double<2>(C, X, W);
  inverse_double<4>(C, X, W);
}

__device__ __forceinline__ void store_tile(double* dst, const double* src) {
  for (int q = threadIdx.x; q < kTile / 2; q += kBandThreads)
    reinterpret_cast<double2*>(dst)[q] =
        *reinterpret_cast<const double2*>(src + (q / (kT / 2)) * kMmaLd + 2 * (q % (kT / 2)));
}

// The diagonal, from the first block row to the last.  The next row's two tiles are fetched while
// this row's factor is inverted, if the workers have them by then.
__device__ void band_chain(const BandWork& B, double* sm) {
  double* As = sm;                  // C_{J,J-1}; the next row's at An
  double* An = sm + kStage;
  double* Cs = sm + 2 * kStage;     // the diagonal tile, then L_JJ; the next row's at Cn
  double* Cn = sm + 3 * kStage;
  double* Ls = sm + 4 * kStage;     // L_{J,J-1}; scratch of the inverse
  double* Xs = sm + 5 * kStage;     // Linv of the block row before, then this one's
  __shared__ TileScratch sc;
  __shared__ int go, early;
  const int tid = threadIdx.x, lane = tid & 31;
  const bool sub = B.bands > 0, need = B.bands >= 2;
  double pmin = INFINITY, pmax = 0.0;
  bool bad = false;
  bool fetched = false;
  if (tid == 0) early = 0;
  auto fetch = [&](int J, double* A, double* C) {
    if (sub && J > 0) stage_tile(A, B.tiles + tile_index(J, 1, B.bands));
    stage_commit();
    stage_tile(C, B.tiles + tile_index(J, 0, B.bands));
    stage_commit();
  };
  for (int J = 0; J < B.n_tiles; ++J) {
    if (!fetched) {
      if (tid == 0) go = J < 2 || !need || wait_for(B.prepared + J, 2, B.abort_flag);
      __syncthreads();
      if (!go) break;
      fetch(J, As, Cs);
    }
    stage_wait<1>();
    __syncthreads();
    TileAcc acc;
    if (sub && J > 0) {
      tile_zero(acc);
      tile_mma<true, false>(As, Xs, acc);   // Linv is lower triangular
      double* G = B.tiles + tile_index(J, 1, B.bands);
      tile_each(kMmaLd, [&](int o, int i, int j) { *reinterpret_cast<double2*>(Ls + o) = make_double2(acc[i][j][0], acc[i][j][1]); });
      tile_each(kT, [&](int o, int i, int j) { *reinterpret_cast<double2*>(G + o) = make_double2(acc[i][j][0], acc[i][j][1]); });
    }
    stage_wait<0>();
    __syncthreads();
    if (sub && J > 0) {
      if (need) publish(B.progress + J, J);
      else __syncthreads();
      tile_syrk(Ls, Cs);
      __syncthreads();
    }
    auto look = [&] {   // is the next row prepared?
      if (lane == 0 && J + 1 < B.n_tiles && (J < 1 || !need || ld_relaxed(B.prepared + J + 1) >= 2)) {
        fence_gpu();
        early = J + 1;
      }
    };
    tile_cholesky(Cs, Xs, Ls, sc, look, [&] {
      fetched = J + 1 < B.n_tiles && early > J;
      if (fetched) fetch(J + 1, An, Cn);
    });
    store_tile(B.inv + (size_t)J * kTile, Xs);
    if (need) publish(B.progress + J, J + 1);
    store_tile(B.tiles + tile_index(J, 0, B.bands), Cs);
    if (tid >= kBandThreads - 32) {   // the last warp: the row's pivots
      for (int i = lane; i < kT; i += 32) {
        if (J * kT + i < B.n) {
          const double p = sc.pivot[i];
          if (p > 0.0) {
            pmin = fmin(pmin, p);
            pmax = fmax(pmax, p);
          } else {
            bad = true;
          }
        }
      }
    }
    if (fetched) {
      double* a = As;
      As = An;
      An = a;
      double* c = Cs;
      Cs = Cn;
      Cn = c;
    }
    __syncthreads();
  }
  if (tid >= kBandThreads - 32) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      pmin = fmin(pmin, __shfl_xor_sync(FEAB_FULL_MASK, pmin, o));
      pmax = fmax(pmax, __shfl_xor_sync(FEAB_FULL_MASK, pmax, o));
    }
    bad = __any_sync(FEAB_FULL_MASK, bad);
    if (lane == 0) {
      B.st->piv_min = (unsigned long long)__double_as_longlong(pmin);
      B.st->piv_max = (unsigned long long)__double_as_longlong(pmax);
      if (bad) B.st->status = FEAB_NOT_SPD;
    }
  }
}

// Tasks of slot J (block column J), bands + 1 of them: 0 the tile (J + 2, J); 1 and 2 the tiles (J + 2,
// J + 1) and (J + 2, J + 2) for the chain; then the tiles (I, J), I = J + 3 .. J + bands.
__device__ void band_worker(const BandWork& B, double* sm) {
  __shared__ int task, ready, go;
  const int tid = threadIdx.x, b = B.bands;
  const long long tasks = b >= 2 ? (long long)B.n_tiles * (b + 1) : 0;
  while (true) {
    if (tid == 0) task = atomicAdd(B.next_task, 1);
    __syncthreads();
    const int tk = task;
    if (tk >= tasks) return;
    const int J = tk / (b + 1), q = tk - J * (b + 1);
    const bool chain_tile = q == 1 || q == 2;
    const int I = J + (q < 3 ? 2 : q);
    const int col = q == 1 ? J + 1 : (q == 2 ? J + 2 : J);
    if (I >= B.n_tiles || (!chain_tile && I - J > b)) {
      __syncthreads();
      continue;
    }
    const int K0 = max(0, I - b), K1 = chain_tile ? J + 1 : J;   // terms K0 .. K1 - 1
    const bool diag = col == I;
    double* G = B.tiles + tile_index(I, I - col, b);
    TileAcc acc;
    double2 c0[2][4];
    tile_each(kT, [&](int o, int i, int j) { c0[i][j] = __ldcg(reinterpret_cast<const double2*>(G + o)); });
    tile_zero(acc);
    int known = 0;   // thread 0: both rows' tiles of columns < known are stored
    auto poll = [&](int want) {
      known = min(ld_relaxed(B.progress + I), ld_relaxed(B.progress + col));
      return known >= want;
    };
    auto block_until = [&](int want) {   // thread 0
      if (known >= want) return true;
      const bool ok = wait_for(B.progress + I, want, B.abort_flag) && wait_for(B.progress + col, want, B.abort_flag);
      known = want;
      return ok;
    };
    auto issue = [&](int K) {
      double* buf = sm + (K & 1) * 2 * kStage;
      stage_tile(buf, B.tiles + tile_index(I, I - K, b));
      if (!diag) stage_tile(buf + kStage, B.tiles + tile_index(col, col - K, b));
      stage_commit();
    };
    bool issued = false;   // the next term's copies are on their way
    for (int K = K0; K < K1; ++K) {
      if (!issued) {
        if (tid == 0) go = block_until(K + 1);
        __syncthreads();
        if (!go) return;
        issue(K);
      }
      if (tid == 0) {
        ready = K + 1 < K1 && known >= K + 2;
        if (!ready && K + 1 < K1 && poll(K + 2)) {
          fence_gpu();
          ready = 1;
        }
      }
      __syncthreads();
      issued = ready;
      if (issued) {
        issue(K + 1);
        stage_wait<1>();
      } else {
        stage_wait<0>();
      }
      __syncthreads();
      const double* buf = sm + (K & 1) * 2 * kStage;
      if (!diag) tile_mma<false, false>(buf, buf + kStage, acc);
      else tile_mma<false, true>(buf, buf, acc);
      __syncthreads();
    }
    if (chain_tile) {
      tile_each(kT, [&](int o, int i, int j) {
        *reinterpret_cast<double2*>(G + o) = make_double2(c0[i][j].x - acc[i][j][0], c0[i][j].y - acc[i][j][1]);
      });
      publish(B.prepared + I, 0);
    } else {
      tile_each(kMmaLd, [&](int o, int i, int j) {
        *reinterpret_cast<double2*>(sm + o) = make_double2(c0[i][j].x - acc[i][j][0], c0[i][j].y - acc[i][j][1]);
      });
      if (tid == 0) go = wait_for(B.progress + J, J + 1, B.abort_flag);
      __syncthreads();
      if (!go) return;
      stage_tile(sm + kStage, B.inv + (size_t)J * kTile);
      stage_commit();
      stage_wait<0>();
      __syncthreads();
      tile_zero(acc);
      tile_mma<true, false>(sm, sm + kStage, acc);   // Linv is lower triangular
      tile_each(kT, [&](int o, int i, int j) {
        *reinterpret_cast<double2*>(G + o) = make_double2(acc[i][j][0], acc[i][j][1]);
      });
      publish(B.progress + I, J + 1);
    }
  }
}

__global__ void __launch_bounds__(kBandThreads, 1) k_band_factor(BandWork B) {
  extern __shared__ __align__(16) double fsm[];
  if (blockIdx.x == 0) band_chain(B, fsm);
  else band_worker(B, fsm);
}

// ---------------------------------------------------------------- solves
// Both triangular solves in one kernel of one cluster.  CTA c of C owns the block rows J = c (mod C).
// Forward, w_J = b_J - sum_K L_JK y_K grows in registers as the y_K come in (each thread keeps its
// share of the sums of its CTA's next P rows, unreduced), and when y_{J-1} is in, the owner of J
// reduces w_J, forms y_J = Linv_JJ w_J and writes it into every CTA's shared memory (st.async, which
// counts the bytes on the receiver's barrier).  Backward the same with L_IJ^T and Linv_JJ^T.  A tile
// is used once, so one more warp streams the tiles in the order of their use through a ring in shared
// memory (bulk copies).
// Vector q + 32 goes where vector q was: every CTA sends a vector between the two (it has a row among
// any 16, and at most 31 vectors lie between its last row forward and its first backward), and it
// has taken in all vectors before the one that it sends.  Every wait is bounded: a CTA whose wait runs out
// goes on without waiting, so that barriers stay matched, sends NaN and sets the solve's error flag.
//
// What bounds it: latency, 1.1 us per block row (two 64 x 64 products by 512 threads, each with its
// reduction, and one hop to another SM), while a CTA's tiles per block row (bands / C) come in
// faster than that; wide bands are bound by what 16 SMs read (about 1.4 TB/s).  Measured, two
// launches per block row -> one kernel, both directions: 64x16x16 elements (867 block rows, 28
// bands) 19.0 -> 2.1 ms (1.84 with the 15 bands of nodes in layers), 96x24x24 (2,813, 59 bands) 63.3 -> 8.3 ms (6.4
// with 31 bands), 33x9x8 (140, 9) 2.07 -> 0.36 ms (0.27 with 5 bands).
constexpr int kSolveWarps = 16;
constexpr int kSolveThreads = 32 * kSolveWarps;       // that compute; one more warp fetches the tiles
constexpr int kSolveCta = kSolveThreads + 32;
constexpr int kSolveRing = 6;                          // tiles
constexpr int kSolveSlots = 32;                        // vectors on their way
constexpr int kSolveMaxCluster = 16;
constexpr int kSolveMaxRows = 8;                       // P: pending rows of a CTA
constexpr int kPartLd = kT + 2;

struct SolveShared {
  double ring[kSolveRing][kTile];
  double vec[kSolveSlots][kT];
  double part[kSolveWarps][kPartLd];
  double w[kT];
  unsigned long long full[kSolveRing], empty[kSolveRing], arrived[kSolveSlots];
  int abort_flag;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* m, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long* m, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(m)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* m) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(m)) : "memory");
}
__device__ __forceinline__ bool mbar_done(unsigned long long* m, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(smem_u32(m)), "r"(parity)
      : "memory");
  return done != 0;
}

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long v;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(v));
  return v;
}
constexpr unsigned long long kSolveLimitNs = 4000000000ull;
constexpr int kSolveLate = 4096;                       // polls beyond it: the context may have been switched out

// False when the wait runs out, or another wait of the CTA has.  (A clock that leaves such time out, and telling
// the other CTAs, each cost the wide bands 2 to 4 %: it is code in every wait.)
__device__ __forceinline__ bool mbar_wait(unsigned long long* m, uint32_t parity, volatile int* abort_flag) {
  const uint32_t a = smem_u32(m);
  unsigned long long began = 0;
  int late = 0;
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n " FEAB_MBAR_TRY ".parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if (*abort_flag || FEAB_WAIT_CYCLES == 0) break;
    if (began == 0) began = now_ns();
    else if (now_ns() - began > kSolveLimitNs && ++late > kSolveLate) break;
  }
  *abort_flag = 1;
  return false;
}
__device__ __forceinline__ void solve_sync() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct SolveArgs {
  const double* tiles;
  const double* inv;
  const double* b;
  double* x;      // y after the forward pass, then the solution
  int32_t* error_flag;
  int32_t bands, n_tiles;
};

// The tiles that CTA c uses, in order, passed to fn(address): forward, for each K, the tiles (J, K) of
// its rows J > K, nearest first, Linv_JJ behind the tile (K + 1, K); backward the mirror image.
template <typename F>
__device__ __forceinline__ void solve_tiles(const SolveArgs& A, int c, int C, F fn) {
  const int b = A.bands, NT = A.n_tiles;
  if (c == 0) fn(A.inv);
  for (int K = 0; K < NT - 1; ++K) {
    int J = K + 1 + (c - (K + 1) % C + C) % C;
    if (J == K + 1) {
      if (b > 0) fn(A.tiles + tile_index(J, 1, b));
      fn(A.inv + (size_t)J * kTile);
      J += C;
    }
    for (; J <= min(K + b, NT - 1); J += C) fn(A.tiles + tile_index(J, J - K, b));
  }
  if (c == (NT - 1) % C) fn(A.inv + (size_t)(NT - 1) * kTile);
  for (int K = NT - 1; K > 0; --K) {
    int J = K - 1 - ((K - 1) % C - c + C) % C;
    if (J == K - 1) {
      if (b > 0) fn(A.tiles + tile_index(K, 1, b));
      fn(A.inv + (size_t)J * kTile);
      J -= C;
    }
    for (; J >= max(K - b, 0); J -= C) fn(A.tiles + tile_index(K, K - J, b));
  }
}

// A thread's eight values of a tile.
struct TilePart {
  double2 t[4];
};
// Forward: thread (rp = tid / 16, h = tid % 16) holds rows 2 rp and 2 rp + 1, columns 2 h + {0, 1, 32, 33}.
__device__ __forceinline__ TilePart fwd_part(const double* T) {
  const int rp = threadIdx.x >> 4, h = threadIdx.x & 15;
  TilePart p;
#pragma unroll
  for (int u = 0; u < 4; ++u)
    p.t[u] = *reinterpret_cast<const double2*>(T + (2 * rp + (u >> 1)) * kT + 32 * (u & 1) + 2 * h);
  return p;
}
__device__ __forceinline__ void fwd_product(const TilePart& p, const double2 (&y)[2], double (&a)[2]) {
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const double s = fma(p.t[2 * u].x, y[0].x, p.t[2 * u].y * y[0].y);
    a[u] = fma(p.t[2 * u + 1].x, y[1].x, fma(p.t[2 * u + 1].y, y[1].y, a[u])) + s;
  }
}
// Sums over the 16 lanes of a row pair: row 2 rp in lanes h < 8, row 2 rp + 1 in the others.
__device__ __forceinline__ double fwd_reduce(const double (&a)[2]) {
  const bool up = (threadIdx.x & 8) != 0;
  double s = (up ? a[1] : a[0]) + __shfl_xor_sync(FEAB_FULL_MASK, up ? a[0] : a[1], 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(FEAB_FULL_MASK, s, o);
  return s;
}
// Backward: lane l holds columns 2 l, 2 l + 1 of rows 4 w .. 4 w + 3 (warp w).
__device__ __forceinline__ TilePart bwd_part(const double* T) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  TilePart p;
#pragma unroll
  for (int u = 0; u < 4; ++u) p.t[u] = *reinterpret_cast<const double2*>(T + (4 * warp + u) * kT + 2 * lane);
  return p;
}
__device__ __forceinline__ void bwd_product(const TilePart& p, const double (&x)[4], double (&a)[2]) {
  const double s0 = fma(p.t[0].x, x[0], p.t[1].x * x[1]), s1 = fma(p.t[0].y, x[0], p.t[1].y * x[1]);
  a[0] = fma(p.t[2].x, x[2], fma(p.t[3].x, x[3], a[0])) + s0;
  a[1] = fma(p.t[2].y, x[2], fma(p.t[3].y, x[3], a[1])) + s1;
}
// Sums over the warps: column tid / 8, in its eight lanes.
__device__ __forceinline__ double bwd_reduce(SolveShared& S, const double (&a)[2]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, col = threadIdx.x >> 3, h = threadIdx.x & 7;
  *reinterpret_cast<double2*>(&S.part[warp][2 * lane]) = make_double2(a[0], a[1]);
  solve_sync();
  double s = S.part[h][col] + S.part[h + 8][col];
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(FEAB_FULL_MASK, s, o);
  return s;
}

template <int P>
__global__ void __launch_bounds__(kSolveCta, 1) k_band_solve(SolveArgs A) {
  extern __shared__ __align__(128) unsigned char solve_dyn[];
  SolveShared& S = *reinterpret_cast<SolveShared*>(solve_dyn);
  const int tid = threadIdx.x, C = gridDim.x, c = blockIdx.x, b = A.bands, NT = A.n_tiles;
  volatile int* abort_flag = &S.abort_flag;
  if (tid == 0) {
    S.abort_flag = 0;
    for (int i = 0; i < kSolveRing; ++i) {
      mbar_init(&S.full[i], 1);
      mbar_init(&S.empty[i], kSolveWarps);
    }
    for (int i = 0; i < kSolveSlots; ++i) {
      mbar_init(&S.arrived[i], 1);
      mbar_expect(&S.arrived[i], kT * 8);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  cluster_sync_all();
  int issued = 0;   // tiles (the fetching thread)
  if (tid >= kSolveThreads) {
    // the tiles, each into the next free place of the ring
    if ((tid & 31) == 0) {
      int slot = 0;
      uint32_t phase = 0;
      bool ok = true;
      solve_tiles(A, c, C, [&](const double* src) {
        if (!ok) return;
        // a warp that gave up on a tile leaves its place all the same: the tile may still be on its way
        ok = mbar_wait(&S.empty[slot], phase ^ 1, abort_flag) && !*abort_flag;
        if (!ok) return;
        ++issued;
        mbar_expect(&S.full[slot], kTile * 8);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         smem_u32(S.ring[slot])),
                     "l"(src), "r"((uint32_t)(kTile * 8)), "r"(smem_u32(&S.full[slot]))
                     : "memory");
        if (++slot == kSolveRing) {
          slot = 0;
          phase ^= 1;
        }
      });
    }
  } else {
    const int warp = tid >> 5, lane = tid & 31, rp = tid >> 4, h = tid & 15;
    int slot = 0;
    uint32_t phase = 0;
    bool ok = true;
    auto tile = [&] {
      ok = ok && mbar_wait(&S.full[slot], phase, abort_flag);
      return (const double*)S.ring[slot];
    };
    auto release = [&] {
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.empty[slot]);
      if (++slot == kSolveRing) {
        slot = 0;
        phase ^= 1;
      }
    };
    // vector number q of the solve (y_0 .. y_{NT-1}, then x_{NT-1} .. x_0), entry i = v of this thread's
    // eight lanes, to every CTA: with the neighbours' entry, each of the 16 lanes of two entries sends
    // both to one CTA
    auto send = [&](int q, int i, double v) {
      const double other = __shfl_xor_sync(FEAB_FULL_MASK, v, 8);
      const int r = lane & 15;
      const bool up = (lane & 8) != 0;
      if (r < C) {
        const uint32_t dst = smem_u32(&S.vec[q % kSolveSlots][i & ~1]), bar = smem_u32(&S.arrived[q % kSolveSlots]);
        uint32_t rd, rb;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rd) : "r"(dst), "r"(r));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rb) : "r"(bar), "r"(r));
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(rd),
                     "l"(__double_as_longlong(up ? other : v)), "l"(__double_as_longlong(up ? v : other)), "r"(rb)
                     : "memory");
      }
    };
    auto receive = [&](int q) {
      ok = ok && mbar_wait(&S.arrived[q % kSolveSlots], (q / kSolveSlots) & 1, abort_flag);
      if (tid == 0 && ok) mbar_expect(&S.arrived[q % kSolveSlots], kT * 8);
      return (const double*)S.vec[q % kSolveSlots];
    };
    double acc[P][2];
    auto shift = [&] {
#pragma unroll
      for (int p = 0; p + 1 < P; ++p) {
        acc[p][0] = acc[p + 1][0];
        acc[p][1] = acc[p + 1][1];
      }
      acc[P - 1][0] = acc[P - 1][1] = 0.0;
    };
#pragma unroll
    for (int p = 0; p < P; ++p) acc[p][0] = acc[p][1] = 0.0;
    // ---- forward
    // The tile (J, J - 1) and Linv_JJ are in registers before y_{J-1} arrives.
    const int frow = 2 * rp + (h >> 3);
    double rhs = c < NT ? A.b[(size_t)c * kT + frow] : 0.0;   // of the CTA's next row
    TilePart sub{}, diag{};
    auto load_fwd = [&](bool with_sub) {
      if (with_sub) {
        sub = fwd_part(tile());
        release();
      }
      diag = fwd_part(tile());
      release();
    };
    auto finish_fwd = [&](int J) {
      const double wv = rhs - fwd_reduce(acc[0]);
      if ((h & 7) == 0) S.w[frow] = wv;
      solve_sync();
      const double2 w2[2] = {*reinterpret_cast<const double2*>(&S.w[2 * h]),
                             *reinterpret_cast<const double2*>(&S.w[32 + 2 * h])};
      double a[2] = {0.0, 0.0};
      fwd_product(diag, w2, a);
      const double sum = fwd_reduce(a), y = ok ? sum : __longlong_as_double(0x7ff8000000000000ll);
      send(J, frow, y);
      if ((h & 7) == 0) A.x[(size_t)J * kT + frow] = y;
      shift();
      if (J + C < NT) rhs = A.b[(size_t)(J + C) * kT + frow];
    };
    if (c == 0) {
      load_fwd(false);
      finish_fwd(0);
    }
    for (int K = 0; K < NT; ++K) {
      int J = K + 1 + (c - (K + 1) % C + C) % C;
      const bool mine = J == K + 1 && J < NT;
      if (mine) load_fwd(b > 0);
      const double* v = receive(K);
      if (K == NT - 1) break;
      const double2 y[2] = {*reinterpret_cast<const double2*>(v + 2 * h),
                            *reinterpret_cast<const double2*>(v + 32 + 2 * h)};
      if (mine) {
        if (b > 0) fwd_product(sub, y, acc[0]);
        finish_fwd(J);
        J += C;
      }
      const int last = min(K + b, NT - 1);
#pragma unroll
      for (int p = 0; p < P; ++p) {
        if (J + p * C <= last) {
          fwd_product(fwd_part(tile()), y, acc[p]);
          release();
        }
      }
    }
    // ---- backward
    asm volatile("bar.sync 1, 512;" ::: "memory");
#pragma unroll
    for (int p = 0; p < P; ++p) acc[p][0] = acc[p][1] = 0.0;
    const int col = tid >> 3;
    const int top = NT - 1 - ((NT - 1) % C - c + C) % C;   // the CTA's last row (negative: none)
    if (top >= 0) rhs = __ldcg(A.x + (size_t)top * kT + col);
    auto load_bwd = [&](bool with_sub) {
      if (with_sub) {
        sub = bwd_part(tile());
        release();
      }
      diag = bwd_part(tile());
      release();
    };
    auto finish_bwd = [&](int J) {
      const double wv = rhs - bwd_reduce(S, acc[0]);
      if ((tid & 7) == 0) S.w[col] = wv;
      solve_sync();
      const double wr[4] = {S.w[4 * warp], S.w[4 * warp + 1], S.w[4 * warp + 2], S.w[4 * warp + 3]};
      double a[2] = {0.0, 0.0};
      bwd_product(diag, wr, a);
      const double sum = bwd_reduce(S, a), xv = ok ? sum : __longlong_as_double(0x7ff8000000000000ll);
      send(2 * NT - 1 - J, col, xv);
      if ((tid & 7) == 0) A.x[(size_t)J * kT + col] = xv;
      shift();
      if (J - C >= 0) rhs = __ldcg(A.x + (size_t)(J - C) * kT + col);
    };
    if (top == NT - 1) {
      load_bwd(false);
      finish_bwd(NT - 1);
    }
    for (int K = NT - 1; K > 0; --K) {
      int J = K - 1 - ((K - 1) % C - c + C) % C;
      const bool mine = J == K - 1;
      if (mine) load_bwd(b > 0);
      const double* v = receive(2 * NT - 1 - K);
      const double xr[4] = {v[4 * warp], v[4 * warp + 1], v[4 * warp + 2], v[4 * warp + 3]};
      if (mine) {
        if (b > 0) bwd_product(sub, xr, acc[0]);
        finish_bwd(J);
        J -= C;
      }
      const int last = max(K - b, 0);
#pragma unroll
      for (int p = 0; p < P; ++p) {
        if (J - p * C >= last) {
          bwd_product(bwd_part(tile()), xr, acc[p]);
          release();
        }
      }
    }
    receive(2 * NT - 1);   // x_0: nothing is on its way to this CTA when it leaves
  }
  __syncwarp();
  cluster_sync_all();
  if (*abort_flag) {
    // what nobody waited for may still be on its way into this CTA's memory: the tiles, and 0.1 ms for vectors
    for (int i = 0; i < kSolveRing; ++i) {
      const int uses = issued / kSolveRing + (i < issued % kSolveRing ? 1 : 0);
      DrainLimit limit;
      while (uses > 0 && !mbar_done(&S.full[i], (uses - 1) & 1) && !limit.over()) {
      }
    }
    for (const long long t0 = clock64(); clock64() - t0 < 200000;) {
    }
    if (tid == 0) *A.error_flag = 1;
  }
}

// Wider bands than the cluster kernel's pending rows, or no place for the cluster: one launch per block row.
// Forward step K of L y = b: every CTA forms y_K = Linv_KK w_K (two threads per row), CTA 0 writes
// it, and CTA i < n_below applies tile (K + 1 + i, i + 1): w_{K+1+i} -= L_{K+1+i,K} y_K.
__global__ void __launch_bounds__(128) k_band_fwd(const double* __restrict__ tiles, const double* __restrict__ inv,
                                                 int bands, int K, int n_below, double* __restrict__ w,
                                                 double* __restrict__ y) {
  __shared__ double wk[kT];
  __shared__ double ys[kT];
  if (threadIdx.x < kT) wk[threadIdx.x] = w[K * kT + threadIdx.x];
  __syncthreads();
  const int r = threadIdx.x >> 1, h = threadIdx.x & 1;
  const double* Iv = inv + (size_t)K * kTile;
  double s = 0.0;
#pragma unroll 8
  for (int c = 32 * h; c < 32 * h + 32; ++c) s += Iv[r * kT + c] * wk[c];
  s += __shfl_xor_sync(FEAB_FULL_MASK, s, 1);
  if (h == 0) ys[r] = s;
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x < kT) y[K * kT + threadIdx.x] = ys[threadIdx.x];
  if ((int)blockIdx.x < n_below) {
    const int I = K + 1 + blockIdx.x;
    const double* T = tiles + tile_index(I, I - K, bands);
    double t = 0.0;
#pragma unroll 8
    for (int c = 32 * h; c < 32 * h + 32; ++c) t += T[(size_t)r * kT + c] * ys[c];
    t += __shfl_xor_sync(FEAB_FULL_MASK, t, 1);
    if (h == 0) w[I * kT + r] -= t;
  }
}

// Backward step K of L^T x = y: every CTA forms x_K = Linv_KK^T w_K (two threads per column), CTA
// 0 writes it, and CTA i < n_above applies tile (K, i + 1) transposed: w_{K-1-i} -= L_{K,K-1-i}^T
// x_K.
__global__ void __launch_bounds__(128) k_band_bwd(const double* __restrict__ tiles, const double* __restrict__ inv,
                                                 int bands, int K, int n_above, double* __restrict__ w,
                                                 double* __restrict__ x) {
  __shared__ double wk[kT];
  __shared__ double xs[kT];
  if (threadIdx.x < kT) wk[threadIdx.x] = w[K * kT + threadIdx.x];
  __syncthreads();
  const int c = threadIdx.x >> 1, h = threadIdx.x & 1;
  const double* Iv = inv + (size_t)K * kTile;
  double s = 0.0;
#pragma unroll 8
  for (int r = 32 * h; r < 32 * h + 32; ++r) s += Iv[r * kT + c] * wk[r];
  s += __shfl_xor_sync(FEAB_FULL_MASK, s, 1);
  if (h == 0) xs[c] = s;
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x < kT) x[K * kT + threadIdx.x] = xs[threadIdx.x];
  if ((int)blockIdx.x < n_above) {
    const int J = K - 1 - blockIdx.x;
    const double* T = tiles + tile_index(K, K - J, bands);
    double t = 0.0;
#pragma unroll 8
    for (int r = 32 * h; r < 32 * h + 32; ++r) t += T[(size_t)r * kT + c] * xs[r];
    t += __shfl_xor_sync(FEAB_FULL_MASK, t, 1);
    if (h == 0) w[J * kT + c] -= t;
  }
}

}  // namespace
}  // namespace feab


using namespace feab;

namespace {
BandState* band_state(const feab_band* B) { return reinterpret_cast<BandState*>(B->storage); }
double* band_tiles(const feab_band* B) {
  return reinterpret_cast<double*>(static_cast<char*>(B->storage) + FEAB_BAND_HEADER_BYTES);
}
// The inverses of the diagonal factor tiles, one per block row, after the band.
double* band_inv(const feab_band* B) {
  return band_tiles(B) + (size_t)B->n_tiles * (size_t)(B->bands + 1) * kTile;
}
// progress and prepared, two counters per block row, in use with two bands or more while the factorisation
// runs: in the tiles of block row 0 that lie left of the matrix (bands tiles, never read), behind the
// inverses when there are more counters than those hold.
size_t band_flag_bytes(int32_t n_tiles, int32_t bands) {
  return bands >= 2 ? 2 * (size_t)n_tiles * sizeof(int32_t) : 0;
}
bool band_flags_inside(int32_t n_tiles, int32_t bands) {
  return band_flag_bytes(n_tiles, bands) <= (size_t)bands * kTile * sizeof(double);
}
int32_t* band_flags(const feab_band* B) {
  return reinterpret_cast<int32_t*>(band_flags_inside(B->n_tiles, B->bands) ? band_tiles(B) + kTile
                                                                            : band_inv(B) + (size_t)B->n_tiles * kTile);
}
bool band_ok(const feab_band* B) {
  return B && B->storage && B->n > 0 && B->bands >= 0 && B->n_tiles == (B->n + kT - 1) / kT &&
         (reinterpret_cast<uintptr_t>(B->storage) & 255) == 0;
}
}  // namespace

extern "C" size_t feab_band_bytes(int32_t n, int32_t bandwidth) {
  if (n <= 0 || bandwidth < 0) return 0;
  const size_t nt = (size_t)(n + kT - 1) / kT, bands = (size_t)(bandwidth + kT - 1) / kT;
  const size_t flags = band_flags_inside((int32_t)nt, (int32_t)bands) ? 0 : band_flag_bytes((int32_t)nt, (int32_t)bands);
  return FEAB_BAND_HEADER_BYTES + nt * (bands + 2) * (size_t)kTile * sizeof(double) + flags;
}

extern "C" int32_t feab_band_width(const feab_csr* A, const int32_t* iperm, int32_t* scratch, int32_t* bandwidth_out,
                                   cudaStream_t s) {
  if (!A || !iperm || !scratch || !bandwidth_out || A->n <= 0 || !A->row_ptr || !A->col_idx) return FEAB_BAD_ARG;
  FEAB_CUDA(cudaMemsetAsync(scratch, 0, 2 * sizeof(int32_t), s));
  const int threads = 256, rows = threads / 32;
  k_band_width<<<(A->n + rows - 1) / rows, threads, 0, s>>>(A->row_ptr, A->col_idx, A->n, iperm, scratch, scratch + 1);
  count_launches(1);
  FEAB_CHECK_LAUNCH();
  int32_t h[2] = {0, 0};
  FEAB_CUDA(cudaMemcpyAsync(h, scratch, sizeof(h), cudaMemcpyDeviceToHost, s));
  FEAB_CUDA(cudaStreamSynchronize(s));
  if (h[1]) return FEAB_BAD_ARG;
  *bandwidth_out = h[0];
  return FEAB_OK;
}

extern "C" int32_t feab_band_assemble(const feab_csr* A, const int32_t* iperm, int32_t bandwidth, feab_band* B,
                                      cudaStream_t s) {
  if (!A || !iperm || !B || A->n <= 0 || !A->row_ptr || !A->col_idx || !A->vals64 || bandwidth < 0) return FEAB_BAD_ARG;
  B->n = A->n;
  B->n_tiles = (A->n + kT - 1) / kT;
  B->bands = (bandwidth + kT - 1) / kT;
  if (!band_ok(B)) return FEAB_BAD_ARG;
  FEAB_CUDA(cudaMemsetAsync(B->storage, 0, feab_band_bytes(A->n, bandwidth), s));
  BandState* st = band_state(B);
  const int threads = 256, rows = threads / 32;
  k_band_scatter<<<(A->n + rows - 1) / rows, threads, 0, s>>>(A->row_ptr, A->col_idx, A->vals64, A->n, iperm, B->bands,
                                                             band_tiles(B), &st->bad);
  const int pad = B->n_tiles * kT - A->n;
  if (pad > 0) k_band_pad<<<1, kT, 0, s>>>(A->n, B->n_tiles, B->bands, band_tiles(B));
  count_launches(pad > 0 ? 2 : 1);
  FEAB_CHECK_LAUNCH();
  int32_t bad = 0;
  FEAB_CUDA(cudaMemcpyAsync(&bad, &st->bad, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  FEAB_CUDA(cudaStreamSynchronize(s));
  return bad ? FEAB_BAD_ARG : FEAB_OK;
}

extern "C" int32_t feab_band_cholesky(feab_band* B, double* pivots_out, cudaStream_t s) {
  if (!band_ok(B)) return FEAB_BAD_ARG;
  BandState init{};
  init.piv_min = 0x7ff0000000000000ull;  // +inf
  init.piv_max = 0ull;
  BandState* st = band_state(B);
  FEAB_CUDA(cudaMemcpyAsync(st, &init, sizeof(BandState), cudaMemcpyHostToDevice, s));
  const size_t flag_bytes = band_flag_bytes(B->n_tiles, B->bands);
  if (flag_bytes) FEAB_CUDA(cudaMemsetAsync(band_flags(B), 0, flag_bytes, s));
  BandWork W{};
  W.tiles = band_tiles(B);
  W.inv = band_inv(B);
  W.st = st;
  W.progress = band_flags(B);
  W.prepared = W.progress + B->n_tiles;
  W.next_task = &st->next_task;
  W.abort_flag = &st->abort_flag;
  W.n = B->n;
  W.n_tiles = B->n_tiles;
  W.bands = B->bands;
  FEAB_CUDA(cudaFuncSetAttribute(k_band_factor, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFactorSmem));
  // one CTA per SM: the chain and, with two bands or more, at least one worker
  int resident = 0;
  FEAB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, k_band_factor, kBandThreads, kFactorSmem));
  const int64_t tasks = B->bands >= 2 ? (int64_t)B->n_tiles * (B->bands + 1) : 0;
  int grid = (int)std::min<int64_t>((int64_t)sm_count() * std::min(resident, 1), 1 + tasks);
  const int least = tasks > 0 ? 2 : 1;
  if (grid < least) return FEAB_CUDA_ERROR;
  void* args[1] = {&W};
  // a context with fewer SMs at hand than the device has: any number of workers does
  cudaError_t e;
  while ((e = cudaLaunchCooperativeKernel((const void*)k_band_factor, dim3(grid), dim3(kBandThreads), args, kFactorSmem,
                                          s)) == cudaErrorCooperativeLaunchTooLarge &&
         grid > least) {
    cudaGetLastError();
    grid = std::max(least, grid / 2);
  }
  FEAB_CUDA(e);
  count_launches(1);
  FEAB_CHECK_LAUNCH();
  if (flag_bytes) FEAB_CUDA(cudaMemsetAsync(band_flags(B), 0, flag_bytes, s));   // left as it was
  BandState h{};
  FEAB_CUDA(cudaMemcpyAsync(&h, st, sizeof(BandState), cudaMemcpyDeviceToHost, s));
  FEAB_CUDA(cudaStreamSynchronize(s));
  if (pivots_out) {
    double lo, hi;
    std::memcpy(&lo, &h.piv_min, sizeof(double));
    std::memcpy(&hi, &h.piv_max, sizeof(double));
    pivots_out[0] = lo;
    pivots_out[1] = hi;
  }
  if (h.abort_flag) return FEAB_CUDA_ERROR;
  return h.status == FEAB_OK ? FEAB_OK : h.status;
}

extern "C" int32_t feab_band_solve(const feab_band* B, const double* b, double* x, double* work, cudaStream_t s) {
  return feab_band_solve_flag(B, b, x, work, B && B->storage ? &band_state(B)->solve_error : nullptr, s);
}

extern "C" int32_t feab_band_solve_flag(const feab_band* B, const double* b, double* x, double* work,
                                        int32_t* error_flag, cudaStream_t s) {
  if (!band_ok(B) || !b || !x || !work || !error_flag || x == b || x == work || b == work) return FEAB_BAD_ARG;
  const double* tiles = band_tiles(B);
  const double* inv = band_inv(B);
  const int NT = B->n_tiles, bands = B->bands;
  // A CTA's pending rows, bands / C, are registers; up to 8 bands one portable cluster has a tile per
  // CTA and block row.
  const int C = bands > 8 ? kSolveMaxCluster : 8, rows = (bands + C - 1) / C;
  if (rows <= kSolveMaxRows) {
    SolveArgs A{tiles, inv, b, x, error_flag, bands, NT};
    const void* fn = rows <= 1 ? (const void*)k_band_solve<1> : rows <= 2 ? (const void*)k_band_solve<2>
                   : rows <= 4 ? (const void*)k_band_solve<4> : (const void*)k_band_solve<kSolveMaxRows>;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(kSolveCta);
    cfg.dynamicSmemBytes = sizeof(SolveShared);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    void* args[1] = {&A};
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SolveShared));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaLaunchKernelExC(&cfg, fn, args);
    if (e == cudaSuccess) {
      count_launches(1);
      return FEAB_OK;
    }
    cudaGetLastError();   // the cluster has no place (a part of a device): a launch per block row needs none
  }
  const size_t bytes = (size_t)NT * kT * sizeof(double);
  // forward: work = b, updated in place; y into x
  FEAB_CUDA(cudaMemcpyAsync(work, b, bytes, cudaMemcpyDeviceToDevice, s));
  for (int K = 0; K < NT; ++K) {
    const int below = std::min(bands, NT - 1 - K);
    k_band_fwd<<<std::max(1, below), 128, 0, s>>>(tiles, inv, bands, K, below, work, x);
  }
  // backward: x (= y) updated in place; the solution into work, then copied to x
  for (int K = NT - 1; K >= 0; --K) {
    const int above = std::min(bands, K);
    k_band_bwd<<<std::max(1, above), 128, 0, s>>>(tiles, inv, bands, K, above, x, work);
  }
  count_launches(2 * (uint64_t)NT);
  FEAB_CHECK_LAUNCH();
  FEAB_CUDA(cudaMemcpyAsync(x, work, bytes, cudaMemcpyDeviceToDevice, s));
  // rows past n are identity rows with b = 0, so x is 0 there
  return FEAB_OK;
}
