// Dense products of tall row-major panels with small matrices, in FP64 on the CUDA cores, for
// the Rayleigh-Ritz steps of the modal subspace iteration and for forming POD modes:
//   feab_panel_gram:   C = X^T Y  (X, Y: n x k panels, k <= 64; C: k x k)
//   feab_panel_small:  Z = Y V    (Y: n x k panel, V: k x m, m <= 64; Z: n x m panel)
// The reference forms these with dense NumPy/LAPACK products (solver.py:2047-2114 through
// scipy's eigsh, rom_engine/src/rom_engine/pod.py:140-160).  Both stream the panels once; the
// Gram reduces per-CTA partials in a fixed order, so its result is deterministic.
#include <algorithm>
#include "feab_common.cuh"

namespace feab {
namespace {

constexpr int kP = 64;         // largest panel width
constexpr int kPTile = 32;     // rows per staged tile
constexpr int kPThreads = 256;
constexpr int kPReduceWarps = 8;

// Stage rows [r0, r0 + kPTile) of an n x k panel (leading dimension ld) into a kPTile x 64
// shared tile, zero beyond n and beyond column k.
__device__ __forceinline__ void stage_tile(const double* __restrict__ A, int64_t n, int k, int ld, int64_t r0,
                                           double* __restrict__ t) {
  for (int e = threadIdx.x; e < kPTile * kP; e += kPThreads) {
    const int r = e >> 6, c = e & 63;
    t[e] = (r0 + r < n && c < k) ? __ldcs(A + (r0 + r) * (int64_t)ld + c) : 0.0;
  }
}

// One CTA per SM: thread (rg, bi, bj) owns C[bi + 8u][bj + 8v] (u, v < 8) over the rows
// r = rg (mod 4) of each tile; the 4 row groups are summed in a fixed order, CTAs by
// k_panel_gram_reduce.
__global__ void __launch_bounds__(kPThreads, 1) k_panel_gram(const double* __restrict__ X, int ldx,
                                                            const double* __restrict__ Y, int ldy, int64_t n, int k,
                                                            double* __restrict__ part) {
  __shared__ double xs[kPTile * kP];
  __shared__ double ys[kPTile * kP];
  const int tid = threadIdx.x, rg = tid >> 6, t = tid & 63, bi = t >> 3, bj = t & 7;
  double acc[8][8];
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < 8; ++v) acc[u][v] = 0.0;
  const int64_t tiles = (n + kPTile - 1) / kPTile;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    __syncthreads();
    stage_tile(X, n, k, ldx, tile * kPTile, xs);
    stage_tile(Y, n, k, ldy, tile * kPTile, ys);
    __syncthreads();
    for (int r = rg; r < kPTile; r += 4) {
      double a[8], b[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        a[u] = xs[r * kP + bi + 8 * u];
        b[u] = ys[r * kP + bj + 8 * u];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int v = 0; v < 8; ++v) acc[u][v] = fma(a[u], b[v], acc[u][v]);
    }
  }
  // the 64 x 64 partial of this CTA, row groups summed in order; rows 0..31 go to xs and
  // rows 32..63 to ys (together 64 x 64 doubles)
  double* red = xs;
  for (int g = 0; g < 4; ++g) {
    __syncthreads();
    if (rg == g) {
#pragma unroll
      for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          const int row = bi + 8 * u, col = bj + 8 * v;
          double* cell = (row < kPTile ? red + row * kP : ys + (row - kPTile) * kP) + col;
          *cell = g == 0 ? acc[u][v] : *cell + acc[u][v];
        }
    }
  }
  __syncthreads();
  for (int e = tid; e < kP * kP; e += kPThreads) {
    const int row = e >> 6, col = e & 63;
    part[(int64_t)blockIdx.x * kP * kP + e] = row < kPTile ? xs[row * kP + col] : ys[(row - kPTile) * kP + col];
  }
}

// C[i][j] = sum over CTAs of part[cta][i][j] (i, j < k), one warp per entry, fixed order.
__global__ void __launch_bounds__(32 * kPReduceWarps) k_panel_gram_reduce(const double* __restrict__ part, int ctas,
                                                                         int k, double* __restrict__ C) {
  const int idx = blockIdx.x * kPReduceWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (idx >= k * k) return;
  const int i = idx / k, j = idx % k;
  double s = 0.0;
  for (int c = lane; c < ctas; c += 32) s += __ldg(part + (int64_t)c * kP * kP + i * kP + j);
  s = warp_sum(s);
  if (lane == 0) C[idx] = s;
}

// Z = Y V, Y of FP64 or FP32 values, on the FP64 tensor path (mma.sync m8n8k4): a warp forms eight rows and
// up to 16 columns at a time, with V's fragments in registers for the whole launch.  Lane l reads four
// adjacent values of row l / 4 of Y for each 16 columns of it, from k = 16 kb + 4 (l % 4), and step s of
// that block multiplies the four lanes' s-th values, k = 16 kb + 4 (l % 4) + s, so a row's 16 values
// are one or two sectors and nothing passes through shared memory.  More than 16 columns are
// more column groups (gridDim.y), each of which reads Y.  What bounds it: reading Y once (16 us
// at 418,176 x 64 FP32) and the tensor rate (23 us).  Measured there with m = 10: 303 us when every
// output read its row of Y from L1 by itself, 152 us with rows and V staged in shared memory.
constexpr int kSmallSteps = kP / 4;

__device__ __forceinline__ void panel_dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// The lane's 16 values of a row: four adjacent ones of each 16 columns; zeros past column k and for no row.
// VEC: 64 columns, rows at multiples of 16 bytes.
template <typename T, bool VEC>
__device__ __forceinline__ void panel_row(const T* __restrict__ row, bool valid, int k, int t, T (&y)[16]) {
#pragma unroll
  for (int kb = 0; kb < 4; ++kb) {
    const int c = 16 * kb + 4 * t;
    if constexpr (VEC && sizeof(T) == 4) {
      const float4 v = valid ? __ldcs(reinterpret_cast<const float4*>(row + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
      y[4 * kb] = v.x;
      y[4 * kb + 1] = v.y;
      y[4 * kb + 2] = v.z;
      y[4 * kb + 3] = v.w;
    } else if constexpr (VEC) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double2 v = valid ? __ldcs(reinterpret_cast<const double2*>(row + c) + h) : make_double2(0.0, 0.0);
        y[4 * kb + 2 * h] = v.x;
        y[4 * kb + 2 * h + 1] = v.y;
      }
    } else {
#pragma unroll
      for (int s = 0; s < 4; ++s) y[4 * kb + s] = valid && c + s < k ? __ldcs(row + c + s) : T(0);
    }
  }
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(kPThreads) k_panel_small(const T* __restrict__ Y, int ldy, int64_t n, int k,
                                                          const double* __restrict__ V, int m, double* __restrict__ Z,
                                                          int ldz) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, c0 = 16 * blockIdx.y;
  double b[2][kSmallSteps];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int q = 0; q < kSmallSteps; ++q) {
      const int r = 16 * (q >> 2) + 4 * t + (q & 3), c = c0 + 8 * j + g;
      b[j][q] = r < k && c < m ? V[r * m + c] : 0.0;
    }
  const int64_t step = 8 * ((int64_t)gridDim.x * (kPThreads / 32));
  int64_t r = 8 * ((int64_t)blockIdx.x * (kPThreads / 32) + (threadIdx.x >> 5)) + g;
  T y[16];
  panel_row<T, VEC>(Y + r * ldy, r < n, k, t, y);
  for (; r - g < n; r += step) {
    T next[16];
    panel_row<T, VEC>(Y + (r + step) * ldy, r + step < n, k, t, next);
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
    for (int q = 0; q < kSmallSteps; ++q) {
      panel_dmma(acc[0], (double)y[q], b[0][q]);
      panel_dmma(acc[1], (double)y[q], b[1][q]);
    }
    if (r < n) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int c = c0 + 8 * j + 2 * t;
        if (c < m) Z[r * ldz + c] = acc[j][0];
        if (c + 1 < m) Z[r * ldz + c + 1] = acc[j][1];
      }
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) y[q] = next[q];
  }
}

template <typename T>
int32_t launch_panel_small(const T* Y, int32_t ldy, int64_t n, int32_t k, const double* V, int32_t m, double* Z,
                           int32_t ldz, cudaStream_t s) {
  if (!Y || !V || !Z || n <= 0 || k < 1 || k > kP || m < 1 || m > kP || ldy < k || ldz < m ||
      static_cast<const void*>(Y) == Z)
    return FEAB_BAD_ARG;
  const int64_t groups = (n + 7) / 8, blocks = (groups + kPThreads / 32 - 1) / (kPThreads / 32);
  const dim3 grid((unsigned)std::min<int64_t>(blocks, 4 * (int64_t)sm_count()), (m + 15) / 16);
  const bool vec = k == kP && (reinterpret_cast<uintptr_t>(Y) & 15) == 0 && (ldy * sizeof(T)) % 16 == 0;
  if (vec) k_panel_small<T, true><<<grid, kPThreads, 0, s>>>(Y, ldy, n, k, V, m, Z, ldz);
  else k_panel_small<T, false><<<grid, kPThreads, 0, s>>>(Y, ldy, n, k, V, m, Z, ldz);
  count_launches(1);
  FEAB_CHECK_LAUNCH();
  return FEAB_OK;
}

int panel_grid(int64_t n) {
  const int64_t tiles = (n + kPTile - 1) / kPTile;
  return (int)std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)sm_count()));
}

}  // namespace
}  // namespace feab

using namespace feab;

extern "C" size_t feab_panel_gram_workspace_bytes(int64_t n) {
  if (n <= 0) return 0;
  return sizeof(double) * (size_t)panel_grid(n) * kP * kP;
}

extern "C" int32_t feab_panel_gram(const double* X, int32_t ldx, const double* Y, int32_t ldy, int64_t n, int32_t k,
                                   double* C, void* workspace, size_t workspace_bytes, cudaStream_t s) {
  if (!X || !Y || !C || !workspace || n <= 0 || k < 1 || k > kP || ldx < k || ldy < k) return FEAB_BAD_ARG;
  if (feab_panel_gram_workspace_bytes(n) > workspace_bytes) return FEAB_BAD_ARG;
  const int grid = panel_grid(n);
  double* part = static_cast<double*>(workspace);
  k_panel_gram<<<grid, kPThreads, 0, s>>>(X, ldx, Y, ldy, n, k, part);
  k_panel_gram_reduce<<<(k * k + kPReduceWarps - 1) / kPReduceWarps, 32 * kPReduceWarps, 0, s>>>(part, grid, k, C);
  count_launches(2);
  FEAB_CHECK_LAUNCH();
  return FEAB_OK;
}

extern "C" int32_t feab_panel_small(const double* Y, int32_t ldy, int64_t n, int32_t k, const double* V, int32_t m,
                                    double* Z, int32_t ldz, cudaStream_t s) {
  return launch_panel_small(Y, ldy, n, k, V, m, Z, ldz, s);
}

extern "C" int32_t feab_panel_small_f32(const float* Y, int32_t ldy, int64_t n, int32_t k, const double* V, int32_t m,
                                        double* Z, int32_t ldz, cudaStream_t s) {
  return launch_panel_small(Y, ldy, n, k, V, m, Z, ldz, s);
}
