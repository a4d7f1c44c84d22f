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

// Z = Y V, Y of FP64 or FP32 values: a CTA stages 128 rows of Y (padded, so that a warp's 32 rows read
// one column without bank conflicts) and V in shared memory; thread (row, half) forms eight columns
// of its row at a time, the sums over j in order.  What bounds it: reading Y once (33 us at 418,176 x
// 64 FP64) and, close behind, the shared-memory reads (V's values are broadcasts, two per read).
// Measured there with m = 10: 303 us when every output read its row of Y from L1 by itself.
constexpr int kSmallRows = 128;
constexpr int kSmallLd = kP + 1;
constexpr size_t kSmallSmem = sizeof(double) * (kSmallRows * kSmallLd + kP * kP);

template <typename T>
__global__ void __launch_bounds__(kPThreads) k_panel_small(const T* __restrict__ Y, int ldy, int64_t n, int k,
                                                          const double* __restrict__ V, int m, double* __restrict__ Z,
                                                          int ldz) {
  extern __shared__ __align__(16) double small_sm[];
  double* vs = small_sm;                  // vs[j * mp + c], mp = m rounded up to 8, zeros past m
  double* ys = small_sm + kP * kP;        // ys[r * kSmallLd + j]
  const int tid = threadIdx.x, mp = (m + 7) & ~7;
  for (int e = tid; e < k * mp; e += kPThreads) {
    const int j = e / mp, c = e - j * mp;
    vs[e] = c < m ? V[j * m + c] : 0.0;
  }
  const int r = tid & (kSmallRows - 1), h = tid / kSmallRows;
  for (int64_t r0 = (int64_t)blockIdx.x * kSmallRows; r0 < n; r0 += (int64_t)gridDim.x * kSmallRows) {
    __syncthreads();
    const int rows = (int)min((int64_t)kSmallRows, n - r0);
    for (int e = tid; e < kSmallRows * kP; e += kPThreads) {
      const int i = e / kP, j = e % kP;
      if (i < rows && j < k) ys[i * kSmallLd + j] = (double)__ldcs(Y + (r0 + i) * (int64_t)ldy + j);
    }
    __syncthreads();
    if (r < rows) {
      for (int c0 = 8 * h; c0 < m; c0 += 16) {
        double s[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) s[c] = 0.0;
#pragma unroll 4
        for (int j = 0; j < k; ++j) {
          const double y = ys[r * kSmallLd + j];
          const double2* vj = reinterpret_cast<const double2*>(vs + j * mp + c0);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const double2 vv = vj[c];
            s[2 * c] = fma(y, vv.x, s[2 * c]);
            s[2 * c + 1] = fma(y, vv.y, s[2 * c + 1]);
          }
        }
        double* z = Z + (r0 + r) * (int64_t)ldz + c0;
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (c0 + c < m) z[c] = s[c];
      }
    }
  }
}

template <typename T>
int32_t launch_panel_small(const T* Y, int32_t ldy, int64_t n, int32_t k, const double* V, int32_t m, double* Z,
                           int32_t ldz, cudaStream_t s) {
  if (!Y || !V || !Z || n <= 0 || k < 1 || k > kP || m < 1 || m > kP || ldy < k || ldz < m ||
      static_cast<const void*>(Y) == Z)
    return FEAB_BAD_ARG;
  FEAB_CUDA(cudaFuncSetAttribute(k_panel_small<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem));
  const int64_t tiles = (n + kSmallRows - 1) / kSmallRows;
  const int grid = (int)std::min<int64_t>(tiles, 2 * (int64_t)sm_count());
  k_panel_small<T><<<grid, kPThreads, kSmallSmem, s>>>(Y, ldy, n, k, V, m, Z, ldz);
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
