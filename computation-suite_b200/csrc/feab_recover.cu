// Hex8 strain / stress recovery (fea_engine/src/fea_engine/recovery.py:196-227, :258-334):
// values at the 2x2x2 Gauss points, sigma = D B u (or the engineering strain B u), moved to the
// corner nodes by the lumped L2 projection
//   value_a = sum_e sum_q N_a(q) |detJ| w val_q / sum_e sum_q N_a(q) |detJ| w
// over the elements e sharing node a, plus the volume-averaged element values
//   elem_e = sum_q |detJ| w val_q / sum_q |detJ| w,
// and optionally the von Mises stress of both (recovery.py:386-420).
//
// Two kernels.  k_recover_elements: 8 lanes per element, lane q holding the corner with the signs of
// Gauss point q.  The trilinear shape functions are products of one function per direction, so the
// derivatives of the coordinates and displacements at the Gauss points are three exchanges between
// the two lanes that differ in one sign (a difference along one direction, interpolations along the
// others), and the projection sum_q N_c(q) w_q val_q is three more with the same two weights.
// Everything stays in registers.  The element's corner records (6 numerators + denominator, padded
// to 64 bytes) go to scratch.  k_recover_nodes: one thread per node adds the corner records of its
// elements (16-byte loads) in ascending element order, the order of the reference's np.add.at over
// the connectivity, so the result is deterministic with no atomics.
#include "feab_hex8.cuh"

namespace feab {
namespace {

constexpr int kRecElems = 16;                 // elements per 128-thread block
constexpr int kRecThreads = kRecElems * 8;
constexpr int kRecord = 8;                    // doubles per (element, corner): 6 numerators, denominator, pad

// The two values of the linear shape functions (1 -+ xi) / 2 at the Gauss abscissas: the nearer corner's
// and the farther one's.
constexpr double kNear = 0.5 * (1.0 + FEAB_GAUSS2), kFar = 0.5 * (1.0 - FEAB_GAUSS2);

// Corner with the signs of Gauss point q (xi: bit 2, eta: bit 1, zeta: bit 0).
__device__ __forceinline__ int corner_of(int q) {
  return ((q & 1) << 2) | ((q & 2) ? ((q & 4) ? 2 : 3) : ((q & 4) ? 1 : 0));
}

// The value of the lane whose sign along the direction of `bit` is the other one.
__device__ __forceinline__ double other(double v, int bit) { return __shfl_xor_sync(FEAB_FULL_MASK, v, bit); }
__device__ __forceinline__ double interpolate(double v, double o) { return fma(kNear, v, kFar * o); }

// Natural derivatives, at the lane's Gauss point, of the trilinear field with corner values v.  h_*: 1/2 times the
// lane's sign along each direction.
__device__ __forceinline__ void natural_gradient(double v, double h_xi, double h_eta, double h_zeta, double (&d)[3]) {
  const double ox = other(v, 4);
  const double dx = h_xi * (v - ox), ix = interpolate(v, ox);
  const double odx = other(dx, 2), oix = other(ix, 2);
  const double dxi = interpolate(dx, odx), dy = h_eta * (ix - oix), iy = interpolate(ix, oix);
  const double ody = other(dy, 1), oiy = other(iy, 1);
  d[0] = interpolate(dxi, other(dxi, 1));
  d[1] = interpolate(dy, ody);
  d[2] = h_zeta * (iy - oiy);
}

__device__ __forceinline__ double mises(const double (&s)[6]) {
  const double a = s[0] - s[1], b = s[1] - s[2], c = s[2] - s[0];
  return sqrt(0.5 * (a * a + b * b + c * c) + 3.0 * (s[3] * s[3] + s[4] * s[4] + s[5] * s[5]));
}

// What bounds it: FP64 arithmetic (about 230 operations per Gauss point, with shape function tables and every
// derivative summed over the 8 corners it was some 450), the exchanges (114 per warp) and the 64-byte
// records.  rec may be NULL (element values only).
__global__ void __launch_bounds__(kRecThreads) k_recover_elements(const double* __restrict__ coords,
                                                                  const int32_t* __restrict__ conn, int64_t n_elem,
                                                                  Mat6 D, int use_d, const double* __restrict__ u,
                                                                  double* __restrict__ rec, double* __restrict__ elem,
                                                                  double* __restrict__ elem_vm,
                                                                  feab_device_status* st) {
  const int q = threadIdx.x & 7;
  const int64_t e0 = (int64_t)blockIdx.x * kRecElems + (threadIdx.x >> 3);
  const bool live = e0 < n_elem;
  const int64_t e = live ? e0 : n_elem - 1;    // spare lanes repeat the last element and write nothing
  const int c = corner_of(q);
  const int64_t node = conn[e * 8 + c];
  const double h_xi = (q & 4) ? 0.5 : -0.5, h_eta = (q & 2) ? 0.5 : -0.5, h_zeta = (q & 1) ? 0.5 : -0.5;
  double J[3][3], G[3][3], inv[3][3];          // J[i][j] = d X_j / d xi_i, G[i][j] = d u_j / d xi_i
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    double d[3];
    natural_gradient(coords[node * 3 + j], h_xi, h_eta, h_zeta, d);
#pragma unroll
    for (int i = 0; i < 3; ++i) J[i][j] = d[i];
    natural_gradient(u[node * 3 + j], h_xi, h_eta, h_zeta, d);
#pragma unroll
    for (int i = 0; i < 3; ++i) G[i][j] = d[i];
  }
  const double det = invert3(J, inv);
  if (live && !(fabs(det) >= 1e-300)) set_status(reinterpret_cast<int*>(st), FEAB_DEGENERATE_ELEMENT, e);
  // H[i][j] = d u_j / d x_i
  double H[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) H[i][j] = fma(inv[i][0], G[0][j], fma(inv[i][1], G[1][j], inv[i][2] * G[2][j]));
  // rows xx, yy, zz, xy, yz, xz with engineering shear (recovery.py:169-193)
  const double eps[6] = {H[0][0], H[1][1], H[2][2], H[1][0] + H[0][1], H[2][1] + H[1][2], H[2][0] + H[0][2]};
  const double w = fabs(det);                  // Gauss weights are 1
  double v[7];
#pragma unroll
  for (int s = 0; s < 6; ++s) {
    double x = eps[s];
    if (use_d) {
      x = 0.0;
#pragma unroll
      for (int j = 0; j < 6; ++j) x += D.d[s * 6 + j] * eps[j];
    }
    v[s] = w * x;
  }
  v[6] = w;
  if (elem || elem_vm) {
    double m[7];
#pragma unroll
    for (int s = 0; s < 7; ++s) {
      m[s] = v[s];
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) m[s] += __shfl_xor_sync(FEAB_FULL_MASK, m[s], o);
    }
    double avg[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) avg[s] = m[s] / m[6];
    if (live && elem && q < 6)
      elem[e * 6 + q] = q == 0 ? avg[0] : q == 1 ? avg[1] : q == 2 ? avg[2] : q == 3 ? avg[3] : q == 4 ? avg[4] : avg[5];
    if (live && elem_vm && q == 0) elem_vm[e] = mises(avg);
  }
  if (rec) {
#pragma unroll
    for (int s = 0; s < 7; ++s)
#pragma unroll
      for (int bit = 4; bit > 0; bit >>= 1) v[s] = interpolate(v[s], other(v[s], bit));
    if (live) {
      double2* r = reinterpret_cast<double2*>(rec + (e * 8 + c) * kRecord);
      r[0] = make_double2(v[0], v[1]);
      r[1] = make_double2(v[2], v[3]);
      r[2] = make_double2(v[4], v[5]);
      r[3] = make_double2(v[6], 0.0);
    }
  }
}

__global__ void k_recover_nodes(const int32_t* __restrict__ conn, const int32_t* __restrict__ inc_ptr,
                                const int32_t* __restrict__ inc_elem, int32_t n_nodes, const double* __restrict__ rec,
                                double* __restrict__ nodal, double* __restrict__ nodal_vm) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= n_nodes) return;
  double num[6] = {0, 0, 0, 0, 0, 0}, den = 0.0;
  for (int k = inc_ptr[a]; k < inc_ptr[a + 1]; ++k) {
    const int64_t e = inc_elem[k];
    const int4 c0 = *reinterpret_cast<const int4*>(conn + e * 8);
    const int4 c1 = *reinterpret_cast<const int4*>(conn + e * 8 + 4);
    const int c = c0.x == a ? 0 : c0.y == a ? 1 : c0.z == a ? 2 : c0.w == a ? 3
                : c1.x == a ? 4 : c1.y == a ? 5 : c1.z == a ? 6 : 7;
    const double2* r = reinterpret_cast<const double2*>(rec + (e * 8 + c) * kRecord);
    const double2 r0 = r[0], r1 = r[1], r2 = r[2], r3 = r[3];
    num[0] += r0.x;
    num[1] += r0.y;
    num[2] += r1.x;
    num[3] += r1.y;
    num[4] += r2.x;
    num[5] += r2.y;
    den += r3.x;
  }
  double v[6];
#pragma unroll
  for (int s = 0; s < 6; ++s) v[s] = den > 0.0 ? num[s] / den : 0.0;
  if (nodal) {
    double2* o = reinterpret_cast<double2*>(nodal + (int64_t)a * 6);
    o[0] = make_double2(v[0], v[1]);
    o[1] = make_double2(v[2], v[3]);
    o[2] = make_double2(v[4], v[5]);
  }
  if (nodal_vm) nodal_vm[a] = mises(v);
}

}  // namespace
}  // namespace feab

using namespace feab;

extern "C" size_t feab_hex8_recover_scratch_bytes(int64_t n_elem) {
  return n_elem > 0 ? sizeof(double) * (size_t)kRecord * 8 * (size_t)n_elem : 0;
}

extern "C" int32_t feab_hex8_recover(const double* coords, const int32_t* conn, int64_t n_elem, int32_t n_nodes,
                                     const int32_t* inc_ptr, const int32_t* inc_elem, const double* D_host,
                                     const double* u, double* nodal, double* nodal_vm, double* elem, double* elem_vm,
                                     void* scratch, size_t scratch_bytes, feab_device_status* status,
                                     cudaStream_t s) {
  if (!coords || !conn || !inc_ptr || !inc_elem || !u || n_elem <= 0 || n_nodes <= 0) return FEAB_BAD_ARG;
  if (!nodal && !nodal_vm && !elem && !elem_vm) return FEAB_BAD_ARG;
  if (!scratch || scratch_bytes < feab_hex8_recover_scratch_bytes(n_elem)) return FEAB_BAD_ARG;
  // the record, connectivity and nodal accesses are 16-byte vector accesses
  if ((reinterpret_cast<uintptr_t>(scratch) & 15u) || (reinterpret_cast<uintptr_t>(conn) & 15u) ||
      (reinterpret_cast<uintptr_t>(nodal) & 15u))
    return FEAB_BAD_ARG;
  if ((nodal_vm || elem_vm) && !D_host) return FEAB_BAD_ARG;  // von Mises is of the stress
  if (n_elem > (int64_t)INT32_MAX * kRecElems) return FEAB_BAD_ARG;
  Mat6 D;
  for (int i = 0; i < 36; ++i) D.d[i] = D_host ? D_host[i] : 0.0;
  double* rec = static_cast<double*>(scratch);
  const int64_t grid = (n_elem + kRecElems - 1) / kRecElems;
  k_recover_elements<<<(unsigned)grid, kRecThreads, 0, s>>>(coords, conn, n_elem, D, D_host ? 1 : 0, u,
                                                             nodal || nodal_vm ? rec : nullptr, elem, elem_vm, status);
  if (nodal || nodal_vm) {
    const int threads = 256;
    k_recover_nodes<<<(n_nodes + threads - 1) / threads, threads, 0, s>>>(conn, inc_ptr, inc_elem, n_nodes, rec, nodal,
                                                                         nodal_vm);
    count_launches(2);
  } else {
    count_launches(1);
  }
  FEAB_CHECK_LAUNCH();
  return FEAB_OK;
}
