// Resident PCG on the sliced operator: the whole solve in one kernel, for operators of up to
// kResMaxSlices slices per SM.
//
// One CTA per SM owns a contiguous run of slices, and so of rows, for the whole solve.  Each of
// its rows of x, r, p and D^-1 lives in the registers of one thread.  Its part of K lives on the
// SM as far as it fits: the first blocks of every warp in registers, the next in shared memory,
// the rest is read from L2.  Columns are renumbered at the start to a list of the rows that the
// CTA's slices refer to, so that p is fetched once per iteration into shared memory and the
// gathers read it there.  An iteration is
//   fetch (z, p_old) of the list, p = z + beta p_old -> SpMV -> p.Ap -> [sum 1]
//   -> x, r, z of the own rows, publish (z, p) -> r.r, r.z -> [sum 2] -> convergence test, beta
// The arithmetic is the step kernels' (the reference recurrence); only the order of the sums
// differs.
//
// The sums over the CTAs.  Within one cluster (small operators) every CTA writes its partial sum
// into every other's shared memory and the cluster barrier orders it.  Across the grid every CTA
// writes its partial sum and the sum's number as one 16-byte word into each CTA's inbox in global
// memory and waits for its own inbox to fill.  Either way each CTA adds the partial sums in CTA
// order, so all hold the same scalars, take the same decisions, and results are reproducible.
// Inboxes and the published (z, p) alternate between two buffers: a CTA writes a buffer again
// only after a sum that every CTA enters after it has read that buffer.  Each wait is bounded; a
// CTA whose wait runs out reports it and leaves, and so do the others.
//
// What bounds it: latency.  The step kernels spent 18 to 22 us per iteration whatever the size below
// a thousand slices: one warp walks a slice's 84 column steps alone, and every iteration pays three
// launches.  Here 16 warps share the CTA's slices, and an iteration is two exchanges (3 us each with
// 148 CTAs, 1.3 us in a cluster of 16), one fetch of p from L2 (1 us) and the products.  Measured,
// us per iteration, step kernels -> resident:
//   elements      slices   FP64            mixed
//   20x4x4            16   18.4 ->  5.2    21.5 ->  6.1
//   37x11x9          139   18.5 ->  7.6    20.5 ->  8.4
//   64x16x16         578   20.1 -> 10.0    29.4 -> 10.4
//   80x20x20        1103   22.9 -> 19.6    35.3 -> 18.1
// Above 8 slices per SM most of K comes from L2 or HBM in every iteration, and the step kernels stream it through
// their ring with more warps to wait for it.  Below, they lose to the launches: whole solves at 80x20x20,
// resident against the steps with the ring, FP64 21.2 and 25.7 ms, mixed 18.6 and 26.8 ms.
#pragma once

namespace feab {
namespace {

constexpr int kResThreads = 512;
constexpr int kResWarps = kResThreads / 32;
constexpr int kResMaxCtas = 160;              // CTAs of a grid-wide sum (one thread per inbox word)
constexpr int kResMaxSlices = 8;              // slices per CTA: 96 rows each, two rows per thread
constexpr int kResMaxCluster = 16;
constexpr int kResSpinLimit = 1 << 21;  // polls of one word before a wait gives up (seconds)
static_assert(96 * kResMaxSlices <= 2 * kResThreads, "a thread has at most two rows");

struct ResArgs {
  ulonglong2* inbox;   // 2 banks x gridDim inboxes x gridDim senders, words {value 0, value 1 and phase}
  double2* zp[2];      // published (z, p): the z, p0 and the p1, Ap vectors' storage
  int32_t resume;      // 0: p = z = D^-1 r; 1: continue from the published (z, p)
  int32_t max_steps;   // iterations of this launch
  int32_t smem_bytes;  // dynamic shared memory
};

// Results of a launch beside PcgState: does the operator fit the kernel's shared memory?
constexpr int kResMisfit = -1;   // PcgState::done

// blocks of 4 column steps that a warp keeps in registers (24 registers each, mixed 18), as many as
// the 128 registers of a thread hold without spills
#ifndef FEAB_RES_RB
#define FEAB_RES_RB(KIND, ROWS) ((ROWS) == 1 ? ((KIND) == FEAB_PREC_FP64 ? 1 : 2) : 1)
#endif

template <int KIND>
struct ResTuning {
  static constexpr int kBlockBytes = KIND == FEAB_PREC_FP64 ? 3072 : 2304;   // of 32 lanes, in shared memory
};

// A lane's values of one block of 4 column steps.
template <int KIND>
struct ResVals {
  double v[KIND == FEAB_PREC_FP64 ? 3 : 1][4];
  uint4 h[KIND == FEAB_PREC_FP64 ? 1 : 3];
  uint2 l[KIND == FEAB_PREC_FP64 ? 1 : 3];
};

template <int KIND>
__device__ __forceinline__ void res_load(const SellView& V, size_t b, int lane, ResVals<KIND>& B) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const size_t o = (3 * b + 4 * k) * 32;
    if (KIND == FEAB_PREC_FP64) {
      const double2* vp = reinterpret_cast<const double2*>(V.v64 + o) + 2 * lane;
      const double2 p0 = __ldcs(vp), p1 = __ldcs(vp + 1);
      B.v[k][0] = p0.x;
      B.v[k][1] = p0.y;
      B.v[k][2] = p1.x;
      B.v[k][3] = p1.y;
    } else {
      B.h[k] = __ldcs(reinterpret_cast<const uint4*>(V.vhi + o) + lane);
      B.l[k] = __ldcs(reinterpret_cast<const uint2*>(V.vlo + o) + lane);
    }
  }
}

// The same to and from a block of shared memory: 16-byte (8-byte) words, lane by lane.
template <int KIND>
__device__ __forceinline__ void res_store_smem(unsigned char* blk, int lane, const ResVals<KIND>& B) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (KIND == FEAB_PREC_FP64) {
      reinterpret_cast<double2*>(blk)[(2 * k) * 32 + lane] = make_double2(B.v[k][0], B.v[k][1]);
      reinterpret_cast<double2*>(blk)[(2 * k + 1) * 32 + lane] = make_double2(B.v[k][2], B.v[k][3]);
    } else {
      reinterpret_cast<uint4*>(blk)[k * 32 + lane] = B.h[k];
      reinterpret_cast<uint2*>(blk + 3 * 512)[k * 32 + lane] = B.l[k];
    }
  }
}

template <int KIND>
__device__ __forceinline__ void res_load_smem(const unsigned char* blk, int lane, ResVals<KIND>& B) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (KIND == FEAB_PREC_FP64) {
      const double2 p0 = reinterpret_cast<const double2*>(blk)[(2 * k) * 32 + lane];
      const double2 p1 = reinterpret_cast<const double2*>(blk)[(2 * k + 1) * 32 + lane];
      B.v[k][0] = p0.x;
      B.v[k][1] = p0.y;
      B.v[k][2] = p1.x;
      B.v[k][3] = p1.y;
    } else {
      B.h[k] = reinterpret_cast<const uint4*>(blk)[k * 32 + lane];
      B.l[k] = reinterpret_cast<const uint2*>(blk + 3 * 512)[k * 32 + lane];
    }
  }
}

// a_k += sum_u value(k, u) h[local column u].
template <int KIND>
__device__ __forceinline__ void res_use(const ResVals<KIND>& B, uint2 t, const double* h, double (&a)[3]) {
  const double d[4] = {h[t.x & 0xffffu], h[t.x >> 16], h[t.y & 0xffffu], h[t.y >> 16]};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (KIND == FEAB_PREC_FP64) {
#pragma unroll
      for (int u = 0; u < 4; ++u) a[k] = fma(B.v[k][u], d[u], a[k]);
    } else {
      a[k] = fma(sell_dec48(B.h[k].x, (uint16_t)(B.l[k].x & 0xffffu)), d[0], a[k]);
      a[k] = fma(sell_dec48(B.h[k].y, (uint16_t)(B.l[k].x >> 16)), d[1], a[k]);
      a[k] = fma(sell_dec48(B.h[k].z, (uint16_t)(B.l[k].y & 0xffffu)), d[2], a[k]);
      a[k] = fma(sell_dec48(B.h[k].w, (uint16_t)(B.l[k].y >> 16)), d[3], a[k]);
    }
  }
}

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// A word of an inbox: value 0, and value 1 (never negative) whose sign bit is the word's phase, which
// changes with every use of the word.  One 16-byte access carries both sums and their arrival.
__device__ __forceinline__ void st_word(ulonglong2* p, double v0, double v1, unsigned phase) {
  const unsigned long long w1 = ((unsigned long long)__double_as_longlong(v1) & ~(1ull << 63)) |
                                ((unsigned long long)phase << 63);
  asm volatile("{\n .reg .b128 w;\n mov.b128 w, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], w;\n}" ::"l"(p),
               "l"(__double_as_longlong(v0)), "l"(w1)
               : "memory");
}

__device__ __forceinline__ ulonglong2 ld_word(const ulonglong2* p) {
  ulonglong2 r;
  asm volatile("{\n .reg .b128 w;\n ld.relaxed.gpu.global.b128 w, [%2];\n mov.b128 {%0, %1}, w;\n}"
               : "=l"(r.x), "=l"(r.y)
               : "l"(p)
               : "memory");
  return r;
}

// Writes v to the same place of CTA `rank`'s shared memory in the cluster.
__device__ __forceinline__ void st_cluster(double* p, int rank, double v) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(v) : "memory");
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct ResShared {
  double red[2][kResWarps];
  double vals[2][2][kResMaxCtas];   // [bank]: a cluster's CTAs write the next sum's while this one is read
  int abort_flag;
  int scan[kResWarps];
  int total;
};

// Sums of NV values per thread over all CTAs; the same result in every thread (the second value's
// is a sum of squares).  DATA: writes to global memory made by any CTA before the call are seen by
// all after it.  False when a wait ran out.  `number` starts at 2: a word's first phase is 1.
template <int NV, bool CLUSTER, bool DATA>
__device__ __forceinline__ bool res_sum(double (&v)[NV], ResShared& sh, const ResArgs& Q, unsigned& number) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = gridDim.x, bank = number & 1;
  const unsigned phase = (number >> 1) & 1;
  ++number;
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = warp_sum(v[k]);
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) sh.red[k][warp] = v[k];
  }
  __syncthreads();
  // every warp that publishes adds the warps' sums, in order of a butterfly over 16
  if (32 * warp < G) {
    if (DATA && !CLUSTER) fence_gpu();
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = sh.red[k][lane & (kResWarps - 1)];
#pragma unroll
    for (int o = kResWarps / 2; o > 0; o >>= 1) {
#pragma unroll
      for (int k = 0; k < NV; ++k) v[k] += __shfl_xor_sync(FEAB_FULL_MASK, v[k], o);
    }
  }
  if constexpr (CLUSTER) {
    if (tid < G) {
#pragma unroll
      for (int k = 0; k < NV; ++k) st_cluster(&sh.vals[bank][k][blockIdx.x], tid, v[k]);
    }
    cluster_barrier();
  } else {
    if (tid < G) {
      st_word(Q.inbox + ((size_t)bank * G + tid) * G + blockIdx.x, v[0], NV > 1 ? v[NV - 1] : 0.0, phase);
      const ulonglong2* in = Q.inbox + ((size_t)bank * G + blockIdx.x) * G + tid;
      ulonglong2 w = ld_word(in);
      for (int spin = 0; (unsigned)(w.y >> 63) != phase; ++spin) {
        if (spin >= kResSpinLimit) {
          sh.abort_flag = 1;
          break;
        }
        w = ld_word(in);
      }
      sh.vals[bank][0][tid] = __longlong_as_double((long long)w.x);
      if (NV > 1) sh.vals[bank][1][tid] = __longlong_as_double((long long)(w.y & ~(1ull << 63)));
      if (DATA) fence_gpu();
    }
    __syncthreads();
  }
  double s[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) s[k] = 0.0;
  for (int i = lane; i < G; i += 32) {
#pragma unroll
    for (int k = 0; k < NV; ++k) s[k] += sh.vals[bank][k][i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < NV; ++k) s[k] += __shfl_xor_sync(FEAB_FULL_MASK, s[k], o);
  }
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = s[k];
  return CLUSTER || sh.abort_flag == 0;
}

constexpr int kResSmem = 232448 - 1024 - (int)((sizeof(ResShared) + 1023) / 1024 * 1024);   // dynamic, of 227 KB

// ROWS: rows per thread, 1 for up to five slices per CTA, else 2.
template <int KIND, bool IDX16, bool CLUSTER, int ROWS>
__global__ void __launch_bounds__(kResThreads, 1) k_pcg_resident(PcgArgs A, ResArgs Q) {
  constexpr int RB = FEAB_RES_RB(KIND, ROWS);
  constexpr int kBytes = ResTuning<KIND>::kBlockBytes;
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ ResShared sh;
  PcgState* S = A.S_;
  if (S->done) return;  // the same in every CTA: it is only written after a sum over all CTAs
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const SellView& V = A.sell;
  const int ns = V.n_slices;
  const int s0 = (int)((int64_t)blockIdx.x * ns / gridDim.x), s1 = (int)((int64_t)(blockIdx.x + 1) * ns / gridDim.x);
  const int nsl = s1 - s0, wps = kResWarps / nsl;   // slices, warps per slice
  const int g0 = 32 * s0, g1 = min(32 * s1, V.n_groups);
  const int base0 = __ldg(V.soff + s0), total_blocks = (__ldg(V.soff + s1) - base0) >> 2;
  // the warp's part of its slice: blocks first, first + wps, ...
  const int msl = warp / wps, first = warp - msl * wps;
  const bool works = msl < nsl;
  const int sbase = works ? __ldg(V.soff + s0 + msl) : base0;
  const int nb = works ? (__ldg(V.soff + s0 + msl + 1) - sbase) >> 2 : 0;
  const int nbw = nb > first ? (nb - first + wps - 1) / wps : 0;
  const int lblk = (sbase - base0) >> 2;   // the slice's first block within the CTA

  // ---- shared memory: partial sums, local columns, the list and its p, then blocks of K
  double (*part)[3][32] = reinterpret_cast<double (*)[3][32]>(dyn);
  uint2* const cols = reinterpret_cast<uint2*>(dyn + sizeof(double) * kResWarps * 96);
  int32_t* const list = reinterpret_cast<int32_t*>(cols + (size_t)total_blocks * 32);
  const int words = (A.n + 31) >> 5;
  uint32_t* const bits = reinterpret_cast<uint32_t*>(dyn + Q.smem_bytes) - 2 * words;   // until the list is made
  uint32_t* const rank = bits + words;
  const size_t fixed_bytes = sizeof(double) * kResWarps * 96 + (size_t)total_blocks * 256;
  const bool room = fixed_bytes + 8 * (size_t)words + 16 <= (size_t)Q.smem_bytes;   // the same for the whole CTA
  if (tid == 0) sh.abort_flag = 0;

  // ---- the rows that the CTA refers to
  auto columns = [&](int i, int r0, unsigned (&t)[4]) {   // of the warp's block i
    const size_t b = (size_t)sbase + 4 * (size_t)(first + i * wps);
    if (IDX16) {
      const uint2 q = __ldg(reinterpret_cast<const uint2*>(V.tcol16 + b * 32) + lane);
      t[0] = (unsigned)(r0 + (int)(int16_t)(q.x & 0xffffu));
      t[1] = (unsigned)(r0 + (int)(int16_t)(q.x >> 16));
      t[2] = (unsigned)(r0 + (int)(int16_t)(q.y & 0xffffu));
      t[3] = (unsigned)(r0 + (int)(int16_t)(q.y >> 16));
    } else {
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(V.tcol + b * 32) + lane);
      const unsigned m = KIND == FEAB_PREC_FP64 ? 0xffffffffu : 0x3fffffffu;
      t[0] = q.x & m;
      t[1] = q.y & m;
      t[2] = q.z & m;
      t[3] = q.w & m;
    }
  };
  const SellLane L = works ? sell_lane(V, s0 + msl, lane) : SellLane{0, 0, 0, false};
  int H = 0;
  if (room) {
    for (int i = tid; i < words; i += kResThreads) bits[i] = 0u;
    __syncthreads();
    for (int i = 0; i < nbw; ++i) {
      unsigned t[4];
      columns(i, L.r0, t);
#pragma unroll
      for (int u = 0; u < 4; ++u) atomicOr(bits + (t[u] >> 5), 1u << (t[u] & 31));
    }
    if (works && first == 0)
      for (int k = 0; k < L.f; ++k) atomicOr(bits + ((L.r0 + k) >> 5), 1u << ((L.r0 + k) & 31));
    __syncthreads();
    // rank of each word: thread t owns a run of words
    const int per = (words + kResThreads - 1) / kResThreads, w0 = min(words, tid * per), w1 = min(words, w0 + per);
    int mine = 0;
    for (int i = w0; i < w1; ++i) mine += __popc(bits[i]);
    const int incl = warp_incl_scan(mine, lane);
    if (lane == 31) sh.scan[warp] = incl;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < kResWarps; ++w) {
      if (w < warp) before += sh.scan[w];
      H += sh.scan[w];
    }
    int at = before + incl - mine;
    for (int i = w0; i < w1; ++i) {
      rank[i] = (uint32_t)at;
      at += __popc(bits[i]);
    }
  }
  const size_t list_bytes = ((size_t)H * 4 + 15) & ~size_t(15);
  double* const hp = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(list) + list_bytes);
  const size_t h_bytes = ((size_t)H * 8 + 15) & ~size_t(15);
  const bool fits = room && H > 0 && H <= 65536 &&
                    fixed_bytes + list_bytes + h_bytes + 8 * (size_t)words + 16 <= (size_t)Q.smem_bytes;
  const size_t kroom = fits ? ((size_t)Q.smem_bytes - fixed_bytes - list_bytes - h_bytes) / kBytes : 0;
  const int nsm = (int)(kroom / kResWarps);   // blocks of K per warp in shared memory
  unsigned char* const kblk = reinterpret_cast<unsigned char*>(hp) + h_bytes + (size_t)warp * nsm * kBytes;
  __syncthreads();
  auto local = [&](unsigned row) {
    const uint32_t w = row >> 5, b = row & 31;
    return rank[w] + (uint32_t)__popc(bits[w] & ((1u << b) - 1u));
  };

  // ---- the thread's rows: row (slice, k, lane) of the CTA for t = tid, tid + 512
  int row[ROWS], own[ROWS], pidx[ROWS];
  double xr[ROWS], rv[ROWS], pv[ROWS], dv[ROWS];
  double T[KIND == FEAB_PREC_MIXED ? ROWS : 1][3];
  int xo[KIND == FEAB_PREC_MIXED ? ROWS : 1][3];
  int cur = Q.resume ? S->psel : 0;
#pragma unroll
  for (int m = 0; m < ROWS; ++m) {
    const int t = tid + m * kResThreads, sl = t / 96, k = (t - 96 * sl) >> 5, l = t & 31;
    row[m] = -1;
    own[m] = pidx[m] = 0;
    xr[m] = rv[m] = pv[m] = dv[m] = 0.0;
    if constexpr (KIND == FEAB_PREC_MIXED) {
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        T[m][j] = 0.0;
        xo[m][j] = 0;
      }
    }
    if (fits && sl < nsl) {
      const SellLane R = sell_lane(V, s0 + sl, l);
      if (k < R.f) {
        const int i = R.r0 + k;
        row[m] = i;
        pidx[m] = sl * wps * 96 + k * 32 + l;   // into part, of the slice's first warp
        own[m] = (int)local((unsigned)i);
        dv[m] = A.use_dinv ? A.dinv64[i] : 1.0;
        xr[m] = A.x[i];
        rv[m] = A.r[i];
        const double z = dv[m] * rv[m];
        if (Q.resume) {
          pv[m] = Q.zp[cur][i].y;
        } else {
          pv[m] = z;
          Q.zp[0][i] = make_double2(z, 0.0);
        }
        if constexpr (KIND == FEAB_PREC_MIXED) {
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            if ((R.mask >> j) & 1) {
              xo[m][j] = (int)local((unsigned)(R.r0 + __popc(R.mask & ((1 << j) - 1))));
              T[m][j] = V.S[(int64_t)i * 3 + j];
            }
          }
        }
      }
    }
  }
  // ---- the list and the local columns
  if (fits) {
    for (int i = tid; i < words; i += kResThreads) {
      uint32_t b = bits[i];
      uint32_t at = rank[i];
      while (b) {
        list[at++] = 32 * i + __ffs(b) - 1;
        b &= b - 1;
      }
    }
    for (int i = 0; i < nbw; ++i) {
      unsigned t[4];
      columns(i, L.r0, t);
      cols[(size_t)(lblk + first + i * wps) * 32 + lane] =
          make_uint2(local(t[0]) | (local(t[1]) << 16), local(t[2]) | (local(t[3]) << 16));
    }
  }
  __syncthreads();
  // ---- K: the first blocks of the warp into registers, the next into shared memory
  ResVals<KIND> reg[RB];
  auto block_of = [&](int i) { return (size_t)sbase + 4 * (size_t)(first + i * wps); };
#pragma unroll
  for (int i = 0; i < RB; ++i)
    if (i < nbw) res_load<KIND>(V, block_of(i), lane, reg[i]);
  const int nres = min(nbw, RB + nsm);
  if (fits) {
    for (int i = RB; i < nres; ++i) {
      ResVals<KIND> B;
      res_load<KIND>(V, block_of(i), lane, B);
      res_store_smem<KIND>(kblk + (size_t)(i - RB) * kBytes, lane, B);
    }
  }

  unsigned number = 2;
  const double tol = S->tol, delta = S->delta, bnorm = S->bnorm;
  double rz_old = S->rz_old, beta = Q.resume ? S->beta : 0.0, rmax = S->rmax, rr64 = S->rr64;
  double rr = S->rr, relres = S->relres;
  int iters = S->iters, reliable = S->reliable_updates, status = S->status;
  const int maxiter = S->maxiter;
  int done = 0;
  bool pend = Q.resume != 0;
  // the first sum: everyone's (z, p) is published; does every CTA fit?
  double one[1] = {tid == 0 && !fits ? 1.0 : 0.0};
  if constexpr (CLUSTER) cluster_barrier();   // every CTA has started: its shared memory can be written
  bool ok = res_sum<1, CLUSTER, true>(one, sh, Q, number);
  const bool misfit = one[0] != 0.0;
  const uint2* const mycols = cols + (size_t)(lblk + first) * 32 + lane;
  for (int step = 0; ok && !misfit && step < Q.max_steps; ++step) {
    ResVals<KIND> pre;   // the first block of the part that stays in L2, on its way during the fetch of p
    if (nres < nbw) res_load<KIND>(V, block_of(nres), lane, pre);
    const double2* __restrict__ zp = cur ? Q.zp[1] : Q.zp[0];
    {
      int i = tid;
      for (; i + 3 * kResThreads < H; i += 4 * kResThreads) {
        double2 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = __ldcg(zp + list[i + u * kResThreads]);
#pragma unroll
        for (int u = 0; u < 4; ++u) hp[i + u * kResThreads] = fma(beta, q[u].y, q[u].x);
      }
      double2 q[3];
#pragma unroll
      for (int u = 0; u < 3; ++u)
        if (i + u * kResThreads < H) q[u] = __ldcg(zp + list[i + u * kResThreads]);
#pragma unroll
      for (int u = 0; u < 3; ++u)
        if (i + u * kResThreads < H) hp[i + u * kResThreads] = fma(beta, q[u].y, q[u].x);
    }
    __syncthreads();
    double a[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int i = 0; i < RB; ++i)
      if (i < nbw) res_use<KIND>(reg[i], mycols[(size_t)i * wps * 32], hp, a);
    for (int i = RB; i < nres; ++i) {
      ResVals<KIND> B;
      res_load_smem<KIND>(kblk + (size_t)(i - RB) * kBytes, lane, B);
      res_use<KIND>(B, mycols[(size_t)i * wps * 32], hp, a);
    }
    for (int i = nres; i < nbw; ++i) {
      ResVals<KIND> nxt;
      if (i + 1 < nbw) res_load<KIND>(V, block_of(i + 1), lane, nxt);
      res_use<KIND>(pre, mycols[(size_t)i * wps * 32], hp, a);
      if (i + 1 < nbw) pre = nxt;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) part[warp][k][lane] = a[k];
    __syncthreads();
    double q[ROWS], v[2] = {0.0, 0.0};
    one[0] = 0.0;
#pragma unroll
    for (int m = 0; m < ROWS; ++m) {
      q[m] = 0.0;
      if (row[m] >= 0) {
        const double* pp = &part[0][0][0] + pidx[m];
        for (int w = 0; w < wps; ++w) q[m] += pp[w * 96];
        if constexpr (KIND == FEAB_PREC_MIXED)   // the own-node term of the difference form
          q[m] += T[m][0] * hp[xo[m][0]] + T[m][1] * hp[xo[m][1]] + T[m][2] * hp[xo[m][2]];
        if (pend) pv[m] = hp[own[m]];
        one[0] += pv[m] * q[m];
      }
    }
    if (!(ok = res_sum<1, CLUSTER, false>(one, sh, Q, number))) break;
    const double pAp = one[0];
    if (!(pAp > 0.0)) {  // p^T A p <= 0: A is not SPD (iterative_solvers.py:450-454)
      status = FEAB_NOT_SPD;
      done = 1;
      break;
    }
    const double alpha = rz_old / pAp;
    double2* const zn = cur ? Q.zp[0] : Q.zp[1];
#pragma unroll
    for (int m = 0; m < ROWS; ++m) {
      if (row[m] >= 0) {
        xr[m] = fma(alpha, pv[m], xr[m]);
        rv[m] = fma(-alpha, q[m], rv[m]);
        const double z = dv[m] * rv[m];
        zn[row[m]] = make_double2(z, pv[m]);
        v[0] += rv[m] * z;
        v[1] += rv[m] * rv[m];
      }
    }
    cur ^= 1;
    if (!(ok = res_sum<2, CLUSTER, true>(v, sh, Q, number))) break;
    ++iters;
    rr = v[1];
    const double rel = sqrt(rr) / bnorm;
    bool replace = false;
    if (KIND == FEAB_PREC_FP64) {
      relres = rel;
      if (rel < tol) {
        done = 1;
        status = FEAB_OK;
        break;
      }
      if (iters >= maxiter || !(rel == rel)) {
        done = 1;
        status = FEAB_NOT_CONVERGED;
        break;
      }
    } else {
      replace = rel < tol || sqrt(rr) < delta * rmax || iters >= maxiter || !(rel == rel);
    }
    if (KIND == FEAB_PREC_MIXED && replace) {
      // r = b - K64 x with the FP64 CSR values; the new direction waits for it
#pragma unroll
      for (int m = 0; m < ROWS; ++m)
        if (row[m] >= 0) A.x[row[m]] = xr[m];
      one[0] = 0.0;
      if (!(ok = res_sum<1, CLUSTER, true>(one, sh, Q, number))) break;
      const int hl = lane & 7;
      for (int gb = g0 + 4 * warp; gb < g1; gb += 4 * kResWarps) {
        Group gr;
        gr.g = gb + (lane >> 3);
        gr.valid = gr.g < g1;
        gr.r0 = gr.f = gr.s0 = gr.len = 0;
        if (gr.valid) {
          gr.r0 = __ldg(A.group_ptr + gr.g);
          gr.f = __ldg(A.group_ptr + gr.g + 1) - gr.r0;
          gr.s0 = __ldg(A.row_ptr + gr.r0);
          gr.len = __ldg(A.row_ptr + gr.r0 + 1) - gr.s0;
        }
        double acc[3];
        group_spmv<8, double>(A, A.vals64, gr, hl, [&](int j) { return __ldcg(A.x + j); }, acc);
        if (hl < gr.f) {   // the group's rows in the order of part: (slice, k, lane)
          const int gl = gr.g - g0;
          (&part[0][0][0])[(gl >> 5) * 96 + hl * 32 + (gl & 31)] = pick3(acc, hl);
        }
      }
      __syncthreads();
      v[0] = v[1] = 0.0;
      double2* const zr = cur ? Q.zp[1] : Q.zp[0];
#pragma unroll
      for (int m = 0; m < ROWS; ++m) {
        if (row[m] >= 0) {
          rv[m] = A.b[row[m]] - (&part[0][0][0])[tid + m * kResThreads];
          const double z = dv[m] * rv[m];
          zr[row[m]] = make_double2(z, pv[m]);
          v[0] += rv[m] * z;
          v[1] += rv[m] * rv[m];
        }
      }
      if (!(ok = res_sum<2, CLUSTER, true>(v, sh, Q, number))) break;
      ++reliable;
      rr64 = v[1];
      relres = sqrt(rr64) / bnorm;
      if (relres < tol) {
        done = 1;
        status = FEAB_OK;
        break;
      }
      if (iters >= maxiter || !(relres == relres)) {
        done = 1;
        status = FEAB_NOT_CONVERGED;
        break;
      }
      rmax = sqrt(rr64);
    }
    beta = v[0] / rz_old;
    rz_old = v[0];
    pend = true;
  }
  if (CLUSTER) cluster_barrier();   // no CTA leaves while another may still write its shared memory
  if (!ok) {
    // a wait ran out (a CTA of the grid is missing): every CTA gets here by its own wait
    if (tid == 0) {
      S->status = FEAB_CUDA_ERROR;
      S->done = 1;
    }
    return;
  }
  if (!misfit) {
#pragma unroll
    for (int m = 0; m < ROWS; ++m) {
      if (row[m] >= 0) {
        A.x[row[m]] = xr[m];
        A.r[row[m]] = rv[m];
      }
    }
  }
  if (blockIdx.x == 0 && tid == 0) {
    S->rz_old = rz_old;
    S->beta = beta;
    S->rmax = rmax;
    S->rr = rr;
    S->rr64 = rr64;
    S->relres = relres;
    S->iters = iters;
    S->reliable_updates = reliable;
    S->psel = cur;
    S->status = status;
    S->done = misfit ? kResMisfit : done;
  }
}

}  // namespace
}  // namespace feab
