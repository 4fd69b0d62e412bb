// Routing metadata for the MoE layer: count/cumsum of expert ids and the fused
// top-k -> padded expert-sorted layout.  Integer work, bit-exact by construction:
// no floating-point atomics, no order-dependent atomics (bit masks are built with
// atomicOr, whose result does not depend on arrival order).
//
// Layout of the work: rows are cut into units of 32 (one warp, one row per lane).
//   1. unit_masks_kernel  mask[u][e] = lanes of unit u whose row selects expert e;
//                         valid[u]   = number of valid (row, slot) pairs of the unit
//   2. scan_kernel        per expert: exclusive scan of popc(mask[.][e]) over units
//                         (rows of an expert keep ascending token order) + count[e];
//                         one more block scans valid[.] -> token-major bases, real_TK
//   3. scatter_fill_kernel recomputes the padded offsets in shared memory, writes
//                         every output, then fills pad rows and over-allocated tails
// Small problems run the three steps in one kernel (metadata_cluster_kernel).
#include <cuda_runtime.h>
#include <stdint.h>

#include "smoe_b200.h"

namespace smoe {

constexpr int kMaxTopk = 16;
constexpr int kRtThreads = 256;
constexpr int kUnitsPerBlock = kRtThreads / 32;

__device__ __forceinline__ int warp_excl_scan(int v, int lane) {
  int x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int y = __shfl_up_sync(0xffffffff, x, d);
    if (lane >= d) x += y;
  }
  return x - v;
}

// Block-wide exclusive scan of n values produced by f(i), consumed by g(i, exclusive);
// returns the total.  Blocked partition: each thread owns a contiguous run.
template <typename F, typename G>
__device__ int block_excl_scan(int n, F f, G g, int* s_warp /* >= 33 ints */) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int chunk = (n + blockDim.x - 1) / blockDim.x;
  const int lo = min(tid * chunk, n), hi = min(lo + chunk, n);
  int part = 0;
  for (int i = lo; i < hi; ++i) part += f(i);
  const int wex = warp_excl_scan(part, lane);
  if (lane == 31) s_warp[warp] = wex + part;
  __syncthreads();
  if (warp == 0) {
    const int t = lane < nw ? s_warp[lane] : 0;
    const int ex = warp_excl_scan(t, lane);
    if (lane < nw) s_warp[lane] = ex;
    if (lane == 31) s_warp[32] = ex + t;
  }
  __syncthreads();
  int run = s_warp[warp] + wex;
  for (int i = lo; i < hi; ++i) {
    const int v = f(i);
    g(i, run);
    run += v;
  }
  const int total = s_warp[32];
  __syncthreads();
  return total;
}

// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kRtThreads)
unit_masks_kernel(const int* __restrict__ idx, int N, int K, int E, uint32_t* __restrict__ mask,
                  int* __restrict__ unit_valid) {
  const int lane = threadIdx.x & 31;
  const int unit = blockIdx.x * kUnitsPerBlock + (threadIdx.x >> 5);
  const int units = (N + 31) / 32;
  if (unit >= units) return;
  const int row = unit * 32 + lane;
  uint32_t* m = mask + (size_t)unit * E;
  for (int e = lane; e < E; e += 32) m[e] = 0u;
  __syncwarp();
  int nvalid = 0;
  if (row < N) {
    for (int k = 0; k < K; ++k) {
      const int e = idx[(size_t)row * K + k];
      if (e >= 0 && e < E) {
        atomicOr(&m[e], 1u << lane);
        ++nvalid;
      }
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) nvalid += __shfl_xor_sync(0xffffffff, nvalid, d);
  if (lane == 0) unit_valid[unit] = nvalid;
}

// blocks [0, E): expert e -> unit_off[u][e] = exclusive scan over u of popc(mask[u][e]); counts[e] = total
// block  E     : unit_base[u] = exclusive scan of unit_valid; naept[N] = total
__global__ void __launch_bounds__(kRtThreads)
scan_kernel(const uint32_t* __restrict__ mask, const int* __restrict__ unit_valid, int units, int E, int N,
            int TK_alloc, int* __restrict__ unit_off, int* __restrict__ counts, int* __restrict__ unit_base,
            int* __restrict__ naept) {
  __shared__ int s_warp[33];
  const int e = blockIdx.x;
  if (e < E) {
    const int total = block_excl_scan(
        units, [&](int u) { return __popc(mask[(size_t)u * E + e]); },
        [&](int u, int ex) { unit_off[(size_t)u * E + e] = ex; }, s_warp);
    if (threadIdx.x == 0) counts[e] = total;
  } else {
    const int total = block_excl_scan(
        units, [&](int u) { return unit_valid[u]; }, [&](int u, int ex) { unit_base[u] = ex; }, s_warp);
    if (threadIdx.x == 0) naept[N] = min(total, TK_alloc);
  }
}

// What the scatter and the fill write, and the sizes they go by
struct TopkOut {
  const int* idx;
  const float* probs;
  int N, K, E, alignment, TK_alloc, TKp_alloc, lane_order, pad_mode;
  int *efo, *x_gather, *s_scatter, *s_rev, *naept;
  float* scores;
  int *src_idx, *counts;
};

// Offsets of the experts' segments, in shared memory, and what of the problem fits the buffers
struct Layout {
  int limit;       // expert-sorted positions at or beyond it are not published
  int tot_p;       // padded rows
  int real_TK;     // entries that are published, naept[N]
  bool cut;
};

// s_efo / s_base [E+1]: padded and unpadded offsets from counts(e); the whole block takes part, `first`: this block writes efo
// and, of a cut pass, naept[N]
template <typename C>
__device__ Layout block_layout(const TopkOut& o, C counts, int* s_efo, int* s_base, int* s_warp, bool first) {
  Layout l;
  const int E = o.E, alignment = o.alignment;
  l.tot_p = block_excl_scan(
      E,
      [&](int e) {
        const int c = counts(e);
        return c > 0 ? (c + alignment - 1) / alignment * alignment : 0;
      },
      [&](int e, int ex) { s_efo[e] = ex; }, s_warp);
  const int tot_u = block_excl_scan(
      E, [&](int e) { return counts(e); }, [&](int e, int ex) { s_base[e] = ex; }, s_warp);
  if (threadIdx.x == 0) {
    s_efo[E] = l.tot_p;
    s_base[E] = tot_u;
  }
  __syncthreads();
  // Published offsets never point past the allocation (they can only exceed it when the caller sized the buffers from counts
  // that do not match idx), and neither does anything that a reader of this metadata follows.  Such a pass is `cut`: an entry
  // whose expert-sorted position lies at or beyond `limit` counts as if its slot were masked - expert e keeps its first
  // clamp(limit - s_efo[e]) rows, so the token-major base of a unit is the sum of what its experts keep of the units before -
  // and of what is left the first TK_alloc entries stay; the row of a later one becomes a pad row (it lies among the last rows
  // of its expert: token-major order is ascending there).  naept, s_rev, s_scatter and the scores then agree with each other.
  l.limit = o.TKp_alloc / alignment * alignment;
  if (first)
    for (int e = threadIdx.x; e <= E; e += blockDim.x) o.efo[e] = min(s_efo[e], l.limit);
  l.cut = l.tot_p > l.limit || tot_u > o.TK_alloc;
  l.real_TK = tot_u;
  if (l.cut) {
    const int fit = block_excl_scan(
        E, [&](int e) { return max(min(counts(e), l.limit - s_efo[e]), 0); }, [](int, int) {}, s_warp);
    l.real_TK = min(fit, o.TK_alloc);
    if (first && threadIdx.x == 0) o.naept[o.N] = l.real_TK;
  }
  return l;
}

// ---- scatter: one thread per (row, slot) ----
// A unit of 32 rows is KP warps (KP: slots a row, rounded up to a power of two), slots fastest: the loads of indices and
// probabilities and the three token-major stores of a warp then fall into consecutive addresses, and a launch spreads over
// K times as many SMs as with one row a thread (16384 rows, K=8, E=128: 11.0 -> 6.0 us).
// mask(e) / off(e): rows of the unit that selected e, and e's rows in the units before; base(): entries before the unit.
// Every thread of the block takes part, also for a unit beyond the last.
template <int KP, typename M, typename F, typename B>
__device__ __forceinline__ void scatter_unit(const TopkOut& o, const Layout& l, const int* s_efo, int* s_warp, int unit, M mask,
                                             F off, B base) {
  constexpr int RPW = 32 / KP;                              // rows per warp
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = lane & (KP - 1), rw = lane / KP;            // slot; row within the warp
  const int r = (warp % KP) * RPW + rw;                     // row within the unit
  const int row = unit * 32 + r;
  const bool in = row < o.N && k < o.K;
  int e = in ? o.idx[(size_t)row * o.K + k] : -1;
  if (e < 0 || e >= o.E) e = -1;
  int pos = 0;
  if (e >= 0) {
    pos = s_efo[e] + off(e) + __popc(mask(e) & ((1u << r) - 1u));
    if (pos >= l.limit) e = -1;
  }
  const uint32_t ball = __ballot_sync(0xffffffffu, e >= 0);
  if (lane == 0) s_warp[warp] = __popc(ball);
  __syncthreads();
  int tm_base = 0;
  if (unit * 32 < o.N) {
    if (!l.cut) tm_base = base();
    else
      for (int j = 0; j < o.E; ++j) tm_base += max(min(off(j), l.limit - s_efo[j]), 0);
  }
  for (int w = warp - warp % KP; w < warp; ++w) tm_base += s_warp[w];
  const int row_base = tm_base + __popc(ball & ((1u << (rw * KP)) - 1u));        // rw * KP <= 31
  const int cap = l.cut ? l.real_TK : o.TK_alloc;
  if (row < o.N && k == 0) o.naept[row] = min(row_base, cap);
  int rank = 0;
  if (o.lane_order == 0) {
#pragma unroll
    for (int j = 0; j < KP; ++j) {
      const int ej = __shfl_sync(0xffffffffu, e, rw * KP + j);
      rank += (ej >= 0 && ej < e) ? 1 : 0;
    }
  } else {
    rank = __popc(ball & ((1u << lane) - 1u)) - __popc(ball & ((1u << (rw * KP)) - 1u));
  }
  if (e >= 0) {
    const int tm = row_base + rank;
    const bool kept = tm < cap;
    o.x_gather[pos] = kept ? row : 0;
    o.s_scatter[pos] = kept ? tm : l.real_TK;
    if (kept) {
      o.s_rev[tm] = pos;
      o.src_idx[tm] = row * o.K + k;
      if (tm < o.TKp_alloc) o.scores[tm] = o.probs[(size_t)row * o.K + k];
    }
  }
}

// ---- pad rows and over-allocated tails ---- (thread gtid of nthreads, whole warps)
// A warp takes an expert's padding, so that nobody has to look for the expert of a row (a binary search by a thread per row
// before: 64 rows x 8 over 128 experts 13.8 -> 12.3 us between two events, 8192 x 8 over 8 19.5 -> 17.4).
__device__ __forceinline__ void fill_pads(const TopkOut& o, const Layout& l, const int* s_efo, const int* s_base, int gtid,
                                          int nthreads) {
  const bool sentinel = o.pad_mode == 0 || l.cut;
  for (int e = gtid >> 5; e < o.E; e += nthreads >> 5) {
    const int first = s_efo[e] + s_base[e + 1] - s_base[e], end = min(s_efo[e + 1], l.limit);
    for (int pos = first + (gtid & 31); pos < end; pos += 32) {
      o.x_gather[pos] = 0;
      o.s_scatter[pos] = sentinel ? l.real_TK : l.real_TK + (s_efo[e] - s_base[e]) + (pos - first);
    }
  }
  // the tail, where virtual numbering continues, and what a cut pass leaves of an alignment step
  for (int pos = min(l.tot_p, l.limit) + gtid; pos < o.TKp_alloc; pos += nthreads) {
    o.x_gather[pos] = 0;
    o.s_scatter[pos] = sentinel || pos < l.tot_p ? l.real_TK : pos;
  }
  for (int i = l.real_TK + gtid; i < o.TKp_alloc; i += nthreads) o.scores[i] = 0.f;
  for (int i = l.real_TK + gtid; i < o.TK_alloc; i += nthreads) {
    o.s_rev[i] = 0;
    o.src_idx[i] = 0;
  }
}

template <int KP>
__global__ void __launch_bounds__(KP > 8 ? 32 * KP : 256)
scatter_fill_kernel(const TopkOut o, const uint32_t* __restrict__ mask, const int* __restrict__ unit_off,
                    const int* __restrict__ unit_base, int scatter_blocks) {
  extern __shared__ int s_mem[];
  int* s_efo = s_mem;                // [E+1] padded offsets
  int* s_base = s_mem + (o.E + 1);   // [E+1] unpadded offsets
  int* s_warp = s_base + (o.E + 1);  // [33]
  const int* counts = o.counts;
  const Layout l = block_layout(o, [&](int e) { return counts[e]; }, s_efo, s_base, s_warp, blockIdx.x == 0);
  if ((int)blockIdx.x < scatter_blocks) {
    const int unit = blockIdx.x * ((int)blockDim.x / (32 * KP)) + (threadIdx.x >> 5) / KP;
    scatter_unit<KP>(
        o, l, s_efo, s_warp, unit, [&](int e) { return mask[(size_t)unit * o.E + e]; },
        [&](int e) { return unit_off[(size_t)unit * o.E + e]; }, [&]() { return unit_base[unit]; });
  }
  fill_pads(o, l, s_efo, s_base, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// ---------------------------------------------------------------------------
// The same metadata from one cluster of CTAs, for problems small enough that three launches and the gaps between them cost more
// than the work: masks and counts stay in shared memory, each CTA takes a run of units, and what the CTAs before it hold of an
// expert is read out of their shared memory.  Between two events, launches included: 64 rows x 8 over 128 experts 17.4 -> 12.3
// us, 1024 x 8 over 8 experts 18.5 -> 14.3; from 2048 x 8 on the scatter wants more than eight SMs (17.4 against 19.4).
constexpr int kMetaCluster = 8, kMetaThreads = 512;
constexpr int kMetaEntries = 8192;                   // rows x slots up to which it is taken
constexpr size_t kMetaSmem = 48 * 1024;

__host__ __device__ inline size_t meta_cluster_smem(int units, int E) {
  const int upc = (units + kMetaCluster - 1) / kMetaCluster;
  return sizeof(int) * ((size_t)upc * E * 2 + upc + 1 + 3 * (size_t)E + 2 * (E + 1) + 33);
}

__device__ __forceinline__ int ld_cluster(const int* p, int rank) {
  uint32_t a, v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return (int)v;
}

template <int KP>
__global__ void __cluster_dims__(kMetaCluster, 1, 1) __launch_bounds__(kMetaThreads)
metadata_cluster_kernel(const TopkOut o) {
  extern __shared__ int s_mem[];
  const int E = o.E, K = o.K, tid = threadIdx.x, rank = blockIdx.x;
  const int units = (o.N + 31) / 32, upc = (units + kMetaCluster - 1) / kMetaCluster;
  const int u0 = min(rank * upc, units), nu = min(upc, units - u0);
  uint32_t* s_mask = reinterpret_cast<uint32_t*>(s_mem);     // [upc][E]
  int* s_off = s_mem + (size_t)upc * E;                      // [upc][E] rows of e in this CTA's units before
  int* s_valid = s_off + (size_t)upc * E;                    // [upc + 1] entries of a unit, then of the units before it
  int* s_cnt = s_valid + upc + 1;                            // [E] rows of e in this CTA's units (read by the others)
  int* s_tot = s_cnt + E;                                    // [E] rows of e
  int* s_first = s_tot + E;                                  // [E] rows of e in the CTAs before
  int* s_efo = s_first + E;
  int* s_base = s_efo + (E + 1);
  int* s_warp = s_base + (E + 1);

  for (int i = tid; i < nu * E; i += kMetaThreads) s_mask[i] = 0u;
  for (int i = tid; i <= upc; i += kMetaThreads) s_valid[i] = 0;
  __syncthreads();
  const int row0 = u0 * 32, n_in = max(min(o.N - row0, nu * 32), 0) * K;
  for (int i = tid; i < n_in; i += kMetaThreads) {
    const int e = o.idx[(size_t)row0 * K + i], r = i / K;
    if (e >= 0 && e < E) {
      atomicOr(&s_mask[(r >> 5) * E + e], 1u << (r & 31));
      atomicAdd(&s_valid[r >> 5], 1);                        // whole numbers: the order does not matter
    }
  }
  __syncthreads();
  for (int e = tid; e < E; e += kMetaThreads) {
    int run = 0;
    for (int u = 0; u < nu; ++u) {
      s_off[u * E + e] = run;
      run += __popc(s_mask[u * E + e]);
    }
    s_cnt[e] = run;
  }
  if (tid == kMetaThreads - 1) {
    int run = 0;
    for (int u = 0; u <= upc; ++u) {
      const int v = s_valid[u];
      s_valid[u] = run;
      run += v;
    }
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  for (int e = tid; e < E; e += kMetaThreads) {
    int v[kMetaCluster], tot = 0, before = 0;
#pragma unroll
    for (int q = 0; q < kMetaCluster; ++q) v[q] = ld_cluster(s_cnt + e, q);
#pragma unroll
    for (int q = 0; q < kMetaCluster; ++q) {
      if (q < rank) before += v[q];
      tot += v[q];
    }
    s_tot[e] = tot;
    s_first[e] = before;
    if (rank == 0) o.counts[e] = tot;
  }
  int entries = 0, all_entries = 0;                          // of the CTAs before, of all
#pragma unroll
  for (int q = 0; q < kMetaCluster; ++q) {
    const int v = ld_cluster(s_valid + upc, q);
    if (q < rank) entries += v;
    all_entries += v;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // this CTA has read the others' shared memory
  if (rank == 0 && tid == 0) o.naept[o.N] = min(all_entries, o.TK_alloc);    // (a cut pass writes it again, below)
  __syncthreads();
  const Layout l = block_layout(o, [&](int e) { return s_tot[e]; }, s_efo, s_base, s_warp, rank == 0);
  constexpr int UPB = kMetaThreads / (32 * KP);              // units of a pass over the block
  for (int ub = 0; ub < nu; ub += UPB) {
    const int lu = ub + (tid >> 5) / KP;
    const int unit = lu < nu ? u0 + lu : units;              // `units`: no rows
    scatter_unit<KP>(
        o, l, s_efo, s_warp, unit, [&](int e) { return s_mask[lu * E + e]; },
        [&](int e) { return s_first[e] + s_off[lu * E + e]; }, [&]() { return entries + s_valid[lu]; });
    __syncthreads();                                         // s_warp is written again
  }
  fill_pads(o, l, s_efo, s_base, rank * kMetaThreads + tid, kMetaCluster * kMetaThreads);
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");        // nobody reads this CTA's shared memory any more
}

// ---------------------------------------------------------------------------
template <typename T>
__global__ void count_kernel(const T* __restrict__ ids, int64_t n, int E, int* __restrict__ count) {
  extern __shared__ int s_cnt[];
  const bool use_smem = E <= 8192;
  if (use_smem) {
    for (int e = threadIdx.x; e < E; e += blockDim.x) s_cnt[e] = 0;
    __syncthreads();
  }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = (int64_t)ids[i];
    if (e >= 0 && e < E) atomicAdd(use_smem ? &s_cnt[e] : &count[e], 1);
  }
  if (use_smem) {
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x)
      if (s_cnt[e]) atomicAdd(&count[e], s_cnt[e]);
  }
}

__global__ void __launch_bounds__(kRtThreads)
cumsum_kernel(const int* __restrict__ count, int E, int* __restrict__ cumsum) {
  __shared__ int s_warp[33];
  block_excl_scan(E, [&](int e) { return count[e]; }, [&](int e, int ex) { cumsum[e] = ex + count[e]; }, s_warp);
}

}  // namespace smoe

using namespace smoe;

extern "C" {

int smoe_count_cumsum(const void* ids, int ids_is_int64, int64_t n, int64_t E, int32_t* count, int32_t* cumsum,
                      void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (E <= 0 || n < 0 || !count) return SMOE_ERR_ARG;
  cudaMemsetAsync(count, 0, sizeof(int) * E, stream);
  if (n > 0) {
    const int threads = 512;
    int blocks = (int)((n + threads * 4 - 1) / (threads * 4));
    if (blocks > 592) blocks = 592;
    const size_t smem = E <= 8192 ? sizeof(int) * E : 0;
    if (ids_is_int64)
      count_kernel<int64_t><<<blocks, threads, smem, stream>>>((const int64_t*)ids, n, (int)E, count);
    else
      count_kernel<int32_t><<<blocks, threads, smem, stream>>>((const int32_t*)ids, n, (int)E, count);
  }
  if (cumsum) cumsum_kernel<<<1, kRtThreads, 0, stream>>>(count, (int)E, cumsum);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int64_t smoe_topk_metadata_workspace(int64_t N, int64_t E) {
  const int64_t units = (N + 31) / 32 + 1;
  return (units * E * 2 + units * 2 + 64) * 4;
}

int smoe_topk_metadata(const int32_t* idx, const float* probs, int64_t N, int64_t K, int64_t E, int64_t alignment,
                       int64_t TK_alloc, int64_t TKp_alloc, int lane_order, int pad_mode, int32_t* efo,
                       int32_t* x_gather_idx, int32_t* s_scatter_idx, int32_t* s_reverse_scatter_idx, int32_t* naept,
                       float* topk_scores, int32_t* score_src_idx, int32_t* counts, void* workspace, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (K <= 0 || K > kMaxTopk || E <= 0 || E > 4096 || N < 0 || alignment <= 0) return SMOE_ERR_SHAPE;
  if (N * K >= (int64_t)1 << 31 || TKp_alloc >= (int64_t)1 << 31) return SMOE_ERR_SHAPE;
  if (!workspace || !efo || !counts) return SMOE_ERR_ARG;
  TK_alloc = TK_alloc < 0 ? 0 : TK_alloc >= (int64_t)1 << 31 ? ((int64_t)1 << 31) - 1 : TK_alloc;
  const int units = (int)((N + 31) / 32);
  TopkOut o{idx, probs, (int)N, (int)K, (int)E, (int)alignment, (int)TK_alloc, (int)TKp_alloc, lane_order, pad_mode, efo,
            x_gather_idx, s_scatter_idx, s_reverse_scatter_idx, naept, topk_scores, score_src_idx, counts};
  // slots a row, rounded up: a unit of 32 rows is that many warps of the scatter
  const int kp = K <= 1 ? 1 : K <= 2 ? 2 : K <= 4 ? 4 : K <= 8 ? 8 : 16;
  if (N * K <= kMetaEntries && TKp_alloc <= 4 * kMetaEntries && meta_cluster_smem(units, (int)E) <= kMetaSmem) {
    auto one = kp == 1   ? metadata_cluster_kernel<1>
               : kp == 2 ? metadata_cluster_kernel<2>
               : kp == 4 ? metadata_cluster_kernel<4>
               : kp == 8 ? metadata_cluster_kernel<8>
                         : metadata_cluster_kernel<16>;
    one<<<kMetaCluster, kMetaThreads, meta_cluster_smem(units, (int)E), stream>>>(o);
    return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
  }
  uint32_t* mask = (uint32_t*)workspace;
  int* unit_off = (int*)(mask + (size_t)(units + 1) * E);
  int* unit_valid = unit_off + (size_t)(units + 1) * E;
  int* unit_base = unit_valid + units + 1;
  const int ublocks = (units + kUnitsPerBlock - 1) / kUnitsPerBlock;
  if (ublocks > 0)
    unit_masks_kernel<<<ublocks, kRtThreads, 0, stream>>>(idx, (int)N, (int)K, (int)E, mask, unit_valid);
  scan_kernel<<<(int)E + 1, kRtThreads, 0, stream>>>(mask, unit_valid, units, (int)E, (int)N, (int)TK_alloc, unit_off,
                                                     counts, unit_base, naept);
  const int threads = kp > 8 ? 32 * kp : kRtThreads, units_per_block = threads / (32 * kp);
  const int sblocks = (units + units_per_block - 1) / units_per_block;
  int fill_blocks = (int)((TKp_alloc + threads - 1) / threads);
  if (fill_blocks > 296) fill_blocks = 296;
  int grid = sblocks > fill_blocks ? sblocks : fill_blocks;
  if (grid < 1) grid = 1;
  const size_t smem = sizeof(int) * (2 * (E + 1) + 33);
  auto scatter_fill = kp == 1   ? scatter_fill_kernel<1>
                      : kp == 2 ? scatter_fill_kernel<2>
                      : kp == 4 ? scatter_fill_kernel<4>
                      : kp == 8 ? scatter_fill_kernel<8>
                                : scatter_fill_kernel<16>;
  scatter_fill<<<grid, threads, smem, stream>>>(o, mask, unit_off, unit_base, sblocks);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// smoe_topk_metadata_static: the same routing-metadata computation for callers
// that must not allocate - code running inside a CUDA-graph capture or a stream
// callback, a serving loop that forbids cudaMalloc after start-up, a host
// framework whose allocator this library cannot reach.  The scratch that
// smoe_topk_metadata takes from its caller lives here in a fixed device array
// that every GPU loading the library holds until the process exits.
// ---------------------------------------------------------------------------
namespace smoe {

constexpr size_t kStaticScratchBytes = 1u << 20;   // 1 MiB: e.g. 16384 rows x 128 experts, or 65536 rows x 32
static __device__ __align__(256) unsigned char g_topk_scratch[kStaticScratchBytes];

constexpr int kMaxDevices = 64;
static void* g_scratch_addr[kMaxDevices] = {nullptr};   // device address of g_topk_scratch, per device

// In host code the array's name is only a handle; the address a kernel can use
// comes from cudaGetSymbolAddress, asked once per device with that device current.
static int static_scratch(void** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return SMOE_ERR_ARG;
  if (g_scratch_addr[dev] == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_topk_scratch) != cudaSuccess || p == nullptr) return SMOE_ERR_DRIVER;
    g_scratch_addr[dev] = p;
  }
  *out = g_scratch_addr[dev];
  return SMOE_OK;
}

}  // namespace smoe

extern "C" {

int64_t smoe_topk_metadata_static_capacity(void) { return (int64_t)smoe::kStaticScratchBytes; }

int smoe_topk_metadata_static(const int32_t* idx, const float* probs, int64_t N, int64_t K, int64_t E,
                              int64_t alignment, int64_t TK_alloc, int64_t TKp_alloc, int lane_order, int pad_mode,
                              int32_t* efo, int32_t* x_gather_idx, int32_t* s_scatter_idx,
                              int32_t* s_reverse_scatter_idx, int32_t* naept, float* topk_scores,
                              int32_t* score_src_idx, int32_t* counts, void* stream) {
  if (N < 0 || E <= 0) return SMOE_ERR_SHAPE;
  // the scratch need grows with rows x experts; anything beyond the fixed array is refused, never truncated
  if (smoe_topk_metadata_workspace(N, E) > (int64_t)smoe::kStaticScratchBytes) return SMOE_ERR_SHAPE;
  void* scratch = nullptr;
  const int rc = smoe::static_scratch(&scratch);
  if (rc != SMOE_OK) return rc;
  // nothing in the scratch has to start at zero: the first kernel clears the bit masks it builds on, and every
  // other word is written before it is read, so the previous call's contents are harmless
  return smoe_topk_metadata(idx, probs, N, K, E, alignment, TK_alloc, TKp_alloc, lane_order, pad_mode, efo,
                            x_gather_idx, s_scatter_idx, s_reverse_scatter_idx, naept, topk_scores, score_src_idx,
                            counts, scratch, stream);
}

}  // extern "C"
