// Token-side kernels: the top-k weighted gather-reduce ("combine"), the score
// gather to expert-sorted rows, the ds partial-sum/permute, and the router's
// top-k softmax forward/backward.  All reductions run in a fixed order, so two
// runs on the same inputs give the same bits.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "smoe_b200.h"

namespace smoe {

__device__ __forceinline__ void acc_bf16x8(const uint4& v, float w, float (&a)[8]) {
  const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    a[2 * i] = fmaf(w, __uint_as_float(u[i] << 16), a[2 * i]);
    a[2 * i + 1] = fmaf(w, __uint_as_float(u[i] & 0xFFFF0000u), a[2 * i + 1]);
  }
}
__device__ __forceinline__ uint32_t cvt_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// One block per token; a thread owns 8 consecutive columns (16-byte accesses).
// Lanes of the token are added in ascending order.  Being the last kernel of a forward pass, it may also leave the status word
// where the host looks for it (`host_word`, null: not): a kernel of its own for that one store costs a launch, 3 us and a gap.
// ROWS: rows of a token whose loads are in flight together
template <int ROWS>
__global__ void __launch_bounds__(512)
combine_kernel(const uint4* __restrict__ y, const int* __restrict__ s_rev, const int* __restrict__ naept,
               const float* __restrict__ scores, uint4* __restrict__ out, int H8, const int* __restrict__ status,
               volatile int* host_word) {
  const int64_t t = blockIdx.x;
  if (host_word != nullptr && t == 0 && threadIdx.x == 0) *host_word = *status;
  const int beg = naept[t], end = naept[t + 1];
  for (int c = threadIdx.x; c < H8; c += blockDim.x) {
    float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int j = beg; j < end; j += ROWS) {
      const int n = end - j;                 // rows of this batch that exist; the same for the whole block
      uint4 v[ROWS];
      float w[ROWS];
#pragma unroll
      for (int u = 0; u < ROWS; ++u) {
        if (u >= n) break;
        v[u] = y[(int64_t)s_rev[j + u] * H8 + c];
        w[u] = scores ? scores[j + u] : 1.0f;
      }
#pragma unroll
      for (int u = 0; u < ROWS; ++u) {
        if (u >= n) break;
        acc_bf16x8(v[u], w[u], a);
      }
    }
    out[t * H8 + c] = make_uint4(cvt_bf16x2(a[0], a[1]), cvt_bf16x2(a[2], a[3]), cvt_bf16x2(a[4], a[5]),
                                 cvt_bf16x2(a[6], a[7]));
  }
}

__global__ void gather_scores_kernel(const float* __restrict__ scores, const int* __restrict__ s_scatter, int64_t rows,
                                     float* __restrict__ s) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < rows) s[i] = scores[s_scatter[i]];
}

// Entries at or beyond *real_tk (over-allocated tail) are written as 0 and never scattered.
__global__ void ds_finalize_kernel(const float* __restrict__ part, int partials, int64_t rows,
                                   const int* __restrict__ s_rev, int64_t TK, const int* __restrict__ real_tk,
                                   float* __restrict__ ds, const int* __restrict__ src_idx,
                                   float* __restrict__ scatter_out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= TK) return;
  float a = 0.f;
  const bool real = real_tk == nullptr || i < *real_tk;
  if (real) {
    const int64_t p = s_rev[i];
    for (int t = 0; t < partials; ++t) a += part[(int64_t)t * rows + p];
    if (scatter_out) scatter_out[src_idx[i]] = a;
  }
  if (ds) ds[i] = a;
}

// The same sums, written to the token's slots.  A block takes 64 slots of the table: it first puts the entries of their tokens down at
// the slots they came from, so that a slot finds its entry with one look (or none: masked, zero) and every store is in order.
// Bound by latency (a few hundred bytes a thread in a chain of loads), so blocks are small and a thread's partial sums are loaded
// eight at a time, added in order.  Against a thread searching its token's entries, in blocks of 256, T=1024, K=8, 16 partials:
// 20.5 -> 10.3 us between events, from a cold L2; T=8192 K=8, 12 partials 18.5 -> 10.2; K=1, where nothing was searched, the same up
// to T=8192 and one to two us more from T=16384 on.
constexpr int kDsSlots = 64;

__global__ void __launch_bounds__(kDsSlots)
ds_slots_kernel(const float* __restrict__ part, int partials, int64_t rows, const int* __restrict__ s_rev,
                const int* __restrict__ naept, const int* __restrict__ src_idx, int64_t slots, int K, float* __restrict__ ds) {
  __shared__ int s_entry[kDsSlots];
  const int64_t i0 = blockIdx.x * (int64_t)kDsSlots, i = i0 + threadIdx.x;
  s_entry[threadIdx.x] = -1;
  __syncthreads();
  const int64_t t0 = i0 / K, t1 = (min(i0 + kDsSlots, slots) - 1) / K;
  for (int j = naept[t0] + threadIdx.x, end = naept[t1 + 1]; j < end; j += kDsSlots) {
    const int64_t at = src_idx[j] - i0;
    if (at >= 0 && at < kDsSlots) s_entry[at] = j;
  }
  __syncthreads();
  if (i >= slots) return;
  float a = 0.f;
  const int j = s_entry[threadIdx.x];
  if (j >= 0) {
    const float* p = part + s_rev[j];
    for (int q0 = 0; q0 < partials; q0 += 8) {
      float v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = q0 + q < partials ? p[(int64_t)(q0 + q) * rows] : 0.f;
#pragma unroll
      for (int q = 0; q < 8; ++q) if (q0 + q < partials) a += v[q];
    }
  }
  ds[i] = a;
}

// One warp per row: K rounds of arg-max (lowest index wins ties), then softmax
// over the K selected logits in fp32.  A NaN logit counts as -inf.  A row with
// fewer than K finite logits still gets K distinct, in-range indices: once the
// finite ones are used up, the lowest not-yet-selected index is taken with a
// score of exactly zero (all K scores are zero when nothing in the row is finite).
// Bound by instruction issue (K passes over a lane's PER slots), so PER is the smallest power of two that holds E / 32
// experts: with 32 slots for every E, T=4096, E=32, K=8 took 20 us.  Logits are f32, or bf16 as the router's GEMM left
// them.
__device__ __forceinline__ float logit_of(const float* p, size_t i) { return p[i]; }
__device__ __forceinline__ float logit_of(const __nv_bfloat16* p, size_t i) { return __bfloat162float(p[i]); }

template <int PER, typename L>
__global__ void __launch_bounds__(256)
topk_softmax_kernel(const L* __restrict__ logits, int64_t T, int E, int K, float* __restrict__ scores,
                    int* __restrict__ idx) {
  const int lane = threadIdx.x & 31;
  const int64_t row = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= T) return;
  float v[PER];
  const int per = (E + 31) / 32;
  uint32_t open = 0;       // bit i: this lane's i-th expert exists and has not been selected yet
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = i * 32 + lane;
    const bool in = (i < per && e < E);
    const float x = in ? logit_of(logits, row * E + e) : -INFINITY;
    v[i] = (x != x) ? -INFINITY : x;
    if (in) open |= 1u << i;
  }
  float sel_v = 0.f;
  int sel_i = 0;
  float vmax = 0.f;
  for (int k = 0; k < K; ++k) {
    float bv = -INFINITY;
    int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      if (i < per && ((open >> i) & 1u)) {
        const int e = i * 32 + lane;
        if (bi == 0x7fffffff || v[i] > bv) { bv = v[i]; bi = e; }
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffff, bv, d);
      const int oi = __shfl_xor_sync(0xffffffff, bi, d);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if (k == 0) vmax = bv;
    if (lane == k) { sel_v = bv; sel_i = bi; }
    if ((bi & 31) == lane) open &= ~(1u << (bi >> 5));     // K <= E: an open slot always exists
  }
  float ex = (lane < K && sel_v != -INFINITY) ? expf(sel_v - vmax) : 0.f;
  float sum = ex;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffff, sum, d);
  if (lane < K) {
    scores[row * K + lane] = sum > 0.f ? ex / sum : 0.f;
    idx[row * K + lane] = sel_i;
  }
}

__device__ __forceinline__ void store_grad(float* p, size_t i, float v) { p[i] = v; }
__device__ __forceinline__ void store_grad(__nv_bfloat16* p, size_t i, float v) { p[i] = __float2bfloat16_rn(v); }

template <typename L>
__global__ void __launch_bounds__(256)
topk_softmax_bwd_kernel(const float* __restrict__ scores, const int* __restrict__ idx, const float* __restrict__ ds,
                        int64_t T, int E, int K, L* __restrict__ dlogits) {
  const int lane = threadIdx.x & 31;
  const int64_t row = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= T) return;
  for (int e = lane; e < E; e += 32) store_grad(dlogits, row * E + e, 0.f);
  __syncwarp();
  const float s = lane < K ? scores[row * K + lane] : 0.f;
  const float g = lane < K ? ds[row * K + lane] : 0.f;
  float dot = s * g;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) dot += __shfl_xor_sync(0xffffffff, dot, d);
  if (lane < K) {
    const int e = idx[row * K + lane];
    if (e >= 0 && e < E) store_grad(dlogits, row * E + e, s * (g - dot));     // an out-of-range index is ignored, never written
  }
}

// ---- switch auxiliary loss: E * sum_e (acc_e / |acc|_1) (f_e / |f|_1), acc_e = sum_t softmax(logits_t)_e ----------------
// Written out as tensor operations it is some 35 launches of 2 us per forward + backward, each with its gap.  Three kernels
// instead: per-block sums of the softmax rows, their reduction with the loss, and the gradient.  All sums in f32 in a fixed
// order.  A lane owns the experts lane, lane + 32, ...; a warp walks rows.
constexpr int kAuxBlocks = 148, kAuxWarps = 8;
constexpr float kAuxEps = 1e-12f;      // torch.nn.functional.normalize's lower bound of a norm

// softmax of one row into v (0 beyond E)
template <int PER, typename L>
__device__ __forceinline__ void softmax_row(const L* __restrict__ logits, size_t row, int E, int lane, float (&v)[PER]) {
  float m = -INFINITY;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = i * 32 + lane;
    v[i] = e < E ? logit_of(logits, row * E + e) : -INFINITY;
    m = fmaxf(m, v[i]);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffff, m, d));
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    v[i] = i * 32 + lane < E ? expf(v[i] - m) : 0.f;
    sum += v[i];
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffff, sum, d);
  const float inv = 1.0f / sum;
#pragma unroll
  for (int i = 0; i < PER; ++i) v[i] *= inv;
}

template <int PER, typename L>
__global__ void __launch_bounds__(32 * kAuxWarps)
switch_loss_sums_kernel(const L* __restrict__ logits, int64_t T, int E, float* __restrict__ part /* [blocks, E] */) {
  __shared__ float s_acc[kAuxWarps][PER * 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float acc[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) acc[i] = 0.f;
  for (int64_t row = (int64_t)blockIdx.x * kAuxWarps + warp; row < T; row += (int64_t)gridDim.x * kAuxWarps) {
    float v[PER];
    softmax_row<PER>(logits, row, E, lane, v);
#pragma unroll
    for (int i = 0; i < PER; ++i) acc[i] += v[i];
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) s_acc[warp][i * 32 + lane] = acc[i];
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    float a = 0.f;
    for (int w = 0; w < kAuxWarps; ++w) a += s_acc[w][e];
    part[(size_t)blockIdx.x * E + e] = a;
  }
}

// sum over a block of 256 threads, in a fixed order, to every thread
__device__ __forceinline__ float block_sum(float x, float* s_red) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(0xffffffff, x, d);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = x;
  __syncthreads();
  float a = 0.f;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) a += s_red[w];
  return a;
}

// loss, and grad[e] = d loss / d acc_e
__global__ void __launch_bounds__(256)
switch_loss_finish_kernel(const float* __restrict__ part, int blocks, const int* __restrict__ freq, int E,
                          float* __restrict__ loss, float* __restrict__ grad) {
  __shared__ float s_acc[1024], s_red[8];
  float na = 0.f, nf = 0.f;
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    float a = 0.f;
    for (int b = 0; b < blocks; ++b) a += part[(size_t)b * E + e];
    s_acc[e] = a;
    na += fabsf(a);
    nf += fabsf((float)freq[e]);
  }
  na = block_sum(na, s_red);
  nf = fmaxf(block_sum(nf, s_red), kAuxEps);
  const bool clamped = na < kAuxEps;
  na = fmaxf(na, kAuxEps);
  float dot = 0.f;
  for (int e = threadIdx.x; e < E; e += blockDim.x) dot += (s_acc[e] / na) * ((float)freq[e] / nf);
  dot = block_sum(dot, s_red);
  if (threadIdx.x == 0) *loss = (float)E * dot;
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    const float sign = s_acc[e] > 0.f ? 1.f : (s_acc[e] < 0.f ? -1.f : 0.f);
    grad[e] = (float)E * ((float)freq[e] / nf - (clamped ? 0.f : sign * dot)) / na;
  }
}

template <int PER, typename L>
__global__ void __launch_bounds__(256)
switch_loss_bwd_kernel(const L* __restrict__ logits, int64_t T, int E, const float* __restrict__ grad,
                       const float* __restrict__ dloss, L* __restrict__ dlogits) {
  const int lane = threadIdx.x & 31;
  const int64_t row = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= T) return;
  float v[PER], g[PER], dot = 0.f;
  softmax_row<PER>(logits, row, E, lane, v);
  const float d = *dloss;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = i * 32 + lane;
    g[i] = e < E ? d * grad[e] : 0.f;
    dot = fmaf(v[i], g[i], dot);
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) dot += __shfl_xor_sync(0xffffffff, dot, s);
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = i * 32 + lane;
    if (e < E) store_grad(dlogits, row * E + e, v[i] * (g[i] - dot));
  }
}

// One thread copies the device status word into pinned, device-visible host memory: a kernel store instead of a
// device-to-host memcpy, so that it never queues behind large copies on a copy engine.
__global__ void status_post_kernel(const int* __restrict__ status, volatile int* host_word) { *host_word = *status; }

}  // namespace smoe

using namespace smoe;

extern "C" {

int smoe_combine_post(const void* y_bf16, const int32_t* s_rev, const int32_t* naept, const float* scores, void* out_bf16,
                      int64_t T, int64_t H, const int32_t* status, int32_t* pinned_host_word, void* stream) {
  if (T < 0 || H <= 0 || H % 8) return SMOE_ERR_SHAPE;
  if (((uintptr_t)y_bf16 & 15) || ((uintptr_t)out_bf16 & 15)) return SMOE_ERR_ALIGN;
  if (pinned_host_word && !status) return SMOE_ERR_ARG;
  if (T == 0) return SMOE_OK;
  const int H8 = (int)(H / 8);
  const int threads = H8 >= 512 ? 512 : ((H8 + 31) / 32) * 32;
  // A lone wave of blocks waits for its loads and asks for eight rows at once (64 tokens of 8 rows, H=2048: 11 us with four, 9
  // with eight); with many blocks an SM the registers that takes cost more warps than it gains (T=8192, H=3072: 83 and 93 us)
  auto kern = T <= 296 ? combine_kernel<8> : combine_kernel<4>;
  kern<<<(unsigned)T, threads, 0, (cudaStream_t)stream>>>((const uint4*)y_bf16, s_rev, naept, scores, (uint4*)out_bf16, H8,
                                                          status, pinned_host_word);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_combine(const void* y_bf16, const int32_t* s_rev, const int32_t* naept, const float* scores, void* out_bf16,
                 int64_t T, int64_t H, void* stream) {
  return smoe_combine_post(y_bf16, s_rev, naept, scores, out_bf16, T, H, nullptr, nullptr, stream);
}

int smoe_gather_scores(const float* scores, const int32_t* s_scatter_idx, int64_t rows, float* s, void* stream) {
  if (rows <= 0) return rows == 0 ? SMOE_OK : SMOE_ERR_SHAPE;
  gather_scores_kernel<<<(unsigned)((rows + 255) / 256), 256, 0, (cudaStream_t)stream>>>(scores, s_scatter_idx, rows,
                                                                                         s);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_ds_finalize(const float* ds_partial, int64_t partials, int64_t rows, const int32_t* s_rev, int64_t TK,
                     const int32_t* real_tk, float* ds_tm, const int32_t* src_idx, float* scatter_out, void* stream) {
  if (TK <= 0) return TK == 0 ? SMOE_OK : SMOE_ERR_SHAPE;
  if (scatter_out && !src_idx) return SMOE_ERR_ARG;
  ds_finalize_kernel<<<(unsigned)((TK + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      ds_partial, (int)partials, rows, s_rev, TK, real_tk, ds_tm, src_idx, scatter_out);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_ds_slots(const float* ds_partial, int64_t partials, int64_t rows, const int32_t* s_rev, const int32_t* naept,
                  const int32_t* src_idx, int64_t T, int64_t K, float* ds, void* stream) {
  if (T < 0 || K <= 0 || partials < 0 || T * K >= (int64_t)1 << 31) return SMOE_ERR_SHAPE;
  if (T == 0) return SMOE_OK;
  if (!naept || !ds || (rows > 0 && (!ds_partial || !s_rev || !src_idx))) return SMOE_ERR_ARG;      // no rows: all slots 0
  ds_slots_kernel<<<(unsigned)((T * K + kDsSlots - 1) / kDsSlots), kDsSlots, 0, (cudaStream_t)stream>>>(
      ds_partial, (int)partials, rows, s_rev, naept, src_idx, T * K, (int)K, ds);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_status_post(const int32_t* status, int32_t* pinned_host_word, void* stream) {
  if (!status || !pinned_host_word) return SMOE_ERR_ARG;
  status_post_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(status, pinned_host_word);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

#define SMOE_ROUTER_PER(E, F) \
  ((E) <= 32 ? F(1) : (E) <= 64 ? F(2) : (E) <= 128 ? F(4) : (E) <= 256 ? F(8) : F(32))

int smoe_router_topk(const void* logits, int bf16, int64_t T, int64_t E, int64_t K, float* scores, int32_t* idx,
                     void* stream) {
  if (T < 0 || E <= 0 || E > 1024 || K <= 0 || K > 32 || K > E) return SMOE_ERR_SHAPE;
  if (T == 0) return SMOE_OK;
  const unsigned grid = (unsigned)((T + 7) / 8);
  if (bf16) {
#define SMOE_F(P) topk_softmax_kernel<P, __nv_bfloat16>
    auto kern = SMOE_ROUTER_PER(E, SMOE_F);
#undef SMOE_F
    kern<<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)logits, T, (int)E, (int)K, scores, idx);
  } else {
#define SMOE_F(P) topk_softmax_kernel<P, float>
    auto kern = SMOE_ROUTER_PER(E, SMOE_F);
#undef SMOE_F
    kern<<<grid, 256, 0, (cudaStream_t)stream>>>((const float*)logits, T, (int)E, (int)K, scores, idx);
  }
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_topk_softmax(const float* logits, int64_t T, int64_t E, int64_t K, float* scores, int32_t* idx,
                      void* stream) {
  return smoe_router_topk(logits, 0, T, E, K, scores, idx, stream);
}

int smoe_router_topk_bwd(const float* scores, const int32_t* idx, const float* dscores, int64_t T, int64_t E, int64_t K,
                         void* dlogits, int bf16, void* stream) {
  if (T < 0 || E <= 0 || K <= 0 || K > 32) return SMOE_ERR_SHAPE;
  if (T == 0) return SMOE_OK;
  const unsigned grid = (unsigned)((T + 7) / 8);
  if (bf16)
    topk_softmax_bwd_kernel<__nv_bfloat16><<<grid, 256, 0, (cudaStream_t)stream>>>(scores, idx, dscores, T, (int)E, (int)K,
                                                                    (__nv_bfloat16*)dlogits);
  else
    topk_softmax_bwd_kernel<float><<<grid, 256, 0, (cudaStream_t)stream>>>(scores, idx, dscores, T, (int)E, (int)K,
                                                                    (float*)dlogits);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_topk_softmax_bwd(const float* scores, const int32_t* idx, const float* dscores, int64_t T, int64_t E,
                          int64_t K, float* dlogits, void* stream) {
  return smoe_router_topk_bwd(scores, idx, dscores, T, E, K, dlogits, 0, stream);
}

int64_t smoe_switch_loss_workspace(int64_t E) { return E > 0 ? kAuxBlocks * E * (int64_t)sizeof(float) : 0; }

int smoe_switch_loss(const void* logits, int bf16, const int32_t* freq, int64_t T, int64_t E, float* loss, float* grad,
                     void* workspace, void* stream) {
  if (T < 0 || E <= 0 || E > 1024) return SMOE_ERR_SHAPE;
  if ((T > 0 && !logits) || !freq || !loss || !grad || !workspace) return SMOE_ERR_ARG;
  int64_t blocks = (T + kAuxWarps - 1) / kAuxWarps;
  if (blocks > kAuxBlocks) blocks = kAuxBlocks;
  float* part = (float*)workspace;
  if (blocks > 0) {
    if (bf16) {
#define SMOE_F(P) switch_loss_sums_kernel<P, __nv_bfloat16>
      auto kern = SMOE_ROUTER_PER(E, SMOE_F);
#undef SMOE_F
      kern<<<(unsigned)blocks, 32 * kAuxWarps, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)logits, T, (int)E, part);
    } else {
#define SMOE_F(P) switch_loss_sums_kernel<P, float>
      auto kern = SMOE_ROUTER_PER(E, SMOE_F);
#undef SMOE_F
      kern<<<(unsigned)blocks, 32 * kAuxWarps, 0, (cudaStream_t)stream>>>((const float*)logits, T, (int)E, part);
    }
  }
  switch_loss_finish_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(part, (int)blocks, freq, (int)E, loss, grad);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_switch_loss_bwd(const void* logits, int bf16, const float* grad, const float* dloss, int64_t T, int64_t E,
                         void* dlogits, void* stream) {
  if (T < 0 || E <= 0 || E > 1024) return SMOE_ERR_SHAPE;
  if (T == 0) return SMOE_OK;
  if (!logits || !grad || !dloss || !dlogits) return SMOE_ERR_ARG;
  const unsigned grid = (unsigned)((T + 7) / 8);
  if (bf16) {
#define SMOE_F(P) switch_loss_bwd_kernel<P, __nv_bfloat16>
    auto kern = SMOE_ROUTER_PER(E, SMOE_F);
#undef SMOE_F
    kern<<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)logits, T, (int)E, grad, dloss,
                                                 (__nv_bfloat16*)dlogits);
  } else {
#define SMOE_F(P) switch_loss_bwd_kernel<P, float>
    auto kern = SMOE_ROUTER_PER(E, SMOE_F);
#undef SMOE_F
    kern<<<grid, 256, 0, (cudaStream_t)stream>>>((const float*)logits, T, (int)E, grad, dloss, (float*)dlogits);
  }
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

}  // extern "C"
