// MXFP8 1x32 ue8m0 block-scaled quantizers (HBM-bound; 128-bit global accesses,
// warp-shuffle amax, 32-bit packed scale stores).
//
// Rule for one group of 32 values (amax = max |v|):
//   e8m0 = max(bexp(amax) - 8 + (mantissa(amax) > 0x600000), 0), 0 for zero/denormal amax
//   q    = cvt.rn.satfinite.e4m3( v * 2^(127 - e8m0) )
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx.cuh"
#include "smoe_b200.h"

namespace smoe {

__device__ __forceinline__ int q_e8m0_of(float amax) {
  const int bits = __float_as_int(amax);
  const int bexp = (bits >> 23) & 0xFF;
  const int e = bexp - 8 + ((bits & 0x7FFFFF) > 0x600000 ? 1 : 0);
  return bexp > 0 ? max(e, 0) : 0;
}
__device__ __forceinline__ float q_scale_of(int e8m0) {
  return __int_as_float(min(max(254 - e8m0, 1), 254) << 23);
}
__device__ __forceinline__ uint32_t q_pack4(float a, float b, float c, float d) {
  uint16_t lo, hi;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(lo) : "f"(b), "f"(a));
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(hi) : "f"(d), "f"(c));
  return (uint32_t)lo | ((uint32_t)hi << 16);
}
__device__ __forceinline__ void bf16x8_to_f32(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}
__device__ __forceinline__ size_t isa_offset(size_t row, size_t g, size_t k_tiles) {
  return ((row >> 7) * k_tiles + (g >> 2)) * 512 + (row & 31) * 16 + ((row & 127) >> 5) * 4 + (g & 3);
}

__device__ __forceinline__ uint32_t q_max_bf16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// max of the magnitudes of two bf16 pairs, element by element; the sign bits are those of the product
__device__ __forceinline__ uint32_t q_max_abs_bf16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// q_e8m0_of of two magnitudes, as bf16 pairs: the exponent after rounding up a mantissa above 0x60, less 8, not below 0
__device__ __forceinline__ uint32_t q_e8m0x2(uint32_t m) {
  const uint32_t e = ((m + 0x001F001Fu) >> 7) & 0x01FF01FFu;
  uint32_t r;
  asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(e), "r"(0x00080008u));
  return r - 0x00080008u;
}
// and their scales, 2^(127 - e) as bf16; e <= 247, the exponent of infinity: every maximum starts from 0 and drops NaN
__device__ __forceinline__ uint32_t q_scalex2(uint32_t e2) { return (0x00FE00FEu - e2) << 7; }
// A bf16 pair times a pair of powers of two, in f32: exact, one instruction a value where unpacking and multiplying take two, and
// on another pipe than the conversions; adding -0 keeps the sign of a zero
__device__ __forceinline__ float2 q_scaled(uint32_t w, uint32_t qs) {
  float2 r;
  asm("{\n\t.reg .b16 a, b, c, d;\n\t"
      "mov.b32 {a, b}, %2;\n\tmov.b32 {c, d}, %3;\n\t"
      "fma.rn.f32.bf16 %0, a, c, %4;\n\tfma.rn.f32.bf16 %1, b, d, %4;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "r"(w), "r"(qs), "f"(-0.0f));
  return r;
}
// four bf16 values of a row, each with its scale -> four e4m3 bytes
__device__ __forceinline__ uint32_t q_pack4_scaled(uint32_t a, uint32_t b, uint32_t qa, uint32_t qb) {
  const float2 x = q_scaled(a, qa), y = q_scaled(b, qb);
  return q_pack4(x.x, x.y, y.x, y.y);
}

// --------------------------------------------------------------------- rows
// One warp per row; a lane owns 8 consecutive values, 4 lanes form a group.
__global__ void __launch_bounds__(256)
quant_rows_kernel(const uint4* __restrict__ x, int64_t M, int K, uint2* __restrict__ q, uint8_t* __restrict__ raw,
                  uint8_t* __restrict__ isa, const int* __restrict__ idx, const int* __restrict__ valid_rows) {
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const int groups = K / 32, k_tiles = (K + 127) / 128;
  // with idx: output row `row` is the quantised source row idx[row] (gather fused into the quantizer);
  // rows at or beyond *valid_rows (over-allocated tail) are skipped
  const int64_t m_end = valid_rows ? min((int64_t)*valid_rows, M) : M;
  for (int64_t row = warp0; row < m_end; row += nwarps) {
    const int64_t srow = idx ? idx[row] : row;
    for (int c0 = 0; c0 < K; c0 += 256) {
      const int col = c0 + lane * 8;
      const bool in = col < K;
      float f[8];
      if (in) {
        bf16x8_to_f32(x[(srow * K + col) >> 3], f);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = 0.f;
      }
      float amax = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(f[i]));
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffff, amax, 1));
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffff, amax, 2));
      const int e = q_e8m0_of(amax);
      const float qs = q_scale_of(e);
      if (in) {
        uint2 o;
        o.x = q_pack4(f[0] * qs, f[1] * qs, f[2] * qs, f[3] * qs);
        o.y = q_pack4(f[4] * qs, f[5] * qs, f[6] * qs, f[7] * qs);
        q[(row * K + col) >> 3] = o;
      }
      // gather the 4 group bytes of a 128-column tile into one word (lanes 0 and 16)
      const uint32_t b1 = __shfl_down_sync(0xffffffff, (uint32_t)e, 4);
      const uint32_t b2 = __shfl_down_sync(0xffffffff, (uint32_t)e, 8);
      const uint32_t b3 = __shfl_down_sync(0xffffffff, (uint32_t)e, 12);
      const int g = col >> 5;
      if (in && (lane & 15) == 0) {
        const uint32_t word = (uint32_t)e | (b1 << 8) | (b2 << 16) | (b3 << 24);
        if (g + 3 < groups && (groups & 3) == 0) {       // rows of scales start on words
          if (raw) *reinterpret_cast<uint32_t*>(raw + row * groups + g) = word;
          if (isa) *reinterpret_cast<uint32_t*>(isa + isa_offset(row, g, k_tiles)) = word;
        } else {
          for (int j = 0; j < 4 && g + j < groups; ++j) {
            const uint8_t b = (uint8_t)(word >> (8 * j));
            if (raw) raw[row * groups + g + j] = b;
            if (isa) isa[isa_offset(row, g + j, k_tiles)] = b;
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------- rows, scatter form
// Copies of bytes from this CTA's shared memory to global memory by the copy engine; both addresses and the size are
// multiples of 16.  A thread waits for the copies it has issued itself.
__device__ __forceinline__ void bulk_store(void* dst, const void* src_smem, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
               ::"l"(dst), "r"((uint32_t)__cvta_generic_to_shared(src_smem)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_store_wait() {
  asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group 0;" ::: "memory");
}

// Clears the pad rows (s_scatter[row] >= real_tk) of an expert-sorted e4m3 buffer and their scales; warp w0 of nwarps.  Eight
// lanes look at a row each, so that a warp waits for one load per eight rows (and not for one per row); more than eight rows
// would leave the padding of an expert, which lies together, to a few warps.
__device__ __forceinline__ void clear_pad_rows(int64_t w0, int64_t nwarps, int lane, const int* __restrict__ s_scatter,
                                               int real_tk, int64_t m_end, uint4* __restrict__ q, int k16,
                                               uint8_t* __restrict__ isa, int k_tiles) {
  for (int64_t r0 = w0 * 8; r0 < m_end; r0 += nwarps * 8) {
    uint32_t pads = __ballot_sync(0xffffffffu, lane < 8 && r0 + lane < m_end && s_scatter[r0 + lane] >= real_tk);
    while (pads) {
      const int64_t row = r0 + __ffs((int)pads) - 1;
      pads &= pads - 1;
      for (int c = lane; c < k16; c += 32) q[row * k16 + c] = make_uint4(0, 0, 0, 0);
      if (isa == nullptr) continue;
      for (int kt = lane; kt < k_tiles; kt += 32)
        *reinterpret_cast<uint32_t*>(isa + isa_offset(row, (size_t)kt * 4, k_tiles)) = 0u;
    }
  }
}

// Each token row is read and quantised ONCE and written to every expert-sorted position it occupies
// (positions s_rev[naept[t] .. naept[t+1])): HBM traffic = one read of x + the gathered output, instead of
// re-reading a token once per selected expert.  Pad rows (s_scatter[row] >= real_TK) are zero-filled so that
// the GEMM consuming the buffer only ever sees finite values.
// Blocks [0, token_blocks): one warp per token, row staged in shared memory; the remaining blocks clear pad rows.
// Bound by its writes.  A row leaves as one bulk copy per position, each issued by the lane that has read the position, so
// neither the store instructions of the row nor a chain of loads of positions stands between rows.  Against stores by the warp
// and one dependent load per pad row: T=8192, H=3072, K=E=8 61.5 -> 55 us (258 MB, 4.7 TB/s), T=16384, H=2048, K=8, 128
// experts of skewed load 92 -> 76 us, 2048 tokens of the first layer 24.6 -> 21.
__global__ void __launch_bounds__(256)
quant_rows_scatter_kernel(const uint4* __restrict__ x, int64_t T, int K, const int* __restrict__ naept,
                          const int* __restrict__ s_rev, const int* __restrict__ s_scatter,
                          const int* __restrict__ valid_rows, int64_t rows, uint4* __restrict__ q,
                          uint8_t* __restrict__ isa, int token_blocks) {
  extern __shared__ __align__(16) uint8_t s_rowbuf[];
  // a GEMM launched to do so may fetch its weights meanwhile (gemm_few.cuh)
  next_kernel_may_start();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int k_tiles = K >> 7, k16 = K >> 4;
  if ((int)blockIdx.x < token_blocks) {
    const int64_t t = (int64_t)blockIdx.x * nw + warp;
    if (t >= T) return;
    const int beg = naept[t], end = naept[t + 1];
    if (beg == end) return;
    uint8_t* sq = s_rowbuf + (size_t)warp * ((K + 4 * k_tiles + 15) & ~15);   // 16-byte aligned per warp
    uint32_t* ssc = reinterpret_cast<uint32_t*>(sq + K);
    int pos = beg + lane < end ? s_rev[beg + lane] : 0;      // of the first 32 positions, one a lane
    constexpr int NB = 8;                       // 16-byte loads in flight per lane
    for (int cb = 0; cb < K; cb += 256 * NB) {
      uint4 v[NB];
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int col = cb + b * 256 + lane * 8;
        v[b] = col < K ? x[(t * K + col) >> 3] : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int col = cb + b * 256 + lane * 8;
        const bool in = col < K;
        float f[8];
        bf16x8_to_f32(v[b], f);
        float amax = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(f[i]));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffff, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffff, amax, 2));
        const int e = q_e8m0_of(amax);
        const float qs = q_scale_of(e);
        const uint32_t b1 = __shfl_down_sync(0xffffffff, (uint32_t)e, 4);
        const uint32_t b2 = __shfl_down_sync(0xffffffff, (uint32_t)e, 8);
        const uint32_t b3 = __shfl_down_sync(0xffffffff, (uint32_t)e, 12);
        if (in) {
          uint2 o;
          o.x = q_pack4(f[0] * qs, f[1] * qs, f[2] * qs, f[3] * qs);
          o.y = q_pack4(f[4] * qs, f[5] * qs, f[6] * qs, f[7] * qs);
          *reinterpret_cast<uint2*>(sq + col) = o;
          if ((lane & 15) == 0) ssc[col >> 7] = (uint32_t)e | (b1 << 8) | (b2 << 16) | (b3 << 24);
        }
      }
    }
    fence_proxy_async_smem();
    __syncwarp();
    for (int j0 = beg; j0 < end; j0 += 32) {
      if (j0 > beg) pos = j0 + lane < end ? s_rev[j0 + lane] : 0;
      if (j0 + lane < end) bulk_store(q + (int64_t)pos * k16, sq, (uint32_t)K);
      const int n = min(32, end - j0);
      for (int j = 0; j < n; ++j) {
        const size_t row = (size_t)__shfl_sync(0xffffffffu, pos, j);
        for (int kt = lane; kt < k_tiles; kt += 32)
          *reinterpret_cast<uint32_t*>(isa + isa_offset(row, (size_t)kt * 4, k_tiles)) = ssc[kt];
      }
    }
    bulk_store_wait();
  } else {
    const int64_t m_end = valid_rows ? min((int64_t)*valid_rows, rows) : rows;
    clear_pad_rows((int64_t)(blockIdx.x - token_blocks) * nw + warp, (int64_t)(gridDim.x - token_blocks) * nw, lane,
                   s_scatter, naept[T], m_end, q, k16, isa, k_tiles);
  }
}

// ------------------------------------------------------------- scale gather
__global__ void __launch_bounds__(256)
gather_scales_isa_kernel(const uint8_t* __restrict__ raw, const int* __restrict__ idx, int64_t rows, int groups,
                         int k_tiles, uint8_t* __restrict__ isa) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= rows * k_tiles) return;
  const int64_t row = i / k_tiles;
  const int kt = (int)(i - row * k_tiles);
  const int64_t src = idx ? idx[row] : row;
  uint32_t word;
  if (kt * 4 + 3 < groups && (groups & 3) == 0) {
    word = *reinterpret_cast<const uint32_t*>(raw + src * groups + kt * 4);
  } else {
    word = 0x7F7F7F7Fu;
    for (int j = 0; kt * 4 + j < groups && j < 4; ++j)
      word = (word & ~(0xFFu << (8 * j))) | ((uint32_t)raw[src * groups + kt * 4 + j] << (8 * j));
  }
  *reinterpret_cast<uint32_t*>(isa + isa_offset(row, (size_t)kt * 4, k_tiles)) = word;
}

// ------------------------------------------------------------- row gather
// out[r, :] = q[idx[r], :] (e4m3 bytes) and the row's scales into the ISA layout of (rows, K).
// One block per output row; rows at or beyond *valid_rows (over-allocated tail) are skipped.
__global__ void __launch_bounds__(256)
gather_rows_kernel(const uint4* __restrict__ q, const uint8_t* __restrict__ raw, const int* __restrict__ idx,
                   const int* __restrict__ valid_rows, int K, uint4* __restrict__ out, uint8_t* __restrict__ isa) {
  const int64_t row = blockIdx.x;
  if (valid_rows && row >= *valid_rows) return;
  const int64_t src = idx[row];
  const int k16 = K >> 4, groups = K >> 5, k_tiles = K >> 7;
  for (int c = threadIdx.x; c < k16; c += blockDim.x) out[row * k16 + c] = q[src * k16 + c];
  for (int kt = threadIdx.x; kt < k_tiles; kt += blockDim.x)
    *reinterpret_cast<uint32_t*>(isa + isa_offset(row, (size_t)kt * 4, k_tiles)) =
        *reinterpret_cast<const uint32_t*>(raw + src * groups + kt * 4);
}

// ------------------------------------------------------------- row scatter (already quantised rows)
// The scatter form of gather_rows_kernel: every source row (e4m3 bytes + raw 1x32 scales) is read once and written
// to each expert-sorted position it occupies, s_rev[naept[t] .. naept[t+1]); pad rows are zero-filled by the
// trailing blocks, as in quant_rows_scatter_kernel.  One warp per source row.
__global__ void __launch_bounds__(256)
scatter_rows_fp8_kernel(const uint4* __restrict__ q, const uint8_t* __restrict__ raw, int64_t T, int K,
                        const int* __restrict__ naept, const int* __restrict__ s_rev,
                        const int* __restrict__ s_scatter, const int* __restrict__ valid_rows, int64_t rows,
                        uint4* __restrict__ out, uint8_t* __restrict__ isa, int token_blocks) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int k_tiles = K >> 7, k16 = K >> 4, groups = K >> 5;
  if ((int)blockIdx.x < token_blocks) {
    const int64_t t = (int64_t)blockIdx.x * nw + warp;
    if (t >= T) return;
    const int beg = naept[t], end = naept[t + 1];
    if (beg == end) return;
    for (int c0 = 0; c0 < k16; c0 += 32 * 4) {          // four 16-byte loads in flight per lane
      uint4 v[4];
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int c = c0 + b * 32 + lane;
        v[b] = c < k16 ? q[t * k16 + c] : make_uint4(0, 0, 0, 0);
      }
      for (int j = beg; j < end; ++j) {
        const int64_t pos = s_rev[j];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int c = c0 + b * 32 + lane;
          if (c < k16) out[pos * k16 + c] = v[b];
        }
      }
    }
    if (isa == nullptr) return;                          // payload only: the caller already holds the packed scales
    for (int kt = lane; kt < k_tiles; kt += 32) {
      const uint32_t word = *reinterpret_cast<const uint32_t*>(raw + t * groups + kt * 4);
      for (int j = beg; j < end; ++j)
        *reinterpret_cast<uint32_t*>(isa + isa_offset((size_t)s_rev[j], (size_t)kt * 4, k_tiles)) = word;
    }
  } else {
    const int64_t m_end = valid_rows ? min((int64_t)*valid_rows, rows) : rows;
    clear_pad_rows((int64_t)(blockIdx.x - token_blocks) * nw + warp, (int64_t)(gridDim.x - token_blocks) * nw, lane,
                   s_scatter, naept[T], m_end, out, k16, isa, k_tiles);
  }
}

// ------------------------------------------------------------------ byte transpose
// dst[b][c][r] = src[b][r][c] for a batch of [rows, cols] byte matrices, 64 x 64 tiles through shared memory.  With
// one scale per 32x32 block the transposed bytes of an e4m3 matrix ARE its transposed quantisation.
__global__ void __launch_bounds__(256)
transpose_u8_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int rows, int cols) {
  __shared__ __align__(16) uint8_t s[64][64 + 16];
  const size_t base = (size_t)blockIdx.z * rows * cols;
  const int r0 = blockIdx.y * 64, c0 = blockIdx.x * 64;
  const int tr = threadIdx.x >> 2, seg = (threadIdx.x & 3) * 16;
  *reinterpret_cast<uint4*>(&s[tr][seg]) =
      *reinterpret_cast<const uint4*>(src + base + (size_t)(r0 + tr) * cols + c0 + seg);
  __syncthreads();
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    w[i] = (uint32_t)s[seg + 4 * i][tr] | ((uint32_t)s[seg + 4 * i + 1][tr] << 8) |
           ((uint32_t)s[seg + 4 * i + 2][tr] << 16) | ((uint32_t)s[seg + 4 * i + 3][tr] << 24);
  *reinterpret_cast<uint4*>(dst + base + (size_t)(c0 + tr) * rows + r0 + seg) = make_uint4(w[0], w[1], w[2], w[3]);
}

// ------------------------------------------------------------------ columns
// Tile = 128 rows x 64 columns of src[idx].  Groups run down the rows; the
// e4m3 bytes are written transposed ([dim, rows]) so that the reduction
// dimension of the weight-gradient GEMM is contiguous.
constexpr int CT_ROWS = 128, CT_COLS = 64, CT_PITCH = CT_COLS + 2;

// ISO: one scale per 32x32 block (also emits the non-transposed bytes and the
// row-direction scales); otherwise one scale per (column, 32 rows).
// SRC_FP8: the source is e4m3 bytes with raw row-wise 1x32 scales (`src_scales`, [T, dim/32]); it is
// dequantised exactly (an e4m3 value times a power of two fits bf16) and re-quantised column-wise.
template <bool ISO, bool SRC_FP8>
__global__ void __launch_bounds__(256)
quant_cols_kernel(const void* __restrict__ src_, const uint8_t* __restrict__ src_scales,
                  const int* __restrict__ idx, int64_t rows, int dim, uint8_t* __restrict__ q_t,
                  uint8_t* __restrict__ col_isa, uint8_t* __restrict__ q, uint8_t* __restrict__ row_isa,
                  const int* __restrict__ valid_rows) {
  __shared__ __nv_bfloat16 s_in[CT_ROWS][CT_PITCH];
  __shared__ __align__(16) uint8_t s_out[CT_COLS][CT_ROWS + 16];
  __shared__ uint32_t s_sc[CT_COLS];
  const int tid = threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.x * CT_ROWS;
  // buffers sized at an upper bound: row tiles beyond the last expert's segment are never read by any GEMM
  if (valid_rows != nullptr && r0 >= *valid_rows) return;
  const int c0 = blockIdx.y * CT_COLS;
  const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(src_);

  if (SRC_FP8) {
    // 4 threads x 16 bytes cover one 64-column row; 64 rows per pass
    const uint8_t* src8 = reinterpret_cast<const uint8_t*>(src_);
    const int rr = tid >> 2, cc = (tid & 3) * 16;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      const int r = pass * 64 + rr;
      const int64_t srow = idx ? idx[r0 + r] : (r0 + r);
      const uint4 v = *reinterpret_cast<const uint4*>(src8 + srow * dim + c0 + cc);
      const float sc = __int_as_float((int)src_scales[srow * (dim >> 5) + ((c0 + cc) >> 5)] << 23);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint32_t h2;
        asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"((uint16_t)(w[i >> 1] >> (16 * (i & 1)))));
        s_in[r][cc + 2 * i] = __float2bfloat16_rn(__half2float(__ushort_as_half((unsigned short)(h2 & 0xFFFF))) * sc);
        s_in[r][cc + 2 * i + 1] = __float2bfloat16_rn(__half2float(__ushort_as_half((unsigned short)(h2 >> 16))) * sc);
      }
    }
  } else {
    // load: 8 threads x 16 bytes cover one 64-column row; 32 rows per pass
    const int rr = tid >> 3, cc = (tid & 7) * 8;
#pragma unroll
    for (int pass = 0; pass < 4; ++pass) {
      const int r = pass * 32 + rr;
      const int64_t srow = idx ? idx[r0 + r] : (r0 + r);
      const uint4 v = *reinterpret_cast<const uint4*>(src + srow * dim + c0 + cc);
      uint32_t* d = reinterpret_cast<uint32_t*>(&s_in[r][cc]);
      d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
    }
  }
  __syncthreads();

  const int c = tid & 63, g = tid >> 6;        // column, 32-row group
  float v[32];
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    v[i] = __bfloat162float(s_in[g * 32 + i][c]);
    amax = fmaxf(amax, fabsf(v[i]));
  }
  if (ISO) {  // block amax over the 32 columns of this warp
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffff, amax, d));
  }
  const int e = q_e8m0_of(amax);
  const float qs = q_scale_of(e);
  uint32_t w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) w[i] = q_pack4(v[4 * i] * qs, v[4 * i + 1] * qs, v[4 * i + 2] * qs, v[4 * i + 3] * qs);
  uint4* so = reinterpret_cast<uint4*>(&s_out[c][g * 32]);
  so[0] = make_uint4(w[0], w[1], w[2], w[3]);
  so[1] = make_uint4(w[4], w[5], w[6], w[7]);
  if (g == 0) s_sc[c] = 0;
  __syncthreads();
  atomicOr(&s_sc[c], (uint32_t)e << (8 * g));   // distinct bits per thread: order-free
  __syncthreads();

  // transposed bytes: 8 threads x 16 bytes cover one 128-byte row of s_out (skipped when the caller of the 32x32
  // form wants the row-major payload only)
  if (!ISO || q_t != nullptr) {
    const int cc = tid >> 3, seg = (tid & 7) * 16;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      const int col = pass * 32 + cc;
      *reinterpret_cast<uint4*>(q_t + (size_t)(c0 + col) * rows + r0 + seg) =
          *reinterpret_cast<const uint4*>(&s_out[col][seg]);
    }
  }
  // column scales: logical operand (dim, rows); one word = the 4 groups of this 128-row tile
  if (tid < CT_COLS) {
    const size_t col = c0 + tid;
    *reinterpret_cast<uint32_t*>(col_isa + isa_offset(col, (size_t)(r0 >> 5), (size_t)(rows >> 7))) = s_sc[tid];
  }
  if (ISO) {
    // non-transposed bytes: thread -> (row, 32-byte half of the 64 columns)
    const int r = tid >> 1, h = tid & 1;
    uint32_t o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int cc = h * 32 + i * 4;
      o[i] = (uint32_t)s_out[cc][r] | ((uint32_t)s_out[cc + 1][r] << 8) | ((uint32_t)s_out[cc + 2][r] << 16) |
             ((uint32_t)s_out[cc + 3][r] << 24);
    }
    uint4* dst = reinterpret_cast<uint4*>(q + (size_t)(r0 + r) * dim + c0 + h * 32);
    dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
    dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
    // row scales: logical operand (rows, dim); this tile holds groups c0/32 and c0/32+1 of 128 rows
    if (tid < CT_ROWS) {
      const size_t row = r0 + tid;
      const int gr = tid >> 5;
      const int k_tiles = dim >> 7;
      const int g0 = c0 >> 5;
      const uint8_t b0 = (uint8_t)(s_sc[0] >> (8 * gr));
      const uint8_t b1 = (uint8_t)(s_sc[32] >> (8 * gr));
      *reinterpret_cast<uint16_t*>(row_isa + isa_offset(row, g0, k_tiles)) = (uint16_t)b0 | ((uint16_t)b1 << 8);
    }
  }
}

// ------------------------------------------------------------------ weights, both orientations
// One [N, K] expert matrix per blockIdx.z, one 128x128 tile per block.  A tile of W is read ONCE and leaves twice:
// quantised 1x32 along K in place (q, `row_isa` = ISA scales of the stacked (E*N, K) operand) and 1x32 along N with
// the bytes transposed (q_t [E, K, N], `col_isa` = ISA scales of (K, N) per expert): the operands of the forward and of
// the backward GEMM.  Either direction can be switched off.
// Bound by HBM (2 bytes in, 2 x 33/32 out per weight), so the tile is as wide as the lines: every access of a warp covers
// whole 128-byte lines in both layouts (64-column tiles would leave half lines of q to two blocks).  A thread keeps
// eight 16-byte loads in flight; the row direction needs two shuffles per 32 values, the column direction reads the tile
// back from shared memory two columns at a time (bf16 pairs), so its maximum and its loads are half-rate per value.
// Measured at E=128, H=2048, I=768 (604 M weights, 2.45 GB, one launch per weight): 379 us = 6.5 TB/s, the rate of a copy; 402
// with maxima and scaling in f32 and three blocks an SM (E=8, H=3072, I=1536: 59.4 -> 55.3 for the larger weight; five blocks 1 %
// slower, six 20 %); one launch per expert for the transposed copy and a second read for the row copy took 3719 us (host-bound:
// 256 launches; their kernels alone 1345 us).
constexpr int QW_TILE = 128, QW_PITCH = QW_TILE + 8;      // bf16 elements; 272 bytes: 16-byte aligned rows

template <bool ROW, bool COL>
__global__ void __launch_bounds__(256, 4)
quant_weight_kernel(const __nv_bfloat16* __restrict__ w, int N, int K, uint8_t* __restrict__ q,
                    uint8_t* __restrict__ row_isa, uint8_t* __restrict__ q_t, uint8_t* __restrict__ col_isa) {
  __shared__ __align__(16) __nv_bfloat16 s_in[QW_TILE * QW_PITCH];
  __shared__ __align__(16) uint8_t s_rsc[512], s_csc[512];     // the tile's scales, already in ISA order
  uint8_t* s_out = reinterpret_cast<uint8_t*>(s_in);           // [128 columns][128 rows], once the tile has been consumed
  const int tid = threadIdx.x;
  const int k0 = blockIdx.x * QW_TILE, n0 = blockIdx.y * QW_TILE;
  const size_t base = (size_t)blockIdx.z * N * K;
  const int c8 = (tid & 15) * 8, r = tid >> 4;                 // 16 threads x 16 bytes = one 256-byte row of the tile
  uint4 v[8];
#pragma unroll
  for (int p = 0; p < 8; ++p)
    v[p] = __ldg(reinterpret_cast<const uint4*>(w + base + (size_t)(n0 + p * 16 + r) * K + k0 + c8));
#pragma unroll
  for (int p = 0; p < 8; ++p) {
    const int row = p * 16 + r;
    if (COL) *reinterpret_cast<uint4*>(s_in + row * QW_PITCH + c8) = v[p];
    if (ROW) {
      // from 0 on: a group of nothing but NaN has the maximum 0
      uint32_t m = q_max_abs_bf16x2(q_max_abs_bf16x2(q_max_abs_bf16x2(q_max_abs_bf16x2(0, v[p].x), v[p].y), v[p].z), v[p].w);
      m &= 0x7FFF7FFFu;
      m = q_max_bf16x2(m, __shfl_xor_sync(0xffffffff, m, 1));
      m = q_max_bf16x2(m, __shfl_xor_sync(0xffffffff, m, 2));
      m = q_max_bf16x2(m, __byte_perm(m, m, 0x1032));            // both halves: the maximum of the 32 values
      const uint32_t e = q_e8m0x2(m), qs = q_scalex2(e);
      *reinterpret_cast<uint2*>(q + base + (size_t)(n0 + row) * K + k0 + c8) =
          make_uint2(q_pack4_scaled(v[p].x, v[p].y, qs, qs), q_pack4_scaled(v[p].z, v[p].w, qs, qs));
      if ((tid & 3) == 0) s_rsc[(row & 31) * 16 + (row >> 5) * 4 + ((tid & 15) >> 2)] = (uint8_t)e;
    }
  }
  __syncthreads();
  // ISA tile of (row tile, K tile): 512 contiguous bytes
  if (ROW && tid < 32)
    reinterpret_cast<uint4*>(row_isa + (((size_t)blockIdx.z * N + n0) / 128 * (K / 128) + blockIdx.x) * 512)[tid] =
        reinterpret_cast<const uint4*>(s_rsc)[tid];
  if (COL) {
    const int c2 = tid & 63, g = tid >> 6;                     // columns 2*c2, 2*c2+1; rows [32 g, 32 g + 32)
    uint32_t x[32], am = 0;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      x[i] = *reinterpret_cast<const uint32_t*>(s_in + (g * 32 + i) * QW_PITCH + 2 * c2);
      am = q_max_abs_bf16x2(am, x[i]);
    }
    const uint32_t e2 = q_e8m0x2(am & 0x7FFF7FFFu), qs = q_scalex2(e2);
    __syncthreads();                                           // everyone has read the tile: its memory becomes s_out
    uint32_t o[2][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float2 f[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] = q_scaled(x[4 * i + j], qs);
      o[0][i] = q_pack4(f[0].x, f[1].x, f[2].x, f[3].x);
      o[1][i] = q_pack4(f[0].y, f[1].y, f[2].y, f[3].y);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int col = 2 * c2 + h;
      // 16-byte chunks of a column are stored at chunk ^ (column / 2 & 7): eight threads of neighbouring column pairs hit
      // eight different chunks, and so do the eight readers of one column below
#pragma unroll
      for (int i = 0; i < 2; ++i)
        *reinterpret_cast<uint4*>(s_out + col * 128 + (((2 * g + i) ^ (c2 & 7)) << 4)) =
            make_uint4(o[h][4 * i], o[h][4 * i + 1], o[h][4 * i + 2], o[h][4 * i + 3]);
      s_csc[(col & 31) * 16 + (col >> 5) * 4 + g] = (uint8_t)(e2 >> (16 * h));
    }
    __syncthreads();
    if (tid < 32)
      reinterpret_cast<uint4*>(col_isa + (((size_t)blockIdx.z * K + k0) / 128 * (N / 128) + blockIdx.y) * 512)[tid] =
          reinterpret_cast<const uint4*>(s_csc)[tid];
    const int cc = tid >> 3, ch = tid & 7;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int col = p * 32 + cc;
      *reinterpret_cast<uint4*>(q_t + base + (size_t)(k0 + col) * N + n0 + ch * 16) =
          *reinterpret_cast<const uint4*>(s_out + col * 128 + ((ch ^ ((col >> 1) & 7)) << 4));
    }
  }
}

// ------------------------------------------------------------------ columns of gathered rows
// Column-quantised operands of the weight gradients: row r of the operand is source row idx[r] (or r), one scale per column
// and 32 rows.  FP8: the source is e4m3 with raw row-wise 1x32 scales, dequantised (exact in bf16) first.
// A warp quantises 32 rows x 64 columns by itself: a lane holds eight consecutive rows of eight columns in registers and two
// shuffles complete a column's maximum.  There is no barrier: every form that had one (64 columns staged in bf16, the
// kernel above; 128 x 128 tiles whose bytes cross shared memory, with and without the next tile prefetched) took 86-96 us at
// T=8192, H=3072, K=E=8 (201 MB out), 65 us of it with neither loads nor stores: the warps waited for one another.

// Eight rows of this lane's eight columns, as bf16 pairs of adjacent columns
template <bool FP8>
__device__ __forceinline__ void qc_load(const void* __restrict__ src, const uint8_t* __restrict__ src_scales,
                                        const int (&srow)[8], int dim, int col, uint4 (&v)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const size_t at = (size_t)srow[i] * dim + col;
    if (FP8) {
      const uint2 b = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const uint8_t*>(src) + at));
      v[i] = make_uint4(b.x, b.y, __ldg(src_scales + (size_t)srow[i] * (dim >> 5) + (col >> 5)), 0);
    } else {
      v[i] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(src) + at));
    }
  }
}
// Dequantises (FP8); qs: the scales of the eight columns, as bf16 pairs; returns the scale bytes of columns 2 * sub and
// 2 * sub + 1 in the low bytes of its halves
template <bool FP8>
__device__ __forceinline__ uint32_t qc_scales(uint4 (&v)[8], int sub, uint32_t (&qs)[4]) {
  if (FP8) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float sc = __int_as_float((int)v[i].z << 23);
      const uint32_t w[2] = {v[i].x, v[i].y};
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t h2;
        asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"((uint16_t)(w[j >> 1] >> (16 * (j & 1)))));
        const float lo = __half2float(__ushort_as_half((unsigned short)(h2 & 0xFFFF))) * sc;
        const float hi = __half2float(__ushort_as_half((unsigned short)(h2 >> 16))) * sc;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o[j]) : "f"(hi), "f"(lo));
      }
      v[i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
  uint32_t e_pair = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) m = q_max_abs_bf16x2(m, j == 0 ? v[i].x : j == 1 ? v[i].y : j == 2 ? v[i].z : v[i].w);
    m &= 0x7FFF7FFFu;
    m = q_max_bf16x2(m, __shfl_xor_sync(0xffffffff, m, 8));
    m = q_max_bf16x2(m, __shfl_xor_sync(0xffffffff, m, 16));
    const uint32_t e2 = q_e8m0x2(m);
    qs[j] = q_scalex2(e2);
    if (sub == j) e_pair = e2;
  }
  return e_pair;
}

// What bounds both forms below is the latency of index -> row -> maximum -> store in each warp, not a throughput.  T=8192, H=3072,
// K=E=8, rows form, us: gathered reads alone 31, stores alone 37, loads and arithmetic without stores 49, everything 67.6.  Scales of
// two columns at a time, unpacking and scaling in one instruction a value and scale bytes gathered into whole ISA tiles took a
// quarter of the instructions out and gained 3 %: rows form 69.6 -> 67.6, transposed form 84 -> 82.

// q [rows, dim], read MN-major by the weight-gradient GEMM.  A block is four 32-row groups x 128 columns, column tiles
// fastest.  T=8192, H=3072, K=E=8: 86.0 -> 71.7 us; T=16384, H=2048, K=8, E=128 (285 MB out): 125 -> 102 us, against a warp
// per 32 x 256 slab, whose 255 registers left four warps an SM.
constexpr int QC_TILES = 4;      // row tiles of a block, one after the other
// Column tiles of a strip: a strip of all source rows is what the L2 has to hold while every expert's rows are gathered from it.
// With all columns in one strip a source of 67 MB was read from HBM once per expert.  All columns / 16 / 8 / 4 tiles, us:
// T=8192 H=4096 K=E=8 124 / 92 / 88 / 87, T=8192 H=3072 77 / 71 / 71 / 69, T=16384 H=2048 K=8 E=128, skewed, 109 / 108 / 96 / 96,
// T=4096 H=3072 E=32 41 / 42 / 41 / 42.
constexpr int QC_STRIP = 8;

__global__ void __launch_bounds__(256, 4)
quant_cols_rows_kernel(const void* __restrict__ src, const int* __restrict__ idx, const int* __restrict__ valid_rows,
                       int64_t rows, int dim, uint8_t* __restrict__ q, uint8_t* __restrict__ col_isa) {
  __shared__ __align__(16) uint8_t s_isa[QC_TILES * 512];             // scales of the block's tiles, in ISA order
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane >> 3;
  // strips of QC_STRIP column tiles, one after the other; within a strip column tiles fastest, then row tiles
  const int groups = ((int)(rows >> 7) + QC_TILES - 1) / QC_TILES, strip = blockIdx.x / (QC_STRIP * groups);
  const int width = min(QC_STRIP, (dim >> 7) - strip * QC_STRIP), in_strip = blockIdx.x - strip * QC_STRIP * groups;
  const int ct = strip * QC_STRIP + in_strip % width, rt0 = in_strip / width * QC_TILES;
  const int grp = warp >> 1;                                          // 32-row group of the 128-row tile
  const int col = ct * 128 + (warp & 1) * 64 + (lane & 7) * 8;        // this lane's columns [col, col + 8)
  const int row0 = grp * 32 + sub * 8;                                // and rows of a tile [row0, row0 + 8)
  const int rt_end = min(rt0 + QC_TILES, (int)(rows >> 7));
  int srow[8];                                                        // their source rows, one tile ahead
#pragma unroll
  for (int i = 0; i < 8; ++i) srow[i] = idx ? idx[(int64_t)rt0 * 128 + row0 + i] : rt0 * 128 + row0 + i;
  const int64_t n_valid = valid_rows != nullptr ? min((int64_t)*valid_rows, rows) : rows;
  for (int rt = rt0; rt < rt_end; ++rt) {
    const int64_t r0 = (int64_t)rt * 128;
    if (r0 + 32 * grp >= n_valid) break;                              // over-allocated tail: no GEMM reads it
    uint4 v[8];
    qc_load<false>(src, nullptr, srow, dim, col, v);
    if (rt + 1 < rt_end) {
#pragma unroll
      for (int i = 0; i < 8; ++i) srow[i] = idx ? idx[r0 + 128 + row0 + i] : (int)r0 + 128 + row0 + i;
    }
    uint32_t qs[4];
    const uint32_t e_pair = qc_scales<false>(v, sub, qs);
    uint8_t* dst = q + (size_t)(r0 + row0) * dim + col;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      *reinterpret_cast<uint2*>(dst + (size_t)i * dim) =
          make_uint2(q_pack4_scaled(v[i].x, v[i].y, qs[0], qs[1]), q_pack4_scaled(v[i].z, v[i].w, qs[2], qs[3]));
    }
    const int cc = (col + 2 * sub) & 127;                             // ISA tile of (column tile, row tile)
    uint8_t* isa = s_isa + (rt - rt0) * 512 + (cc >> 5) * 4 + grp;
    isa[(cc & 31) * 16] = (uint8_t)e_pair;
    isa[((cc & 31) + 1) * 16] = (uint8_t)(e_pair >> 16);
  }
  __syncthreads();
  const int rt = rt0 + warp;
  const int64_t left = n_valid - (int64_t)rt * 128;                   // rows of the warp's tile, if it has any
  if (warp >= QC_TILES || rt >= rt_end || left <= 0) return;
  const uint8_t* from = s_isa + threadIdx.x * 16;
  uint8_t* to = col_isa + ((size_t)ct * (size_t)(rows >> 7) + rt) * 512 + lane * 16;
  if (left > 96 && ((uintptr_t)col_isa & 15) == 0) {
    *reinterpret_cast<uint4*>(to) = *reinterpret_cast<const uint4*>(from);
  } else {       // a tile that is not full (byte g of a word is row group g's), or scales that start anywhere: byte by byte
#pragma unroll 1
    for (int i = 0; i < 16; ++i)
      if ((i & 3) * 32 < left) to[i] = from[i];
  }
}

// q [dim, rows]: the reduction dimension contiguous.  A warp walks the four 32-row groups of a 128-row tile, gathers the bytes
// of its 64 columns in 8 KB of shared memory of its own and then stores them as whole 128-byte lines (32-byte pieces
// straight from the registers: 96 us).  Same sizes as above: 96 -> 85 and 137 -> 117 us.
constexpr int QT_WARPS = 4;

template <bool FP8>
__global__ void __launch_bounds__(32 * QT_WARPS, 6)
quant_cols_t_kernel(const void* __restrict__ src, const uint8_t* __restrict__ src_scales, const int* __restrict__ idx,
                    const int* __restrict__ valid_rows, int64_t rows, int dim, uint8_t* __restrict__ q_t,
                    uint8_t* __restrict__ col_isa) {
  __shared__ __align__(16) uint8_t s_bytes[QT_WARPS][64 * 128];       // [column][row], 8-byte chunks swizzled
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, l8 = lane & 7, sub = lane >> 3;
  const int64_t r0 = (int64_t)blockIdx.x * 128;
  const int c0 = (blockIdx.y * QT_WARPS + warp) * 64;                 // this warp's columns [c0, c0 + 64)
  if (c0 >= dim) return;
  const int col = c0 + l8 * 8;
  int srow[8];                                                        // source rows of a group, one group ahead
#pragma unroll
  for (int i = 0; i < 8; ++i) srow[i] = idx ? idx[r0 + sub * 8 + i] : (int)r0 + sub * 8 + i;
  if (valid_rows != nullptr && r0 >= *valid_rows) return;             // over-allocated tail: no GEMM reads it
  uint8_t* s = s_bytes[warp];
  const int swz = (l8 & 3) << 2;                                      // chunk c of a column lies at slot c ^ swz
  uint32_t sc0 = 0, sc1 = 0;                                          // four scale bytes of columns 2 * sub, 2 * sub + 1
#pragma unroll 1
  for (int g = 0; g < 4; ++g) {
    uint4 v[8];
    qc_load<FP8>(src, src_scales, srow, dim, col, v);
    if (g < 3) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int64_t r = r0 + (g + 1) * 32 + sub * 8 + i;
        srow[i] = idx ? idx[r] : (int)r;
      }
    }
    uint32_t qs[4];
    const uint32_t e_pair = qc_scales<FP8>(v, sub, qs);
    sc0 |= (e_pair & 0xFF) << (8 * g);
    sc1 |= (e_pair >> 16) << (8 * g);
#pragma unroll
    for (int j = 0; j < 4; ++j) {                                     // columns 2j and 2j + 1 of the lane
      float2 f[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = q_scaled(j == 0 ? v[i].x : j == 1 ? v[i].y : j == 2 ? v[i].z : v[i].w, qs[j]);
      uint8_t* d = s + (l8 * 8 + 2 * j) * 128 + (((g * 4 + sub) ^ swz) << 3);
      *reinterpret_cast<uint2*>(d) = make_uint2(q_pack4(f[0].x, f[1].x, f[2].x, f[3].x), q_pack4(f[4].x, f[5].x, f[6].x, f[7].x));
      *reinterpret_cast<uint2*>(d + 128) =
          make_uint2(q_pack4(f[0].y, f[1].y, f[2].y, f[3].y), q_pack4(f[4].y, f[5].y, f[6].y, f[7].y));
    }
  }
  __syncwarp();
#pragma unroll
  for (int p = 0; p < 16; ++p) {
    const int c = p * 4 + sub;
    const uint4 o = *reinterpret_cast<const uint4*>(s + c * 128 + ((l8 ^ (((c >> 3) & 3) << 1)) << 4));
    *reinterpret_cast<uint4*>(q_t + (size_t)(c0 + c) * rows + r0 + l8 * 16) = o;
  }
  const int cc = (col + 2 * sub) & 127;                               // ISA tile of (column tile, row tile)
  uint8_t* isa = col_isa + ((size_t)(col >> 7) * (size_t)(rows >> 7) + blockIdx.x) * 512 + (cc >> 5) * 4;
  *reinterpret_cast<uint32_t*>(isa + (cc & 31) * 16) = sc0;
  *reinterpret_cast<uint32_t*>(isa + ((cc & 31) + 1) * 16) = sc1;
}

}  // namespace smoe

using namespace smoe;

// ------------------------------------------------- gathered rows, both directions
// One warp owns 32 consecutive expert-sorted rows x 256 columns (a lane: 8 columns of every row, 32 x 16-byte
// loads in flight).  Column scales (one per column and 32 rows) need no communication at all, row scales
// (one per row and 32 columns) two shuffles per row.  Both payloads leave row-major: the column-scaled one is a
// weight-gradient operand read MN-major by the tensor core, so no transposed copy is written.
__global__ void __launch_bounds__(128)
quant_dual_kernel(const uint4* __restrict__ x, const int* __restrict__ idx, const int* __restrict__ valid_rows,
                  int64_t rows, int K, uint2* __restrict__ q_row, uint8_t* __restrict__ row_isa,
                  uint2* __restrict__ q_col, uint8_t* __restrict__ col_isa) {
  const int lane = threadIdx.x & 31;
  const int64_t task = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  const int cbs = K >> 8;
  const int64_t rg = task / cbs;
  const int cb = (int)(task - rg * cbs);
  const int64_t r0 = rg * 32;
  int64_t limit = rows;
  if (valid_rows) limit = min(limit, (int64_t)*valid_rows);
  if (r0 >= limit) return;
  const int col0 = cb * 256 + lane * 8;
  const int64_t my_row = idx ? (int64_t)idx[r0 + lane] : r0 + lane;
  uint4 v[32];
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    const int64_t srow = __shfl_sync(0xffffffff, my_row, r);
    v[r] = x[(srow * K + col0) >> 3];
  }
  float cam[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) cam[j] = 0.f;
  const size_t row_kt = (size_t)((K + 127) >> 7);
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    float f[8];
    bf16x8_to_f32(v[r], f);
    float ram = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      cam[j] = fmaxf(cam[j], fabsf(f[j]));
      ram = fmaxf(ram, fabsf(f[j]));
    }
    ram = fmaxf(ram, __shfl_xor_sync(0xffffffff, ram, 1));
    ram = fmaxf(ram, __shfl_xor_sync(0xffffffff, ram, 2));
    const int e = q_e8m0_of(ram);
    const float qs = q_scale_of(e);
    uint2 o;
    o.x = q_pack4(f[0] * qs, f[1] * qs, f[2] * qs, f[3] * qs);
    o.y = q_pack4(f[4] * qs, f[5] * qs, f[6] * qs, f[7] * qs);
    q_row[((r0 + r) * K + col0) >> 3] = o;
    if ((lane & 3) == 0) row_isa[isa_offset((size_t)(r0 + r), (size_t)(col0 >> 5), row_kt)] = (uint8_t)e;
  }
  float qs[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int e = q_e8m0_of(cam[j]);
    qs[j] = q_scale_of(e);
    col_isa[isa_offset((size_t)(col0 + j), (size_t)rg, (size_t)(rows >> 7))] = (uint8_t)e;
  }
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    float f[8];
    bf16x8_to_f32(v[r], f);
    uint2 o;
    o.x = q_pack4(f[0] * qs[0], f[1] * qs[1], f[2] * qs[2], f[3] * qs[3]);
    o.y = q_pack4(f[4] * qs[4], f[5] * qs[5], f[6] * qs[6], f[7] * qs[7]);
    q_col[((r0 + r) * K + col0) >> 3] = o;
  }
}


// What every column kernel accesses 16 bytes at a time, and its scales by the word
static bool cols_aligned(const void* src, const void* q, const void* isa) {
  return (((uintptr_t)src | (uintptr_t)q) & 15) == 0 && ((uintptr_t)isa & 3) == 0;
}

extern "C" {

int smoe_quant_rows(const void* x_bf16, int64_t M, int64_t K, void* q, void* raw_scales, void* isa_scales,
                    void* stream) {
  if (M < 0 || K <= 0 || K % 32) return SMOE_ERR_SHAPE;
  if (isa_scales && K % 128) return SMOE_ERR_SHAPE;
  if (K % 8 || ((uintptr_t)x_bf16 & 15) || ((uintptr_t)q & 7)) return SMOE_ERR_ALIGN;
  if (M == 0) return SMOE_OK;
  int64_t blocks = (M + 7) / 8;
  if (blocks > 148 * 16) blocks = 148 * 16;
  quant_rows_kernel<<<(int)blocks, 256, 0, (cudaStream_t)stream>>>((const uint4*)x_bf16, M, (int)K, (uint2*)q,
                                                                   (uint8_t*)raw_scales, (uint8_t*)isa_scales, nullptr,
                                                                   nullptr);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_quant_rows_scatter(const void* x_bf16, int64_t T, int64_t K, const int32_t* naept, const int32_t* s_rev,
                            const int32_t* s_scatter_idx, const int32_t* valid_rows, int64_t rows, void* q,
                            void* isa_scales, void* stream) {
  if (T < 0 || rows < 0 || K <= 0 || K % 128 || K > 16384) return SMOE_ERR_SHAPE;
  if (rows == 0) return SMOE_OK;      // nothing routed: not an error, and the (empty) buffers may be null
  if (!naept || !s_rev || !isa_scales) return SMOE_ERR_ARG;
  if (((uintptr_t)x_bf16 & 15) || ((uintptr_t)q & 15)) return SMOE_ERR_ALIGN;
  const int row_bytes = (int)((K + 4 * (K / 128) + 15) & ~(int64_t)15);
  int warps = row_bytes * 8 <= 48 * 1024 ? 8 : (row_bytes * 4 <= 48 * 1024 ? 4 : 2);
  while (warps > 1 && T < 296 * warps) warps /= 2;  // few tokens: two blocks an SM before eight warps a block
  const int token_blocks = (int)((T + warps - 1) / warps);
  int pad_blocks = (int)((rows + 8 * warps - 1) / (8 * warps));
  if (pad_blocks > 296 * 8 / warps) pad_blocks = 296 * 8 / warps;
  if (!s_scatter_idx) pad_blocks = 0;               // pad rows stay as they are
  if (token_blocks + pad_blocks == 0) return SMOE_OK;
  quant_rows_scatter_kernel<<<token_blocks + pad_blocks, warps * 32, (size_t)warps * row_bytes,
                              (cudaStream_t)stream>>>((const uint4*)x_bf16, T, (int)K, naept, s_rev, s_scatter_idx,
                                                      valid_rows, rows, (uint4*)q, (uint8_t*)isa_scales, token_blocks);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_quant_rows_gather(const void* x_bf16, const int32_t* idx, const int32_t* valid_rows, int64_t rows, int64_t K,
                           void* q, void* isa_scales, void* stream) {
  if (rows < 0 || K <= 0 || K % 128) return SMOE_ERR_SHAPE;
  if (rows == 0) return SMOE_OK;      // nothing routed: not an error, and the (empty) buffers may be null
  if (!idx || !isa_scales) return SMOE_ERR_ARG;
  if (((uintptr_t)x_bf16 & 15) || ((uintptr_t)q & 7)) return SMOE_ERR_ALIGN;
  int64_t blocks = (rows + 7) / 8;
  if (blocks > 148 * 16) blocks = 148 * 16;
  quant_rows_kernel<<<(int)blocks, 256, 0, (cudaStream_t)stream>>>((const uint4*)x_bf16, rows, (int)K, (uint2*)q,
                                                                   nullptr, (uint8_t*)isa_scales, idx, valid_rows);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_gather_scales_isa(const void* raw_scales, const int32_t* idx, int64_t rows, int64_t cols, void* isa_scales,
                           void* stream) {
  if (rows < 0 || cols <= 0 || cols % 32) return SMOE_ERR_SHAPE;
  if (rows == 0) return SMOE_OK;
  const int groups = (int)(cols / 32), k_tiles = (int)((cols + 127) / 128);
  const int64_t n = rows * k_tiles;
  gather_scales_isa_kernel<<<(int)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      (const uint8_t*)raw_scales, idx, rows, groups, k_tiles, (uint8_t*)isa_scales);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_gather_rows_fp8(const void* q, const void* raw_scales, const int32_t* idx, const int32_t* valid_rows,
                         int64_t rows, int64_t K, void* q_out, void* isa_out, void* stream) {
  if (rows < 0 || K <= 0 || K % 128) return SMOE_ERR_SHAPE;
  if (rows == 0) return SMOE_OK;      // nothing routed: not an error, and the (empty) buffers may be null
  if (((uintptr_t)q & 15) || ((uintptr_t)q_out & 15) || ((uintptr_t)raw_scales & 3)) return SMOE_ERR_ALIGN;
  const int threads = K / 16 >= 256 ? 256 : (int)((K / 16 + 31) / 32 * 32);
  gather_rows_kernel<<<(unsigned)rows, threads, 0, (cudaStream_t)stream>>>(
      (const uint4*)q, (const uint8_t*)raw_scales, idx, valid_rows, (int)K, (uint4*)q_out, (uint8_t*)isa_out);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_quant_cols_t(const void* src_bf16, const int32_t* idx, const int32_t* valid_rows, int64_t rows, int64_t dim,
                      void* q_t, void* isa, void* stream) {
  if (rows < 0 || rows % 128 || dim <= 0 || dim % 64) return SMOE_ERR_SHAPE;
  if (rows == 0) return SMOE_OK;
  if (!cols_aligned(src_bf16, q_t, isa)) return SMOE_ERR_ALIGN;
  // whole scale tiles (every dim a GEMM takes): the form without barriers; half a tile more: 64 columns staged (dim = 3072:
  // 85 against 96 us)
  if (dim % 128 == 0) {
    quant_cols_t_kernel<false><<<dim3((unsigned)(rows / 128), (unsigned)((dim + 255) / 256)), 32 * QT_WARPS, 0,
                                 (cudaStream_t)stream>>>(src_bf16, nullptr, idx, valid_rows, rows, (int)dim, (uint8_t*)q_t,
                                                         (uint8_t*)isa);
    return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
  }
  dim3 grid((unsigned)(rows / CT_ROWS), (unsigned)(dim / CT_COLS));
  quant_cols_kernel<false, false><<<grid, 256, 0, (cudaStream_t)stream>>>(
      src_bf16, nullptr, idx, rows, (int)dim, (uint8_t*)q_t, (uint8_t*)isa, nullptr, nullptr, valid_rows);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_requant_cols_t(const void* src_fp8, const void* src_scales, const int32_t* idx, const int32_t* valid_rows,
                        int64_t rows, int64_t dim, void* q_t, void* isa, void* stream) {
  if (rows < 0 || rows % 128 || dim <= 0 || dim % 64) return SMOE_ERR_SHAPE;
  if (rows == 0) return SMOE_OK;      // nothing routed: not an error, and the (empty) buffers may be null
  if (!src_scales) return SMOE_ERR_ARG;
  if (!cols_aligned(src_fp8, q_t, isa)) return SMOE_ERR_ALIGN;
  if (dim % 128 == 0) {
    quant_cols_t_kernel<true><<<dim3((unsigned)(rows / 128), (unsigned)((dim + 255) / 256)), 32 * QT_WARPS, 0,
                                (cudaStream_t)stream>>>(src_fp8, (const uint8_t*)src_scales, idx, valid_rows, rows, (int)dim,
                                                        (uint8_t*)q_t, (uint8_t*)isa);
    return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
  }
  dim3 grid((unsigned)(rows / CT_ROWS), (unsigned)(dim / CT_COLS));
  quant_cols_kernel<false, true><<<grid, 256, 0, (cudaStream_t)stream>>>(
      src_fp8, (const uint8_t*)src_scales, idx, rows, (int)dim, (uint8_t*)q_t, (uint8_t*)isa, nullptr, nullptr,
      valid_rows);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_quant_iso32(const void* x_bf16, int64_t rows, int64_t cols, void* q, void* row_isa, void* q_t, void* col_isa,
                     void* stream) {
  if (rows < 0 || rows % 128 || cols <= 0 || cols % 128) return SMOE_ERR_SHAPE;
  if (rows == 0) return SMOE_OK;
  if (!cols_aligned(x_bf16, q, col_isa) || ((uintptr_t)q_t & 15) || ((uintptr_t)row_isa & 1)) return SMOE_ERR_ALIGN;
  dim3 grid((unsigned)(rows / CT_ROWS), (unsigned)(cols / CT_COLS));
  quant_cols_kernel<true, false><<<grid, 256, 0, (cudaStream_t)stream>>>(x_bf16, nullptr, nullptr, rows, (int)cols,
                                                                         (uint8_t*)q_t, (uint8_t*)col_isa, (uint8_t*)q,
                                                                         (uint8_t*)row_isa, nullptr);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_quant_weight(const void* w_bf16, int64_t E, int64_t N, int64_t K, void* q, void* row_isa, void* q_t,
                      void* col_isa, void* stream) {
  if (E < 0 || N < 0 || K < 0 || N % 128 || K % 128 || E > 65535 || N / 128 > 65535) return SMOE_ERR_SHAPE;
  if (E == 0 || N == 0 || K == 0) return SMOE_OK;
  if (!w_bf16 || (q == nullptr) != (row_isa == nullptr) || (q_t == nullptr) != (col_isa == nullptr) || (!q && !q_t))
    return SMOE_ERR_ARG;
  if (((uintptr_t)w_bf16 | (uintptr_t)q | (uintptr_t)row_isa | (uintptr_t)q_t | (uintptr_t)col_isa) & 15)
    return SMOE_ERR_ALIGN;
  const dim3 grid((unsigned)(K / 128), (unsigned)(N / 128), (unsigned)E);
  auto kern = q == nullptr ? quant_weight_kernel<false, true>
                           : (q_t == nullptr ? quant_weight_kernel<true, false> : quant_weight_kernel<true, true>);
  kern<<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)w_bf16, (int)N, (int)K, (uint8_t*)q,
                                               (uint8_t*)row_isa, (uint8_t*)q_t, (uint8_t*)col_isa);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_transpose_u8(const void* src, int64_t batch, int64_t rows, int64_t cols, void* dst, void* stream) {
  if (batch < 0 || rows < 0 || cols < 0 || rows % 64 || cols % 64 || batch > 65535) return SMOE_ERR_SHAPE;
  if (batch == 0 || rows == 0 || cols == 0) return SMOE_OK;
  if (!src || !dst) return SMOE_ERR_ARG;
  if (((uintptr_t)src & 15) || ((uintptr_t)dst & 15)) return SMOE_ERR_ALIGN;
  dim3 grid((unsigned)(cols / 64), (unsigned)(rows / 64), (unsigned)batch);
  if (grid.y > 65535) return SMOE_ERR_SHAPE;
  transpose_u8_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const uint8_t*)src, (uint8_t*)dst, (int)rows, (int)cols);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_quant_dual_gather(const void* x_bf16, const int32_t* idx, const int32_t* valid_rows, int64_t rows, int64_t K,
                           void* q_row, void* row_isa, void* q_col, void* col_isa, void* stream) {
  if (rows < 0 || rows % 128 || K <= 0 || K % 256) return SMOE_ERR_SHAPE;
  if (rows == 0) return SMOE_OK;      // nothing routed: not an error, and the (empty) buffers may be null
  if (!q_col || !col_isa || ((q_row == nullptr) != (row_isa == nullptr))) return SMOE_ERR_ARG;
  if (((uintptr_t)x_bf16 & 15) || ((uintptr_t)q_col & 7) || ((uintptr_t)q_row & 7)) return SMOE_ERR_ALIGN;
  if (q_row) {
    const int64_t tasks = (rows / 32) * (K / 256);
    quant_dual_kernel<<<(unsigned)((tasks + 3) / 4), 128, 0, (cudaStream_t)stream>>>(
        (const uint4*)x_bf16, idx, valid_rows, rows, (int)K, (uint2*)q_row, (uint8_t*)row_isa, (uint2*)q_col,
        (uint8_t*)col_isa);
  } else {
    const int64_t blocks = (K / 128) * ((rows / 128 + QC_TILES - 1) / QC_TILES);
    quant_cols_rows_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(x_bf16, idx, valid_rows, rows, (int)K,
                                                                               (uint8_t*)q_col, (uint8_t*)col_isa);
  }
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

int smoe_scatter_rows_fp8(const void* q, const void* raw_scales, int64_t T, int64_t K, const int32_t* naept,
                          const int32_t* s_rev, const int32_t* s_scatter_idx, const int32_t* valid_rows, int64_t rows,
                          void* q_out, void* isa_out, void* stream) {
  if (T < 0 || rows < 0 || K <= 0 || K % 128) return SMOE_ERR_SHAPE;
  if (rows == 0) return SMOE_OK;      // nothing routed: not an error, and the (empty) buffers may be null
  if (((uintptr_t)q & 15) || ((uintptr_t)q_out & 15) || ((uintptr_t)raw_scales & 3)) return SMOE_ERR_ALIGN;
  if (isa_out != nullptr && raw_scales == nullptr) return SMOE_ERR_ARG;
  const int token_blocks = (int)((T + 7) / 8);
  const int pad_blocks = 148;
  scatter_rows_fp8_kernel<<<(unsigned)(token_blocks + pad_blocks), 256, 0, (cudaStream_t)stream>>>(
      (const uint4*)q, (const uint8_t*)raw_scales, T, (int)K, naept, s_rev, s_scatter_idx, valid_rows, rows,
      (uint4*)q_out, (uint8_t*)isa_out, token_blocks);
  return cudaGetLastError() == cudaSuccess ? SMOE_OK : SMOE_ERR_LAUNCH;
}

}  // extern "C"
