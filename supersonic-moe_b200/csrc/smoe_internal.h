/* Calls between the library's own files and symbols it exports for its own tests and timing experiments.  None is part of the
 * product ABI (include/smoe_b200.h); the exported ones are process-global, unsynchronised, and able to switch stores off. */
#ifndef SMOE_INTERNAL_H_
#define SMOE_INTERNAL_H_

#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

/* bits 0..15: force the GEMM column tile (128, 192, 256 or 384; 0 = automatic); bit 16: epilogues skip their stores;
 * bit 17: force the single-CTA kernel; bit 18: the fused dgated epilogue is skipped whole;
 * timing experiments of the two-CTA main loops: bit 19: no operand loads after the first ring pass; bit 20: the
 * accumulators are handed back undrained (and nothing is stored); bit 21: no scale copies into TMEM;
 * bits 24..25: ring stages left unused; bits 26..30: value + 1 of the L2 prefetch distance (256-wide kernels) or of
 * the head / tail length (256 x 384 kernel), 0 = the kernel's default; bit 31: indexed A rows through TMA gather4
 * instead of the cp.async load warps.  0 restores the defaults. */
int smoe_internal_gemm_knobs(int bits);

/* A device buffer of 8 x 256 int64 that the MMA issuer of CTA pair 0 of the 256 x 384 kernel fills, per tile, with
 * SM-clock stamps and the cycles it spent in each kind of wait (tile start, after the accumulator waits, cycles
 * waiting for operands / scales / the second accumulator, tile end, wait for the first operands); null switches the
 * stamping off (the default). */
int smoe_internal_gemm_trace(void* device_buffer);

#ifdef __cplusplus
}

namespace smoe {
// smoe_gemm_gated_few and smoe_gemm_varlen_m_few as a layer calls them.  `early`: the kernel may begin while the one before it in
// the stream ends, and reads efo, counts and weights before that one's writes are visible: only for a caller that knows the
// kernel before, that it writes none of the three, and that they were complete when it began.
int gemm_gated_few(const void* x_sorted_fp8, const void* a_sf, const void* w1_fp8, const void* w1_sf, const int* efo,
                   const int* counts, void* y1_fp8, void* y1_sf, int64_t rows, int64_t N, int64_t K, int64_t E, int* status,
                   bool early, void* stream);
int gemm_varlen_m_few(const void* a_fp8, const void* a_sf, const void* b_fp8, const void* b_sf, const int* efo,
                      const int* counts, void* c_bf16, int64_t rows, int64_t N, int64_t K, int64_t E, int* status, bool early,
                      void* stream);
}  // namespace smoe
#endif
#endif /* SMOE_INTERNAL_H_ */
