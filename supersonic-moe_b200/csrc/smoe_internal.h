/* Calls between the library's own files, and three symbols it exports for its own tests.  None is part of the product ABI
 * (include/smoe_b200.h); the knobs are process-global and unsynchronised. */
#ifndef SMOE_INTERNAL_H_
#define SMOE_INTERNAL_H_

#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

/* Which of several kernels for the same result runs.  Bits 0..15: force the GEMM column tile (128, 192, 256 or 384; 0 =
 * automatic); bit 17: force the single-CTA kernel; bit 31: indexed A rows through TMA gather4 instead of the cp.async load warps.
 * 0 restores the defaults. */
int smoe_internal_gemm_knobs(int bits);

/* Column tile of smoe_gemm_varlen_m on these sizes (rows: as allocated); 0: the single-CTA kernel. */
int smoe_internal_plain_tile(int64_t rows, int64_t N, int64_t K, int64_t E);

/* 1 where a weight-gradient launch of the 384-column kernel loads the old gradient ahead of its sums: k_tiles of all experts, busy
 * experts of E, output tiles on so many CTA pairs. */
int smoe_internal_reduce_loads(int k_tiles, int busy, int E, int tiles, int pairs);

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
