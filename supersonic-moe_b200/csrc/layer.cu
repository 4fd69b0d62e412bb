// A whole small layer per call: the launches of a forward or a backward pass of the SwiGLU layer, back to back from one
// host function, with every intermediate in a caller-supplied arena.
//
// What bounds a small layer is the host.  At T=256, H=256, I=128, E=8, K=2 the kernels of a forward + backward take 102 us
// and the Python that allocated some 45 tensors and made 20 foreign calls one by one took 870 us; a decode step of 64 tokens
// over 128 experts (196 us of kernels) took 419 us.  Nothing is computed differently here: the functions below call the
// entry points of the library in the order the layer always did, on the same operands.
#include <cuda_runtime.h>
#include <stdint.h>

#include "smoe_b200.h"
#include "smoe_internal.h"

namespace smoe {

// Bump allocator over an arena; a null base only measures.
struct Arena {
  uint8_t* base;
  size_t used = 0;
  explicit Arena(void* p) : base(static_cast<uint8_t*>(p)) {}
  template <typename T = uint8_t>
  T* take(int64_t count) {
    T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
    used += ((size_t)count * sizeof(T) + 255) & ~(size_t)255;
    return p;
  }
};

static int64_t isa_bytes(int64_t rows, int64_t cols) { return (rows + 127) / 128 * ((cols + 127) / 128) * 512; }

// what a forward leaves for its backward (metadata; z where a backward follows)
struct Saved {
  int32_t *efo, *x_gather, *s_scatter, *s_rev, *naept, *src_idx;
  float* scores;
  uint8_t *z, *z_sc;
  size_t bytes;
  Saved(const smoe_layer_args& a, void* arena) {
    Arena m(arena);
    efo = m.take<int32_t>(a.E + 1);
    x_gather = m.take<int32_t>(a.TKp_alloc);
    s_scatter = m.take<int32_t>(a.TKp_alloc);
    s_rev = m.take<int32_t>(a.TK_alloc);
    naept = m.take<int32_t>(a.T + 1);
    src_idx = m.take<int32_t>(a.TK_alloc);
    scores = m.take<float>(a.TKp_alloc);
    z = z_sc = nullptr;
    if (a.keep_z) {
      z = m.take(a.TKp_alloc * 2 * a.I);
      z_sc = m.take(a.TKp_alloc * (2 * a.I / 32));
    }
    bytes = m.used;
  }
};

struct FwdScratch {
  uint8_t *ws, *xg, *xg_sf, *y1, *y1_sf, *y2;
  size_t bytes;
  FwdScratch(const smoe_layer_args& a, void* arena) {
    Arena m(arena);
    ws = m.take(smoe_topk_metadata_workspace(a.T, a.E));
    xg = m.take(a.TKp_alloc * a.H);
    xg_sf = m.take(isa_bytes(a.TKp_alloc, a.H));
    y1 = m.take(a.TKp_alloc * a.I);
    y1_sf = m.take(isa_bytes(a.TKp_alloc, a.I));
    y2 = m.take(a.TKp_alloc * a.H * 2);
    bytes = m.used;
  }
};

// Shapes of which a weight gradient may read an operand as it lies ([rows, dim]), and those of the 256 x 384 kernel
static bool mn_ok(int64_t E, int64_t M, int64_t N) { return E <= 256 && M % 256 == 0 && N % 256 == 0; }
static bool wide_ok(int64_t E, int64_t M, int64_t N) { return E <= 256 && M % 256 == 0 && N % 384 == 0; }

struct BwdScratch {
  bool fused;                       // GemmDGated emits the e4m3 operands itself (256-multiples of I and H)
  int64_t parts;
  float *s, *dsp;
  uint8_t *dg, *dg_sf;              // dout, expert-sorted rows
  uint8_t *dc, *dc_sf;              // dout, column-quantised; null without dw2
  uint8_t *dz, *dz_rsf, *dz_csf, *dz_t;
  uint8_t *y1s, *y1s_sf;            // column-quantised: [rows, I], or [I, rows] when not fused
  uint8_t *dz_bf16, *y1s_bf16;
  uint8_t* dx_exp;                  // null without dx
  uint8_t *xc, *xc_sf;              // x, column-quantised; null without dw1
  size_t bytes;
  BwdScratch(const smoe_layer_args& a, void* arena) {
    Arena m(arena);
    const int64_t R = a.TKp_alloc, H = a.H, I = a.I;
    fused = mn_ok(a.E, I, H);
    parts = fused ? smoe_gemm_dgated_fused_partials(I) : smoe_gemm_dgated_partials(I);
    s = fused ? nullptr : m.take<float>(R);       // scores of expert-sorted rows (the fused kernel looks them up itself)
    // room for the narrowest column tile, 128 columns in two groups, whatever tile is in use: the size follows from the arguments
    // alone, and may be remembered by them
    dsp = m.take<float>(2 * ((I + 127) / 128) * R);
    dg = m.take(R * H);
    dg_sf = m.take(isa_bytes(R, H));
    dc = dc_sf = dx_exp = xc = xc_sf = nullptr;
    if (a.dw2_mode != SMOE_DW_NONE) {
      dc = m.take(R * H);
      dc_sf = m.take(isa_bytes(H, R));
    }
    dz = m.take(R * 2 * I);
    dz_rsf = m.take(isa_bytes(R, 2 * I));
    dz_csf = m.take(isa_bytes(2 * I, R));
    y1s = m.take(R * I);
    y1s_sf = m.take(isa_bytes(I, R));
    dz_t = dz_bf16 = y1s_bf16 = nullptr;
    if (!fused) {
      dz_t = m.take(R * 2 * I);
      dz_bf16 = m.take(R * 2 * I * 2);
      y1s_bf16 = m.take(R * I * 2);
    }
    if (a.out) dx_exp = m.take(R * H * 2);
    if (a.dw1_mode != SMOE_DW_NONE) {
      xc = m.take(R * H);
      xc_sf = m.take(isa_bytes(H, R));
    }
    bytes = m.used;
  }
};

static int check_args(const smoe_layer_args* a) {
  if (!a || a->T < 0 || a->H <= 0 || a->I <= 0 || a->E <= 0 || a->K <= 0 || a->H % 128 || a->I % 128 || a->E > 256 ||
      a->TKp_alloc < 0 || a->TKp_alloc % 128 || a->TK_alloc < 0)
    return SMOE_ERR_SHAPE;
  return SMOE_OK;
}

// the host word to post to, or null while a graph is captured
static int host_word(const smoe_layer_args& a, void* stream, int32_t** word) {
  *word = nullptr;
  if (!a.host_word) return SMOE_OK;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing((cudaStream_t)stream, &cap) != cudaSuccess) return SMOE_ERR_LAUNCH;
  if (cap == cudaStreamCaptureStatusNone) *word = a.host_word;
  return SMOE_OK;
}

#define SMOE_TRY(call)          \
  do {                          \
    const int rc_ = (call);     \
    if (rc_) return rc_;        \
  } while (0)

// Column-quantised B operand of a weight gradient from token-major rows: left [rows, H], or transposed [H, rows]
static int column_operand(const void* src, const Saved& sv, const int32_t* valid, int64_t rows, int64_t H, bool as_rows,
                          void* q, void* sf, void* stream) {
  return as_rows ? smoe_quant_dual_gather(src, sv.x_gather, valid, rows, H, nullptr, nullptr, q, sf, stream)
                 : smoe_quant_cols_t(src, sv.x_gather, valid, rows, H, q, sf, stream);
}

// One weight gradient: operands [dim, rows] or, *_rows, [rows, dim]; mode as in smoe_layer_args
static int wgrad(const void* A, const void* A_sf, bool a_rows, const void* B, const void* B_sf, bool b_rows,
                 const int32_t* efo, void* c, int64_t M, int64_t N, int64_t rows, int64_t E, int mode, int32_t* status,
                 void* stream) {
  const int layout = (a_rows ? 1 : 0) | (b_rows ? 2 : 0);
  if (mode == SMOE_DW_BF16) return smoe_gemm_wgrad_bf16(A, A_sf, B, B_sf, efo, c, M, N, rows, E, layout, status, stream);
  const int acc = mode == SMOE_DW_ACCUMULATE;
  if (layout) return smoe_gemm_wgrad_mn(A, A_sf, B, B_sf, efo, (float*)c, M, N, rows, E, acc, layout, status, stream);
  return smoe_gemm_wgrad(A, A_sf, B, B_sf, efo, (float*)c, M, N, rows, E, acc, status, stream);
}

// Whether an inference call has so few rows per expert that reading the weights bounds its GEMMs.  The host knows the mean and the
// most an expert can get, T rows (a token takes an expert once), not the busiest one.
//   One tile of 64 rows an expert at most: the weights are read once in either form, and this one loses only where every expert
//   is nearly full.  Gated + plain GEMM, routed rows as M against weights as M, us, even loads:
//     E=128 H=2048 I=768, K=8:  4 rows 147 / 115, 32 rows 152 / 133, 48 rows 152 / 150, 64 rows 152 / 215
//     E=32 H=3072 I=1536, K=8:  8 rows 115 / 93, 40 rows 115 / 106, 50 rows 115 / 120
//     E=K=8 H=I=4096:           1 row 100 / 84, 32 rows 100 / 91, 64 rows 101 / 105
//   More: a busy expert's weights are fetched once per 64 rows where the other form needs one pass per 256.  Few rows on average
//   and a bound on what one slot, and all K, put on the same experts keep that small.  Whole forward, replayed from a graph, cold
//   L2, general / this, us (even load; Zipf(1.2), mean of three; all tokens on the same K experts), admitted | beyond the rule:
//     E=128 H=2048 I=768 K=8   T=160  168 / 139, 102 / 95, 49 / 52  |  T=320  168 / 146, 117 / 120, 57 / 78
//                                                                      T=640  174 / 162, 141 / 178, 65 / 121
//     E=128 H=2048 I=768 K=1   T=576  168 / 139, 60 / 51, 43 / 37   |  T=5120  186 / 170, 98 / 154, 72 / 131
//     E=256 H=2048 I=768 K=4   T=320  303 / 238, 89 / 85, 47 / 55   |  T=576  303 / 238, 95 / 104, 53 / 70
//     E=128 H=4096 I=1536 K=4  T=160  509 / 407, 168 / 162, 66 / 84 |  T=256  520 / 420, 183 / 194, 63 / 106
//   Over the 208 points measured that the rule admits (10 layer sizes, 8 to 256 experts, K = 1 to 8) an even load gains 6 to 47 %
//   (median 24), one slot of every token on one expert 0 to 43 (20), a Zipf load 19 in the median and loses at most 6 (one draw of
//   three, 125 / 133); all K slots of all tokens on the same experts, as identical tokens have it, gains 12 in the median and loses
//   at worst a quarter of calls as short as those above.
static bool few_rows(const smoe_layer_args& a) {
  if (a.T <= 40) return true;
  if (a.T <= 64) return a.T * a.K <= 40 * a.E;
  constexpr int64_t kWave = 148;                            // tiles of 128 weight rows x 64 routed rows at a time
  const int64_t slot = (a.T + 63) / 64 * ((a.H > 2 * a.I ? a.H : 2 * a.I) / 128);   // tiles, all tokens on one expert
  return a.T * a.K <= 10 * a.E && slot <= kWave && slot * a.K <= 3 * kWave;
}

}  // namespace smoe

using namespace smoe;

extern "C" {

int64_t smoe_layer_bytes(const smoe_layer_args* a, int which) {
  if (check_args(a)) return -1;
  return (int64_t)(which == 0   ? Saved(*a, nullptr).bytes
                   : which == 1 ? FwdScratch(*a, nullptr).bytes
                                : BwdScratch(*a, nullptr).bytes);
}

int smoe_layer_forward(const smoe_layer_args* args, void* stream) {
  SMOE_TRY(check_args(args));
  const smoe_layer_args& a = *args;
  const Saved sv(a, a.saved);
  const FwdScratch sc(a, a.scratch);
  const int64_t R = a.TKp_alloc, H = a.H, I = a.I, E = a.E;
  const int32_t *rows = sv.efo + E, *real_tk = sv.naept + a.T;
  SMOE_TRY(smoe_topk_metadata(a.idx, a.probs, a.T, a.K, E, 128, a.TK_alloc, R, a.lane_order, a.pad_mode, sv.efo, sv.x_gather,
                              sv.s_scatter, sv.s_rev, sv.naept, sv.scores, sv.src_idx, a.counts, sc.ws, stream));
  SMOE_TRY(smoe_quant_rows_scatter(a.x, a.T, H, sv.naept, sv.s_rev, a.keep_z ? sv.s_scatter : nullptr, rows, R, sc.xg,
                                   sc.xg_sf, stream));
  if (!a.keep_z && few_rows(a)) {
    // Both may begin early: the quantizer, launched the ordinary way, began when offsets, counts and weights were complete, and
    // neither it nor the up-projection writes any of them.  T > 0, so that the quantizer is there
    const bool early = a.T > 0;
    SMOE_TRY(gemm_gated_few(sc.xg, sc.xg_sf, a.w1, a.w1_sf, sv.efo, a.counts, sc.y1, sc.y1_sf, R, 2 * I, H, E, a.status, early,
                            stream));
    SMOE_TRY(gemm_varlen_m_few(sc.y1, sc.y1_sf, a.w2, a.w2_sf, sv.efo, a.counts, sc.y2, R, H, I, E, a.status, early, stream));
  } else {
    if (a.keep_z)
      SMOE_TRY(smoe_gemm_gated(sc.xg, R, nullptr, sc.xg_sf, a.w1, a.w1_sf, sv.efo, sv.z, sv.z_sc, sc.y1, sc.y1_sf, R, 2 * I, H,
                               E, a.status, stream));
    else
      SMOE_TRY(smoe_gemm_gated_infer(sc.xg, sc.xg_sf, a.w1, a.w1_sf, sv.efo, sv.s_scatter, real_tk, sc.y1, sc.y1_sf, R, 2 * I,
                                     H, E, a.status, stream));
    SMOE_TRY(smoe_gemm_varlen_m_live(sc.y1, sc.y1_sf, a.w2, a.w2_sf, sv.efo, sv.s_scatter, real_tk, sc.y2, R, H, I, E,
                                     a.status, stream));
  }
  int32_t* word;
  SMOE_TRY(host_word(a, stream, &word));
  return smoe_combine_post(sc.y2, sv.s_rev, sv.naept, sv.scores, a.out, a.T, H, a.status, word, stream);
}

int smoe_layer_backward(const smoe_layer_args* args, void* stream) {
  SMOE_TRY(check_args(args));
  const smoe_layer_args& a = *args;
  if (!a.keep_z) return SMOE_ERR_ARG;
  const Saved sv(a, a.saved);
  const BwdScratch b(a, a.scratch);
  const int64_t R = a.TKp_alloc, H = a.H, I = a.I, E = a.E;
  const int32_t *rows = sv.efo + E, *real_tk = sv.naept + a.T;
  const bool dw1 = a.dw1_mode != SMOE_DW_NONE, dw2 = a.dw2_mode != SMOE_DW_NONE;
  // dout's column-quantised copy: transposed where dw2 joins the 256 x 384 kernel, else left as rows (13 us cheaper to make
  // at T=8192, H=3072, K=8; the 256 x 256 kernel reads either in the same time)
  const bool dc_rows = b.fused && (!wide_ok(E, I, H) || a.dw2_mode == SMOE_DW_BF16);
  if (!b.fused) SMOE_TRY(smoe_gather_scores(sv.scores, sv.s_scatter, R, b.s, stream));
  SMOE_TRY(smoe_quant_rows_scatter(a.dout, a.T, H, sv.naept, sv.s_rev, sv.s_scatter, rows, R, b.dg, b.dg_sf, stream));
  if (b.fused && dw2) SMOE_TRY(column_operand(a.dout, sv, rows, R, H, dc_rows, b.dc, b.dc_sf, stream));
  if (b.fused) {
    SMOE_TRY(smoe_gemm_dgated_fused_scored(b.dg, b.dg_sf, a.w2, a.w2_sf, sv.efo, sv.z, sv.z_sc, sv.scores, sv.s_scatter, b.dz,
                                           b.dz_rsf, b.dz_csf, b.y1s, b.y1s_sf, b.dsp, R, I, H, E, a.status, stream));
  } else {
    SMOE_TRY(smoe_gemm_dgated(b.dg, R, nullptr, b.dg_sf, a.w2, a.w2_sf, sv.efo, sv.z, sv.z_sc, b.s, b.dz_bf16, b.y1s_bf16,
                              b.dsp, nullptr, R, I, H, E, a.status, stream));
    if (dw2) {
      SMOE_TRY(smoe_quant_cols_t(b.y1s_bf16, nullptr, rows, R, I, b.y1s, b.y1s_sf, stream));
      SMOE_TRY(smoe_quant_cols_t(a.dout, sv.x_gather, rows, R, H, b.dc, b.dc_sf, stream));
    }
    SMOE_TRY(smoe_quant_iso32(b.dz_bf16, R, 2 * I, b.dz, b.dz_rsf, b.dz_t, b.dz_csf, stream));
  }
  if (a.ds) SMOE_TRY(smoe_ds_slots(b.dsp, b.parts, R, sv.s_rev, sv.naept, sv.src_idx, a.T, a.K, a.ds, stream));
  // dx before the weight gradients
  if (a.out) {
    SMOE_TRY(smoe_gemm_varlen_m_live(b.dz, b.dz_rsf, a.w1, a.w1_sf, sv.efo, sv.s_scatter, real_tk, b.dx_exp, R, H, 2 * I, E,
                                     a.status, stream));
    SMOE_TRY(smoe_combine(b.dx_exp, sv.s_rev, sv.naept, nullptr, a.out, a.T, H, stream));
    if (a.dx_ready && cudaEventRecord((cudaEvent_t)a.dx_ready, (cudaStream_t)stream) != cudaSuccess) return SMOE_ERR_LAUNCH;
  }
  bool xc_rows = false;
  if (dw1) {
    xc_rows = mn_ok(E, 2 * I, H) && !wide_ok(E, 2 * I, H);
    SMOE_TRY(column_operand(a.x, sv, rows, R, H, xc_rows, b.xc, b.xc_sf, stream));
  }
  if (a.dw1_mode == SMOE_DW_ACCUMULATE && a.dw2_mode == SMOE_DW_ACCUMULATE && b.fused && !dc_rows && !xc_rows &&
      wide_ok(E, 2 * I, H)) {
    // one launch: one partly filled last wave instead of two
    SMOE_TRY(smoe_gemm_wgrad_mn_pair(b.dz, b.dz_csf, b.xc, b.xc_sf, (float*)a.dw1, 2 * I, b.y1s, b.y1s_sf, b.dc, b.dc_sf,
                                     (float*)a.dw2, I, sv.efo, H, R, E, 1, 1, a.status, stream));
  } else {
    if (a.dw2_mode == SMOE_DW_BF16)      // operands exchanged: the product leaves in the parameter's layout [E,H,I]
      SMOE_TRY(wgrad(b.dc, b.dc_sf, dc_rows, b.y1s, b.y1s_sf, b.fused, sv.efo, a.dw2, H, I, R, E, a.dw2_mode, a.status,
                     stream));
    else if (dw2)
      SMOE_TRY(wgrad(b.y1s, b.y1s_sf, b.fused, b.dc, b.dc_sf, dc_rows, sv.efo, a.dw2, I, H, R, E, a.dw2_mode, a.status,
                     stream));
    if (dw1)
      SMOE_TRY(wgrad(b.fused ? b.dz : b.dz_t, b.dz_csf, b.fused, b.xc, b.xc_sf, xc_rows, sv.efo, a.dw1, 2 * I, H, R, E,
                     a.dw1_mode, a.status, stream));
  }
  int32_t* word;
  SMOE_TRY(host_word(a, stream, &word));
  return word ? smoe_status_post(a.status, word, stream) : SMOE_OK;
}

}  // extern "C"
