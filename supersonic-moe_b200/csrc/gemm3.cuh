// Two-CTA MXFP8 grouped GEMM with a 256 x 384 tile held as TWO accumulators of 256 x 192 (TMEM columns 0..191 and
// 192..383) that share every A tile.
//
// Why: per 128-wide K tile a CTA of this kernel loads A (16 KB) once for two B halves (2 x 12 KB): 40 KB for 768
// tensor clocks instead of 32 KB for 512 - 17 % fewer operand bytes per MMA than the 256 x 256 tile - with no
// multicast load anywhere (each CTA fetches its own rows of A and of both B halves with plain tiled TMA copies).
// When it was written that bought 7-9 % on the plain and weight-gradient GEMMs; since the accumulator hand-back no
// longer stalls (relaxed arrival, see the epilogue) either kernel is the faster one for the plain GEMM, by up to 6 and 11 %,
// as the routed rows have it, and this one stays where N is a multiple of 384 only (`use_gemm3` in gemm.cu has the rule
// and the figures).  It is also the one that runs the two weight gradients of a layer in a single launch.
//
// The two accumulators also hide the accumulator hand-over between tiles: the last J K tiles of a tile are issued
// half 0 first, so the epilogue drains accumulator 0 under the half-1 MMAs of those K tiles, and the next tile
// starts with J K tiles of half 0 while accumulator 1 is still being drained.
//
// Modes: PLAIN (bf16 C through TMA stores) and WGRAD (f32 C through TMA store / reduce-add; A may be MN-major, B is
// K-major).  N must be a multiple of 384.
#pragma once
#include "gemm2.cuh"

namespace smoe {

constexpr int kBN3 = 384;          // tile width
constexpr int kHN3 = 192;          // width of one accumulator
constexpr int kHeadTail3 = 2;      // K tiles issued half-by-half at both ends of a tile

// Reduce-adds of this kernel into a gradient that lies in HBM.  With a few K tiles a tile all SMs together ask for more than HBM
// gives, and what it gives then drops from 6.4 TB/s (read and written) to 5.4: deeper prefetches (kReduceAhead) change nothing, two
// thirds of the SMs would run at the full rate, but how many that takes depends on the clocks.  So a warp has its pieces loaded into
// shared memory, where nobody reads them, and adds to a piece only once it has arrived: never more than two of its pieces are on
// their way.  That costs wherever HBM is not what everybody waits for, so it is done for tiles of at most kReduceLoadKTiles K
// tiles in a launch (`reduce_loads`) that has few K tiles an expert in the mean, where every expert has rows, and many tiles a CTA
// pair.  Loaded over prefetched, E=8 to 128, 1 to 5 K tiles an expert, even, Zipf and single busy experts, from a cold L2, at full
// clocks and behind three large GEMMs, which take the clock down:
//   24 tiles a CTA pair and more, every expert with rows   0.87 to 0.96 and 0.79 to 0.99
//   15 to 24 tiles                                         0.90 to 1.01 and 0.90 to 1.05
//   3 to 15 tiles                                          0.92 to 1.05 and 0.93 to 1.11
//   half the experts without rows, seven eighths           0.90 to 1.11 and 0.92 to 1.18, 1.05 to 1.22 and 1.07 to 1.26
// us: dw1 + dw2, E=8 M=6144 + 3072 N=6144, 1 / 2 / 3 / 4 / 5 K tiles 700 / 707 / 727 / 748 / 764 -> 619 / 629 / 641 / 649 / 663.  At 6
// K tiles either is the better one for some sizes, from 7 on the MMAs do the pacing; 9 in the mean and a Zipf load lose 3 %.  One, three
// or four pieces on their way instead of two: no gain.  The 256-column kernel, with 24 tiles and more and every expert with rows, takes
// 0.83 to 1.01 at full clocks and 0.89 to 1.14 behind large GEMMs, so it prefetches.
constexpr int kReduceLoadKTiles = 5;
constexpr int kReduceLoadMean = 5;
constexpr int kReduceLoadTiles = 24;     // a CTA pair
constexpr int kReduceLoads = 2;
constexpr int kReducePiece = 4096;       // bytes of a piece

// k_tiles: of all experts; busy: experts with rows, of E; tiles: of the launch, for `pairs` CTA pairs
__host__ __device__ inline bool reduce_loads(int k_tiles, int busy, int E, int tiles, int pairs) {
  return k_tiles <= kReduceLoadMean * E && busy == E && tiles >= kReduceLoadTiles * pairs;
}

// Pieces of an existing gradient on their way into the L2; one lane of an epilogue warp
struct OldPieces {
  uint32_t bars;                   // kReduceLoads barriers of this warp
  uint32_t sink;                   // where the bytes land: any warp's may overwrite any other's
  uint32_t asked = 0, seen = 0;
  __device__ void ask(const void* tmap, int c0, int c1) {
    const uint32_t bar = bars + 8 * (asked++ % kReduceLoads);
    mbar_expect_tx(bar, kReducePiece);
    tma_load_2d(sink, tmap, bar, c0, c1);
  }
  __device__ bool await() {
    const uint32_t n = seen++;
    return mbar_wait(bars + 8 * (n % kReduceLoads), (n / kReduceLoads) & 1);
  }
};

template <int MODE>
struct Gemm3Smem {
  static constexpr int A_BYTES = BM * BK;                       // this CTA's 128 rows of A
  static constexpr int BH_BYTES = (kHN3 / 2) * BK;              // this CTA's 96 rows of one B half
  static constexpr int STAGE_BYTES = A_BYTES + 2 * BH_BYTES;    // 40 KB
  static constexpr int SFB_TILES = 3;                           // 128-row scale tiles covering the 384 B rows
  static constexpr int SF_GROUP = kSfGroup2;
  static constexpr int SF_SLOT_BYTES = SF_GROUP * 512 * (1 + SFB_TILES);
  static constexpr int SF_SLOTS = 2;
  static constexpr int SF_BYTES = SF_SLOTS * SF_SLOT_BYTES;
  static constexpr int EPI_WARPS = 8;                           // four TMEM lane quadrants x two column groups
  static constexpr int LEAD_WARPS = 3;                          // operand producer, MMA issuer, scale producer
  static constexpr int THREADS = 32 * (LEAD_WARPS + EPI_WARPS);
  static constexpr int EPI_BUFS = 2;                            // staging buffers per warp, used in turn
  static constexpr int EPI_BYTES_PER_WARP = EPI_BUFS * 2048;    // bf16 32x32 or f32 32x16 per buffer
  static constexpr int EPI_BYTES = EPI_WARPS * EPI_BYTES_PER_WARP;
  static constexpr int SINK_BYTES = MODE == WGRAD ? kReducePiece : 0;      // where pieces of the old gradient land
  static constexpr int AUX_BYTES = 512 + 2 * (kMaxExperts2 + 1) * 4 + 8;
  static constexpr int STAGES = 4;
  static constexpr int TOTAL = STAGES * STAGE_BYTES + SF_BYTES + EPI_BYTES + SINK_BYTES + AUX_BYTES + 1024;
  static_assert((2 * STAGES + 4 + 2 * SF_SLOTS + kReduceLoads * EPI_WARPS) * 8 <= 496, "barrier storage");
  static_assert(TOTAL <= 227 * 1024, "shared memory budget");
  static constexpr int SF_COLS = 4 + 4 * SFB_TILES;             // TMEM columns of one stage's scales
  static constexpr int SF_COL0 = kBN3;
  static_assert(SF_COL0 + STAGES * SF_COLS <= 512, "TMEM budget");
  static constexpr uint32_t TX_BYTES = 2u * STAGE_BYTES;        // both CTAs' A and B per stage
  static constexpr uint32_t SF_TX_BYTES = 2u * SF_SLOT_BYTES;
};

// Tensor maps of a second weight-gradient product that shares the launch (GemmParams::rows2 > 0): two products
// whose tile counts are no multiples of the number of CTA pairs leave one partly filled last wave together instead
// of one each.
struct SecondMaps {
  CUtensorMap a, b, sfa, sfb, c;
};

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__((Gemm3Smem<MODE>::THREADS), 1)
gemm3_mxf8_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                  const __grid_constant__ CUtensorMap tmap_sfa, const __grid_constant__ CUtensorMap tmap_sfb,
                  const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ SecondMaps second,
                  const GemmParams p) {
  static_assert(kReduceAhead <= 3, "pieces fetched before the wait lie in the first half");
  static_assert(MODE == PLAIN || MODE == WGRAD, "the 384-wide tile exists for the plain and weight-gradient GEMMs");
  using S = Gemm3Smem<MODE>;
  constexpr int BN = kBN3, HN = kHN3;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sfring = smem + S::STAGES * S::STAGE_BYTES;
  uint8_t* epi = sfring + S::SF_BYTES;
  uint8_t* sink = epi + S::EPI_BYTES;
  uint8_t* aux = sink + S::SINK_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(aux);     // full[S], empty[S], tfull[2], tempty[2], sffull[2], sfempty[2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(aux + 496);
  volatile int* s_abort = reinterpret_cast<volatile int*>(aux + 500);
  int* s_efo = reinterpret_cast<int*>(aux + 512);
  int* s_pairs = s_efo + (kMaxExperts2 + 1);
  volatile int* s_loads_old = s_pairs + (kMaxExperts2 + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair_id = blockIdx.x >> 1;
  const int n_pairs_grid = gridDim.x >> 1;
  const uint32_t bar_full = smem_u32(bars);
  const uint32_t bar_empty = bar_full + 8 * S::STAGES;
  const uint32_t bar_tfull = bar_empty + 8 * S::STAGES;    // one per accumulator half
  const uint32_t bar_tempty = bar_tfull + 8 * 2;
  const uint32_t bar_sffull = bar_tempty + 8 * 2;
  const uint32_t bar_sfempty = bar_sffull + 8 * S::SF_SLOTS;
  const uint32_t bar_old = bar_sfempty + 8 * S::SF_SLOTS;  // pieces of the old gradient, kReduceLoads a warp

  for (int i = threadIdx.x; i <= p.E; i += blockDim.x) s_efo[i] = p.efo[i];
  __syncthreads();
  if (warp == 2) {
    prefix_row_pairs(s_efo, s_pairs, p.E, lane);
    if (MODE == WGRAD) {
      int busy = 0;
      for (int e = lane; e < p.E; e += 32) busy += s_efo[e + 1] > s_efo[e];
      busy = (int)__reduce_add_sync(0xffffffffu, busy);
      *s_loads_old = reduce_loads(s_efo[p.E] / BK, busy, p.E, p.E * ((p.rows + p.rows2) / (2 * BM)) * (p.N / BN), n_pairs_grid);
    }
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(bar_full + 8 * s, 1);        // leader's: its own producer arms it; both CTAs' copies credit it
      mbar_init(bar_empty + 8 * s, 1);       // one commit arrival per use, in each CTA
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_tfull + 8 * s, 1);                   // commit arrival, in each CTA
      mbar_init(bar_tempty + 8 * s, 2 * S::EPI_WARPS);     // leader's: the epilogue warps of both CTAs
    }
    for (int s = 0; s < S::SF_SLOTS; ++s) {
      mbar_init(bar_sffull + 8 * s, 1);
      mbar_init(bar_sfempty + 8 * s, 1);
    }
    if (MODE == WGRAD)
      for (int s = 0; s < kReduceLoads * S::EPI_WARPS; ++s) mbar_init(bar_old + 8 * s, 1);
    *s_abort = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc2(smem_u32(tmem_slot), 512);
    tmem_relinquish2();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t sf_base = smem_u32(sfring);
  const int n_col_tiles = p.N / BN;
  const int n_total = (MODE == WGRAD) ? p.E * ((p.rows + p.rows2) / (2 * BM)) * n_col_tiles
                                      : s_pairs[p.E] * n_col_tiles;
  const bool a_mn = MODE == WGRAD && p.a_mn;
  constexpr int nst = S::STAGES;

  if (warp == 0) {
    // ------------------------------------------------------------ producer (both CTAs): warp-uniform loops, one
    // elected lane issues
    if (lane == 0) {
      prefetch_tmap(&tmap_a); prefetch_tmap(&tmap_b);
      if (MODE == WGRAD && p.rows2 > 0) { prefetch_tmap(&second.a); prefetch_tmap(&second.b); }
    }
    const uint32_t full0 = map_to_cta(bar_full, 0);
    const int n_total_u = __shfl_sync(0xffffffffu, n_total, 0);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = pair_id; tile < n_total_u && ok; tile += n_pairs_grid) {
      const PairTile tl = pair_tile<BN, MODE>(tile, rank, p, s_efo, s_pairs);
      const int nkt = __shfl_sync(0xffffffffu, tl.nkt, 0);
      if (nkt == 0) continue;
      const int kt0 = __shfl_sync(0xffffffffu, tl.kt0, 0);
      const int valid = __shfl_sync(0xffffffffu, tl.valid, 0);
      const int m0 = __shfl_sync(0xffffffffu, tl.m0, 0);
      const int n0 = __shfl_sync(0xffffffffu, tl.n0, 0);
      const int te = __shfl_sync(0xffffffffu, tl.e, 0);
      const int b_base = (MODE == WGRAD) ? n0 : te * p.N + n0;
      const int b_row = b_base + rank * (HN / 2);        // this CTA's 96 rows of half 0; half 1 lies HN rows further
      const int a_row = valid ? m0 : 0;
      // the phantom half of an odd last row pair: its A rows are not fetched (see gemm2_mxf8_kernel)
      const bool phantom = MODE != WGRAD && __shfl_sync(0xffffffffu, m0 + (rank ? 0 : BM) >= s_efo[te + 1], 0);
      const uint32_t tx_bytes = S::TX_BYTES - (phantom ? S::A_BYTES : 0);
      const bool second_prob = MODE == WGRAD && __shfl_sync(0xffffffffu, tl.prob, 0) != 0;
      const CUtensorMap* ta = second_prob ? &second.a : &tmap_a;
      const CUtensorMap* tb = second_prob ? &second.b : &tmap_b;
      for (int kt = kt0; kt < kt0 + nkt; ++kt) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * stage, phase ^ 1));
        if (!ok) break;
        const uint32_t full = full0 + 8 * stage;
        const uint32_t a_dst = smem_base + stage * S::STAGE_BYTES;
        const uint32_t b_dst = a_dst + S::A_BYTES;
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(bar_full + 8 * stage, tx_bytes);
          if (a_mn) tma_load_2d_pair(a_dst, ta, full, m0, kt * BK);
          else if (!(phantom && rank == 1)) tma_load_2d_pair(a_dst, ta, full, kt * BK, a_row);
          tma_load_2d_pair(b_dst, tb, full, kt * BK, b_row);
          tma_load_2d_pair(b_dst + S::BH_BYTES, tb, full, kt * BK, b_row + HN);
        }
        if (++stage == nst) { stage = 0; phase ^= 1; }
      }
    }
    if (!ok && lane == 0) { *s_abort = 1; atomicCAS(p.status, 0, 201); }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only): warp-uniform loops,
    // one elected lane issues
    if (rank == 0) {
      const uint32_t idesc = make_idesc_mxf8(2 * BM, HN) | (a_mn ? 1u << 15 : 0u);
      const uint32_t idesc_kb[4] = {idesc_with_sf_ids(idesc, 0, 0), idesc_with_sf_ids(idesc, 1, 1),
                                    idesc_with_sf_ids(idesc, 2, 2), idesc_with_sf_ids(idesc, 3, 3)};
      const uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
      const uint32_t sf_hi = (128u >> 4) | (1u << 14);
      const uint32_t a_step = a_mn ? 256u : 2u;
      const uint32_t a_lo0 = ((smem_base & 0x3FFFF) >> 4) | ((a_mn ? (uint32_t)(S::A_BYTES >> 4) : 1u) << 16);
      const uint32_t b_lo0 = (((smem_base + S::A_BYTES) & 0x3FFFF) >> 4) | (1u << 16);
      const uint32_t sf_lo0 = (sf_base & 0x3FFFF) >> 4;
      const int n_total_u = __shfl_sync(0xffffffffu, n_total, 0);
      int stage = 0, sfs = 0;
      uint32_t phase = 0, aphase = 0, sfphase = 0;
      bool ok = true;
      // MMAs of K tile number k (of its tile) held in ring stage st, into accumulator half h
      auto issue_half = [&](int st, int k, int h) {
        const uint32_t a_lo = a_lo0 + st * (S::STAGE_BYTES >> 4);
        const uint32_t b_lo = b_lo0 + st * (S::STAGE_BYTES >> 4) + h * (S::BH_BYTES >> 4);
        const uint32_t sfa_t = tmem_base + S::SF_COL0 + st * S::SF_COLS;
        const uint32_t sfb_t = sfa_t + 4 + 6 * h;              // 192 B rows = six 32-row scale columns per half
#pragma unroll
        for (int kb = 0; kb < BK / 32; ++kb)
          mma_mxf8_pair_lo(tmem_base + h * HN, a_lo + a_step * kb, b_lo + 2u * kb, desc_hi, idesc_kb[kb], sfa_t, sfb_t,
                           (k | kb) != 0);
      };

      for (int tile = pair_id; tile < n_total_u && ok; tile += n_pairs_grid) {
        const PairTile t = pair_tile<BN, MODE>(tile, 0, p, s_efo, s_pairs);
        const int nkt = __shfl_sync(0xffffffffu, t.nkt, 0);
        if (nkt == 0) continue;
        const int J = nkt >= 2 * kHeadTail3 ? kHeadTail3 : 0;      // K tiles issued half-by-half at both ends of a tile
        int held0 = 0, held1 = 0;             // ring stages of the K tiles whose half-1 MMAs are still to come
        static_assert(kHeadTail3 == 2, "held0 / held1");
        ok = __all_sync(0xffffffffu, mbar_wait(bar_tempty, aphase ^ 1));
        if (!ok) break;
        if (J == 0) {
          ok = __all_sync(0xffffffffu, mbar_wait(bar_tempty + 8, aphase ^ 1));
          if (!ok) break;
        }
        tc_fence_after();
        for (int k = 0; k < nkt; ++k) {
          // first touch of K tile k: its operands and scales have landed; scales go to TMEM; half 0 always,
          // half 1 too unless the K tile belongs to the head or the tail of the tile
          const int kg = k & (S::SF_GROUP - 1);
          if (kg == 0) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar_sffull + 8 * sfs, sfphase));
            if (!ok) break;
          }
          ok = __all_sync(0xffffffffu, mbar_wait(bar_full + 8 * stage, phase));
          if (!ok) break;
          const bool both = (k >= J && k < nkt - J);
          const bool sf_done = (kg == S::SF_GROUP - 1 || k == nkt - 1);
          const uint32_t sf_lo = sf_lo0 + ((sfs * S::SF_SLOT_BYTES + kg * 512) >> 4);
          const uint32_t sfa_t = tmem_base + S::SF_COL0 + stage * S::SF_COLS;
          if (elect_one()) {
            tc_cp_sf_pair_lo(sfa_t, sf_lo, sf_hi);
#pragma unroll
            for (int j = 0; j < S::SFB_TILES; ++j)
              tc_cp_sf_pair_lo(sfa_t + 4 + 4 * j, sf_lo + ((S::SF_GROUP * 512 * (1 + j)) >> 4), sf_hi);
            if (sf_done) tc_commit_pair(bar_sfempty + 8 * sfs, 3);   // the copies above were the slot's last readers
            issue_half(stage, k, 0);
            if (both) {
              issue_half(stage, k, 1);
              tc_commit_pair(bar_empty + 8 * stage, 3);
            }
          }
          if (!both) {
            if ((k < J ? k : k - (nkt - J)) == 0) held0 = stage; else held1 = stage;
          }
          if (++stage == nst) { stage = 0; phase ^= 1; }
          if (sf_done) {
            if (++sfs == S::SF_SLOTS) { sfs = 0; sfphase ^= 1; }
          }
          // end of the head / of the tail: the half-1 MMAs of the K tiles held back
          const bool head_end = (J > 0 && k == J - 1), tail_end = (J > 0 && k == nkt - 1);
          if (head_end) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar_tempty + 8, aphase ^ 1));
            if (!ok) break;
            tc_fence_after();
          }
          if (head_end || tail_end) {
            if (elect_one()) {
              if (tail_end) tc_commit_pair(bar_tfull, 3);          // accumulator 0 is complete
              const int kfirst = head_end ? 0 : nkt - J;
              issue_half(held0, kfirst, 1);
              tc_commit_pair(bar_empty + 8 * held0, 3);
              if (J == 2) {
                issue_half(held1, kfirst + 1, 1);
                tc_commit_pair(bar_empty + 8 * held1, 3);
              }
            }
          }
        }
        if (!ok) break;
        if (elect_one()) {
          if (J == 0) tc_commit_pair(bar_tfull, 3);
          tc_commit_pair(bar_tfull + 8, 3);
        }
        aphase ^= 1;
      }
      if (!ok && lane == 0) { *s_abort = 1; atomicCAS(p.status, 0, 202); }
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------------------------------------ scale producer (both CTAs).  A warp of its own:
    // the scales of the next group of K tiles are requested as soon as a slot of their ring is free - up to two
    // groups (eight K tiles) ahead of the MMAs - instead of when the operand ring gets there (two to four K tiles
    // ahead, about the latency of the small copies while L2 is busy with the operands).
    if (lane == 0) {
      prefetch_tmap(&tmap_sfa); prefetch_tmap(&tmap_sfb);
      if (MODE == WGRAD && p.rows2 > 0) { prefetch_tmap(&second.sfa); prefetch_tmap(&second.sfb); }
    }
    const uint32_t sffull0 = map_to_cta(bar_sffull, 0);
    const int n_total_u = __shfl_sync(0xffffffffu, n_total, 0);
    int sfs = 0;
    uint32_t sfphase = 0;
    bool ok = true;
    for (int tile = pair_id; tile < n_total_u && ok; tile += n_pairs_grid) {
      const PairTile tl = pair_tile<BN, MODE>(tile, rank, p, s_efo, s_pairs);
      const int nkt = __shfl_sync(0xffffffffu, tl.nkt, 0);
      if (nkt == 0) continue;
      const int kt0 = __shfl_sync(0xffffffffu, tl.kt0, 0);
      const int valid = __shfl_sync(0xffffffffu, tl.valid, 0);
      const int m0 = __shfl_sync(0xffffffffu, tl.m0, 0);
      const int n0 = __shfl_sync(0xffffffffu, tl.n0, 0);
      const int te = __shfl_sync(0xffffffffu, tl.e, 0);
      const int b_base = (MODE == WGRAD) ? n0 : te * p.N + n0;
      const int sfa_tile = valid ? m0 / 128 : 0;         // phantom half: any in-range tile will do
      const int sfb_tile = b_base / 128;                 // n0 is a multiple of 384, hence of 128
      const bool second_prob = MODE == WGRAD && __shfl_sync(0xffffffffu, tl.prob, 0) != 0;
      const CUtensorMap* tsa = second_prob ? &second.sfa : &tmap_sfa;
      const CUtensorMap* tsb = second_prob ? &second.sfb : &tmap_sfb;
      for (int kt = kt0; kt < kt0 + nkt; kt += S::SF_GROUP) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar_sfempty + 8 * sfs, sfphase ^ 1));
        if (!ok) break;
        if (elect_one()) {
          const uint32_t sffull = sffull0 + 8 * sfs;
          const uint32_t dst = sf_base + sfs * S::SF_SLOT_BYTES;
          if (rank == 0) mbar_expect_tx(bar_sffull + 8 * sfs, S::SF_TX_BYTES);
          tma_load_2d_pair(dst, tsa, sffull, 0, sfa_tile * p.sfa_ktiles + kt);
#pragma unroll
          for (int j = 0; j < S::SFB_TILES; ++j)
            tma_load_2d_pair(dst + S::SF_GROUP * 512 * (1 + j), tsb, sffull, 0,
                             (sfb_tile + j) * p.sfb_ktiles + kt);
        }
        if (++sfs == S::SF_SLOTS) { sfs = 0; sfphase ^= 1; }
      }
    }
    if (!ok && lane == 0) { *s_abort = 1; atomicCAS(p.status, 0, 206); }
  } else {
    // ------------------------------------------------------------ epilogue: 8 warps per CTA, each owns 32 rows
    // (its TMEM lane quadrant) x 96 columns of each accumulator half
    const int q = warp & 3;                      // the TMEM lane quadrant a warp may read is its index modulo 4
    const int grp = (warp - S::LEAD_WARPS) >> 2;
    const int row_in_tile = q * 32 + lane;
    constexpr int CPW = HN / 2;                 // columns per warp and half
    constexpr int NC = CPW / 32;                // 32-column chunks
    const uint32_t stg = smem_u32(epi + (warp - S::LEAD_WARPS) * S::EPI_BYTES_PER_WARP);
    const uint32_t tempty0 = map_to_cta(bar_tempty, 0);
    uint32_t aphase = 0;
    int buf = 0;
    bool ok = true;
    OldPieces old{bar_old + 8 * kReduceLoads * (warp - S::LEAD_WARPS), smem_u32(sink)};
    for (int tile = pair_id; tile < n_total && ok; tile += n_pairs_grid) {
      const PairTile t = pair_tile<BN, MODE>(tile, rank, p, s_efo, s_pairs);
      const size_t grow = (size_t)t.m0 + row_in_tile;
      if (t.nkt == 0) {
        if (MODE == WGRAD && p.out_bf16) {
          uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.c) +
                                                ((size_t)t.e * p.rows + grow) * p.N + t.n0 + grp * (BN / 2));
          for (int i = 0; i < BN / 16; ++i) dst[i] = make_uint4(0, 0, 0, 0);
        } else if (MODE == WGRAD && !p.accumulate) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(t.prob ? p.c2 : p.c) +
                                                    ((size_t)t.e * (t.prob ? p.rows2 : p.rows) + grow) * p.N + t.n0 +
                                                    h * HN + grp * CPW);
            for (int i = 0; i < CPW / 4; ++i) dst[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
        continue;
      }
      if (MODE == PLAIN) {
        const bool live = slab_live(p, t, t.m0 + q * 32);
        // both halves are drained (bf16-packed) before anything is stored, so that neither accumulator waits
        // for the other one's stores
        uint32_t pk[2][NC][16];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (lane == 0) ok = mbar_wait(bar_tfull + 8 * h, aphase);
          ok = __shfl_sync(0xffffffff, ok, 0);
          if (!ok) break;
          tc_fence_after();
          // all of this warp's columns of the half in one go (one wait), the accumulator is handed back before
          // the conversion: the drain is what the next tile's MMAs wait for
          const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + h * HN + grp * CPW;
          uint32_t r[NC][32];
#pragma unroll
          for (int c = 0; c < NC; ++c) tmem_ld32(t_row + c * 32, r[c]);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_relaxed(tempty0 + 8 * h);
#pragma unroll
          for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int i = 0; i < 16; ++i)
              pk[h][c][i] = pack_bf16x2(__uint_as_float(r[c][2 * i]), __uint_as_float(r[c][2 * i + 1]));
        }
        if (!ok) break;
        if (live) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              const uint32_t sb = stg + buf * 2048;
              if (lane == 0) bulk_wait_group_read<S::EPI_BUFS - 1>();   // the store that last read this buffer is done
              __syncwarp();
#pragma unroll
              for (int j = 0; j < 4; ++j)
                st_shared_v4(sb + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4), pk[h][c][4 * j], pk[h][c][4 * j + 1],
                             pk[h][c][4 * j + 2], pk[h][c][4 * j + 3]);
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                tma_store_2d(&tmap_c, sb, t.n0 + h * HN + grp * CPW + c * 32, t.m0 + q * 32);
                bulk_commit_group();
              }
              buf ^= 1;
            }
          }
        }
      } else {  // WGRAD: f32, one half at a time (96 accumulator registers per half)
        const CUtensorMap* dw_map = t.prob ? &second.c : &tmap_c;
        const int dw_row = t.e * (t.prob ? p.rows2 : p.rows) + t.m0 + q * 32, dw_col = t.n0 + grp * CPW;
        const bool load_old = p.accumulate && t.nkt <= kReduceLoadKTiles && *s_loads_old;
        const bool ahead = p.accumulate && !load_old && t.nkt <= kReduceAheadKTiles;
        if (lane == 0) {                                        // the first pieces of the old gradient
          if (load_old)
            for (int c = 0; c < kReduceLoads; ++c) old.ask(dw_map, dw_col + c * 32, dw_row);
          else if (ahead)
            for (int c = 0; c < kReduceAhead; ++c) tma_prefetch_l2_2d(dw_map, dw_col + c * 32, dw_row);
        }
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          if (lane == 0) ok = mbar_wait(bar_tfull + 8 * h, aphase);
          ok = __shfl_sync(0xffffffff, ok, 0);
          if (!ok) break;
          tc_fence_after();
          uint32_t acc[NC][32];
          const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + h * HN + grp * CPW;
#pragma unroll
          for (int c = 0; c < NC; ++c) tmem_ld32(t_row + c * 32, acc[c]);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_relaxed(tempty0 + 8 * h);
          if (p.out_bf16) {
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              const uint32_t sb = stg + buf * 2048;
              if (lane == 0) bulk_wait_group_read<S::EPI_BUFS - 1>();
              __syncwarp();
              stage_bf16_32(sb, lane, acc[c]);
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                tma_store_2d(&tmap_c, sb, t.n0 + h * HN + grp * CPW + c * 32, t.e * p.rows + t.m0 + q * 32);
                bulk_commit_group();
              }
              buf ^= 1;
            }
            continue;
          }
          if (p.accumulate) {                   // whole 128-byte lines, both staging buffers as one (see gemm2.cuh)
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              if (lane == 0) {
                const int a = h * NC + c + (load_old ? kReduceLoads : kReduceAhead);      // piece number, three a half
                const int acol = dw_col + a / NC * HN + a % NC * 32;
                if (load_old) {
                  ok &= old.await();
                  if (a < 2 * NC) old.ask(dw_map, acol, dw_row);
                } else if (ahead && a < 2 * NC) {
                  tma_prefetch_l2_2d(dw_map, acol, dw_row);
                }
                bulk_wait_group_read<0>();
              }
              __syncwarp();
              stage_f32_32(stg, lane, acc[c]);
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                tma_reduce_add_2d(dw_map, stg, dw_col + h * HN + c * 32, dw_row);
                bulk_commit_group();
              }
            }
            ok = __shfl_sync(0xffffffff, ok, 0);
            if (!ok) break;
            continue;
          }
#pragma unroll
          for (int c = 0; c < 2 * NC; ++c) {
            const uint32_t sb = stg + buf * 2048;
            if (lane == 0) bulk_wait_group_read<S::EPI_BUFS - 1>();
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; ++j)
              st_shared_v4(sb + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4), acc[c >> 1][(c & 1) * 16 + 4 * j],
                           acc[c >> 1][(c & 1) * 16 + 4 * j + 1], acc[c >> 1][(c & 1) * 16 + 4 * j + 2],
                           acc[c >> 1][(c & 1) * 16 + 4 * j + 3]);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              const int crow = t.e * (t.prob ? p.rows2 : p.rows) + t.m0 + q * 32;
              const int ccol = t.n0 + h * HN + grp * CPW + c * 16;
              const CUtensorMap* tc = t.prob ? &second.c : &tmap_c;
              tma_store_2d(tc, sb, ccol, crow);
              bulk_commit_group();
            }
            buf ^= 1;
          }
        }
        if (!ok) break;
      }
      aphase ^= 1;
    }
    if (lane == 0) bulk_wait_group<0>();      // all staged stores have left shared memory and are visible
    if (!ok && lane == 0) { *s_abort = 1; atomicCAS(p.status, 0, 203); }
  }

  // common exit: everyone arrives here, also after a failed wait
  __syncthreads();
  if (*s_abort) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  cluster_sync_all();                         // the peer may still be signalling this CTA's barriers
  tc_fence_after();
  if (warp == 1) tmem_dealloc2(tmem_base, 512);
}

}  // namespace smoe
