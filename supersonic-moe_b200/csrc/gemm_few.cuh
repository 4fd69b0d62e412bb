// MXFP8 grouped GEMM for few rows per expert (inference on few tokens): the weights are the M operand.
//
// What bounds such a call is the read of the weights.  With the routed rows as M (the other kernels here) an expert with
// four rows still costs whole 256-row MMAs: 512 tensor clocks per 256 weight rows and 128-wide K tile, on two SMs, which
// is as long as HBM takes to bring them.  Here a CTA computes 128 weight rows x 64 routed rows: the MMAs of a K
// tile take a fraction of that, each SM streams weight tiles of its own through a deep ring, and of the routed rows
// only as many 16-row pieces are fetched as hold live ones.
//
// The accumulator lies transposed (TMEM lane = weight row, column = routed row).  PLAIN: 32 lanes are 32 consecutive bf16 of
// an output row.  GATED: gate and up lie in neighbouring lanes, the 32 values that share a scale in two neighbouring warps.
// Live rows only are computed and written: the first counts[e] of expert e's segment.
//
// Where its caller allows it (see run_few) the kernel starts before the one before it in the stream has ended: until
// wait_for_kernel_before it touches only offsets, counts and weights.  Its set-up and the weights of the first ring pass then lie under the end of the kernel
// before: an inference call replayed from a graph, E=128 H=2048 I=768 64 tokens 130 -> 123 us, E=32 H=3072 I=1536 64 tokens
// 115 -> 104, E=8 16 tokens 57 -> 51 (starting from 167, 139 and 76 with routed rows as M and the kernels around it as they were).
#pragma once
#include "gemm2.cuh"

namespace smoe {

struct FewParams {
  int N, K, E;          // weight rows per expert, reduction length
  const int* efo;       // [E+1] padded row offsets
  const int* counts;    // [E] routed rows
  const uint8_t *w_sf, *x_sf;      // ISA scales of (E*N, K) and (rows, K)
  __nv_bfloat16* c;     // PLAIN: [rows, N]
  uint8_t *y1, *y1_sf;  // GATED: e4m3 [rows, N/2] and its ISA scales
  int* status;
};

constexpr int kFewNT = 64;        // routed rows of a tile

struct FewSmem {
  static constexpr int NT = kFewNT;
  static constexpr int A_BYTES = BM * BK;                       // 128 weight rows
  static constexpr int B_BYTES = NT * BK;
  static constexpr int SF_BYTES = 1024;                         // scales of both, 512 bytes each
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES + SF_BYTES;
  static constexpr int AMAX_BYTES = 2 * 4 * 16 * 4;             // GATED: [buffer][warp][column]
  static constexpr int AUX_BYTES = 512 + AMAX_BYTES + 3 * (kMaxExperts2 + 1) * 4 + 4;
  static constexpr int STAGES = (227 * 1024 - 1024 - AUX_BYTES) / STAGE_BYTES;           // 8
  static constexpr int TOTAL = STAGES * STAGE_BYTES + AUX_BYTES + 1024;
  static constexpr int SF_COL0 = 2 * NT;                        // two accumulators
  static constexpr int SF_COLS = 8;
  static_assert(SF_COL0 + STAGES * SF_COLS <= 512, "TMEM budget");
  static_assert((2 * STAGES + 4) * 8 <= 496, "barrier storage");
};
constexpr int kFewEpiWarps = 4, kFewThreads = 32 * (2 + kFewEpiWarps);

struct FewTile {
  int e, w0;            // expert; first weight row within it
  int row0, live;       // first routed row; live rows of this tile, 1 .. NT
};
// s_tiles[e] = NT-row tiles of the experts before e.  The row tiles of one weight tile are neighbours: L2 serves the weights.
__device__ __forceinline__ FewTile few_tile(int tile, int NW, int E, const int* s_efo, const int* s_live, const int* s_tiles) {
  FewTile t;
  constexpr int NT = kFewNT;
  const int pr = tile / NW;
  int lo = 0, hi = E;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (s_tiles[mid + 1] <= pr) lo = mid + 1; else hi = mid;
  }
  const int nt = s_tiles[lo + 1] - s_tiles[lo], r = tile - s_tiles[lo] * NW;
  t.e = lo;
  t.w0 = r / nt * BM;
  const int j = r % nt;
  t.row0 = s_efo[lo] + j * NT;
  t.live = min(s_live[lo] - j * NT, NT);
  return t;
}

// logical and over the 64 threads of two warps; a barrier between them
__device__ __forceinline__ bool pair_all(bool x, int bar) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, %2, 64, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)x), "r"(bar)
      : "memory");
  return r != 0;
}

template <int MODE>
__global__ void __launch_bounds__(kFewThreads, 1)
gemm_few_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const FewParams p) {
  static_assert(MODE == PLAIN || MODE == GATED, "forward GEMMs");
  using S = FewSmem;
  constexpr int NT = kFewNT;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* aux = smem + S::STAGES * S::STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(aux);            // full[S], empty[S], tfull[2], tempty[2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(aux + 496);
  volatile int* s_abort = reinterpret_cast<volatile int*>(aux + 500);
  float* s_amax = reinterpret_cast<float*>(aux + 512);
  int* s_efo = reinterpret_cast<int*>(aux + 512 + S::AMAX_BYTES);
  int* s_live = s_efo + (kMaxExperts2 + 1);
  int* s_tiles = s_live + (kMaxExperts2 + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  next_kernel_may_start();
  const uint32_t bar_full = smem_u32(bars);
  const uint32_t bar_empty = bar_full + 8 * S::STAGES;
  const uint32_t bar_tfull = bar_empty + 8 * S::STAGES;
  const uint32_t bar_tempty = bar_tfull + 8 * 2;

  for (int i = threadIdx.x; i <= p.E; i += blockDim.x) s_efo[i] = p.efo[i];
  for (int i = threadIdx.x; i < p.E; i += blockDim.x) s_live[i] = max(min(p.counts[i], p.efo[i + 1] - p.efo[i]), 0);
  __syncthreads();
  if (warp == 2) {                                              // exclusive prefix of the row tiles, eight experts a lane
    constexpr int PER = kMaxExperts2 / 32;
    int v[PER], sum = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = lane * PER + i;
      v[i] = e < p.E ? (s_live[e] + NT - 1) / NT : 0;
      sum += v[i];
    }
    int inc = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += y;
    }
    int run = inc - sum;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = lane * PER + i;
      if (e <= p.E) s_tiles[e] = run;
      run += v[i];
    }
    if (lane == 31 && p.E == kMaxExperts2) s_tiles[p.E] = run;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_tfull + 8 * s, 1);
      mbar_init(bar_tempty + 8 * s, kFewEpiWarps);
    }
    *s_abort = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t smem_base = smem_u32(smem);
  const int NW = p.N / BM, nkt = p.K / BK;
  const int n_total = s_tiles[p.E] * NW;

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      prefetch_tmap(&tmap_w);
      prefetch_tmap(&tmap_x);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      // The weights of the first ring pass are asked for before the kernel that makes the routed rows has ended
      const int n_early = (int)blockIdx.x < n_total ? min(S::STAGES, nkt) : 0;
      auto weights = [&](const FewTile& t, int kt, int st) {
        const uint32_t full = bar_full + 8 * st, a_dst = smem_base + st * S::STAGE_BYTES;
        const int w_row = t.e * p.N + t.w0;
        mbar_expect_tx(full, S::A_BYTES + (t.live + 15) / 16 * 16 * BK + S::SF_BYTES);
        tma_load_2d(a_dst, &tmap_w, full, kt * BK, w_row);
        bulk_load(a_dst + S::A_BYTES + S::B_BYTES, p.w_sf + ((size_t)(w_row / 128) * nkt + kt) * 512, 512, full);
      };
      // rows beyond the last 16-row piece keep what the ring held: it reaches accumulator columns that nobody reads
      auto routed_rows = [&](const FewTile& t, int kt, int st) {
        const uint32_t full = bar_full + 8 * st, b_dst = smem_base + st * S::STAGE_BYTES + S::A_BYTES;
        for (int i = 0; i < t.live; i += 16) tma_load_2d(b_dst + i * BK, &tmap_x, full, kt * BK, t.row0 + i);
        bulk_load(b_dst + S::B_BYTES + 512, p.x_sf + ((size_t)(t.row0 / 128) * nkt + kt) * 512, 512, full);
      };
      if (n_early) {
        const FewTile t = few_tile(blockIdx.x, NW, p.E, s_efo, s_live, s_tiles);
        for (int kt = 0; kt < n_early; ++kt) weights(t, kt, kt);
      }
      wait_for_kernel_before();        // every block, also one without tiles: the kernel after this one counts on it
      for (int tile = blockIdx.x; tile < n_total && ok; tile += gridDim.x) {
        const FewTile t = few_tile(tile, NW, p.E, s_efo, s_live, s_tiles);
        for (int kt = 0; kt < nkt; ++kt) {
          if (tile != (int)blockIdx.x || kt >= n_early) {
            ok = mbar_wait(bar_empty + 8 * stage, phase ^ 1);
            if (!ok) break;
            weights(t, kt, stage);
          }
          routed_rows(t, kt, stage);
          if (++stage == S::STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) { *s_abort = 1; atomicCAS(p.status, 0, 301); }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_mxf8(BM, NT);
      int stage = 0, as = 0;
      uint32_t phase = 0, aphase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < n_total && ok; tile += gridDim.x) {
        const FewTile t = few_tile(tile, NW, p.E, s_efo, s_live, s_tiles);
        ok = mbar_wait(bar_tempty + 8 * as, aphase ^ 1);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + as * NT;
        const uint32_t sfb_shift = (uint32_t)(t.row0 & 127) / 32;      // the second half of a 128-row scale tile
        for (int k = 0; k < nkt; ++k) {
          ok = mbar_wait(bar_full + 8 * stage, phase);
          if (!ok) break;
          tc_fence_after();
          const uint32_t a_src = smem_base + stage * S::STAGE_BYTES, b_src = a_src + S::A_BYTES, sf_src = b_src + S::B_BYTES;
          const uint32_t sfa_t = tmem_base + S::SF_COL0 + stage * S::SF_COLS, sfb_t = sfa_t + 4;
          tc_cp_sf(sfa_t, make_desc_sf(sf_src));
          tc_cp_sf(sfb_t, make_desc_sf(sf_src + 512));
          const uint64_t a_desc = make_desc_kmajor_sw128(a_src), b_desc = make_desc_kmajor_sw128(b_src);
#pragma unroll
          for (int kb = 0; kb < BK / 32; ++kb)
            mma_mxf8(d_tmem, a_desc + 2 * kb, b_desc + 2 * kb, idesc_with_sf_ids(idesc, kb, kb), sfa_t, sfb_t + sfb_shift,
                     (k | kb) != 0);
          tc_commit(bar_empty + 8 * stage);
          if (++stage == S::STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        tc_commit(bar_tfull + 8 * as);
        if (++as == 2) { as = 0; aphase ^= 1; }
      }
      if (!ok) { *s_abort = 1; atomicCAS(p.status, 0, 302); }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue: a warp owns 32 weight rows, its TMEM lanes
    const int q = warp & 3;
    int as = 0, buf = 0;
    uint32_t aphase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < n_total && ok; tile += gridDim.x) {
      const FewTile t = few_tile(tile, NW, p.E, s_efo, s_live, s_tiles);
      ok = mbar_wait(bar_tfull + 8 * as, aphase);
      // (a wait that ran out in one of two warps that exchange maxima ends both)
      ok = MODE == GATED ? pair_all(ok, 1 + (q >> 1)) : __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + as * NT;
      const int col = t.w0 + q * 32 + lane;                     // weight row = output column
#pragma unroll 1
      for (int c0 = 0; c0 < t.live; c0 += 16) {
        uint32_t r[16];
        tmem_ld16(t_row + c0, r);
        tmem_ld_wait();
        const int n = t.live - c0;
        const size_t row = (size_t)t.row0 + c0;
        if (MODE == PLAIN) {
          __nv_bfloat16* dst = p.c + row * p.N + col;
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (i < n) dst[(size_t)i * p.N] = __float2bfloat16_rn(__uint_as_float(r[i]));
        } else {
          // both lanes of a pair hold the pair's y; the 32 y of a scale are those of warps q and q ^ 1
          float y[16];
          float mine = 0.f;                                     // lane i: column i's maximum over this warp
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float a = __uint_as_float(r[i]), b = __shfl_xor_sync(0xffffffffu, a, 1);
            const float g = (lane & 1) ? b : a, u = (lane & 1) ? a : b;
            y[i] = bf16_rne((g * fast_sigmoid(g)) * u);
            const float m = warp_max_abs(y[i]);
            if ((lane & 15) == i) mine = m;
          }
          float* am = s_amax + buf * 64;
          if (lane < 16) am[q * 16 + lane] = mine;
          asm volatile("bar.sync %0, 64;" ::"r"(1 + (q >> 1)) : "memory");
          // of column lane & 15; a group of nothing but NaN has the scale of zeros, as in the other kernels (maxima from 0 on)
          const int e = e8m0_of(fmaxf(fmaxf(mine, am[(q ^ 1) * 16 + (lane & 15)]), 0.f));
          const float qs_mine = qscale_of(e);
          buf ^= 1;           // the other buffer next: this one is written again only after one more barrier
          const int Ny = p.N / 2, yc = col >> 1;
          uint8_t* dst = p.y1 + row * Ny + yc;
#pragma unroll
          for (int i = 0; i < 16; i += 2) {                     // even lanes store column i, odd lanes column i + 1
            const float q0 = __shfl_sync(0xffffffffu, qs_mine, i), q1 = __shfl_sync(0xffffffffu, qs_mine, i + 1);
            const float v = (lane & 1) ? y[i + 1] * q1 : y[i] * q0;
            const int t_i = i + (lane & 1);
            if (t_i < n) dst[(size_t)t_i * Ny] = (uint8_t)pack_e4m3x4(v, v, v, v);
          }
          if ((q & 1) == 0 && lane < 16 && lane < n) {
            const size_t rr = row + lane;
            const int g = yc >> 5;
            p.y1_sf[((rr >> 7) * (size_t)(Ny / 128) + g / 4) * 512 + (rr & 31) * 16 + ((rr & 127) >> 5) * 4 + (g & 3)] =
                (uint8_t)e;
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_tempty + 8 * as);
      if (++as == 2) { as = 0; aphase ^= 1; }
    }
    if (!ok && lane == 0) { *s_abort = 1; atomicCAS(p.status, 0, 303); }
  }

  // common exit: everyone arrives here, also after a failed wait
  __syncthreads();
  if (*s_abort) {                             // copies and MMAs in flight may still write this CTA's memory
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

}  // namespace smoe
