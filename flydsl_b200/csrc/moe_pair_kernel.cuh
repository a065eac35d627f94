// Grouped GEMM for large routing blocks (64, 128 or 256 rows) on CTA pairs: a cluster of two CTAs owns up to 256 sorted
// rows of ONE expert x a channel pair (256 columns: stage 1 gate | up, stage 2 two neighbouring tiles) and drives them with
// tcgen05.mma.cta_group::2 (UMMA M = 256, N = 256).  CTA r holds rows [128 r, 128 r + 128) and loads tile r of the channel
// pair: 32 KiB per k-block into each SM for the products of two 128-row items, which take 48 KiB each, and an expert of up
// to 256 rows reads its weights once.  Signalling between the two CTAs, the ring and the two accumulators are those of
// the plain pair form (rows2_kernel.cuh), the epilogue that of the 128-row form (moe_kernel.cuh).
//
// What bounds it: the weight stream where experts are small (800 tokens x top-4, 32 experts, 3072 x 1536: 321 MB read for 302 MB
// of weights at 4.8 TB/s, against 444 MB of the 128-row form), the tensor pipe at the clock that the power cap leaves in
// prefill.  moe_form_us in flyb200_moe.cu lists the times of both forms.
//
// A tile starts at every (256 / tile_m)-th routing block of an expert's run of blocks.  One warp finds these in
// expert_ids before the mainloop and leaves them in shared memory, so that any item can be looked up.
#pragma once
#include "moe_kernel.cuh"
#include "rows2_kernel.cuh"

namespace flyb200 {

constexpr int MOE_PAIR_STAGES = 6;
constexpr int MOE_PAIR_MAX_BLOCKS = 7168;  // routing blocks whose tiles fit the list (two bytes each)
constexpr int MOE_PAIR_GROUP = 16;         // tiles per rasterisation group (at most 4096 rows of activations)
struct MoePairSmem {
  static constexpr int OPERAND = BLOCK_ROWS * KBLOCK_BYTES;  // this CTA's rows, or its weight tile
  static constexpr int OFF_A = 0;
  static constexpr int OFF_B = OFF_A + MOE_PAIR_STAGES * OPERAND;
  static constexpr int OFF_C = OFF_B + MOE_PAIR_STAGES * OPERAND;     // 8 warps x one store stage
  static constexpr int OFF_SW = OFF_C + 8 * STORE_STAGE;              // 1024 weight scales
  static constexpr int OFF_LIST = OFF_SW + 8 * BLOCK_ROWS * 4;        // first routing block of every tile
  static constexpr int OFF_BAR = OFF_LIST + MOE_PAIR_MAX_BLOCKS * 2;  // full[S], empty[S], tfull[2], tempty[2]
  static constexpr int OFF_MISC = OFF_BAR + 8 * (2 * MOE_PAIR_STAGES + 4);
  static constexpr int TOTAL = OFF_MISC + 16;
};
static_assert(MoePairSmem::TOTAL <= 232448, "227 KiB of shared memory per CTA");

// Boxes of 128, 64 and 32 weight rows: whole tiles, and strips of the last round.
struct MoePairWeights {
  CUtensorMap box[3];
};

// Executed by one warp: the first routing blocks of all tiles, in order; returns their number.  `blocks` blocks of
// which `per` make a tile; blocks without an expert belong to none.
__device__ __forceinline__ int moe_pair_tile_list(const int* expert_ids, int experts, int blocks, int per, uint16_t* list, int lane) {
  int count = 0, run = 0, before = -1;  // tiles so far, first block of the current run, expert of the block before
  for (int b0 = 0; b0 < blocks; b0 += 128) {
    int e[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) e[i] = b0 + 32 * i + lane < blocks ? __ldg(expert_ids + b0 + 32 * i + lane) : -1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int b = b0 + 32 * i + lane;
      int prev = __shfl_up_sync(0xffffffffu, e[i], 1);
      if (lane == 0) prev = before;
      const uint32_t starts = __ballot_sync(0xffffffffu, b == 0 || e[i] != prev);
      const uint32_t upto = starts & (0xffffffffu >> (31 - lane));
      const int first = upto != 0 ? b0 + 32 * i + 31 - __clz(upto) : run;
      const bool tile = e[i] >= 0 && e[i] < experts && b < blocks && (b - first) % per == 0;
      const uint32_t tiles = __ballot_sync(0xffffffffu, tile);
      if (tile) list[count + __popc(tiles & ((1u << lane) - 1u))] = static_cast<uint16_t>(b);
      count += __popc(tiles);
      if (starts != 0) run = b0 + 32 * i + 31 - __clz(starts);
      before = __shfl_sync(0xffffffffu, e[i], 31);
    }
  }
  return count;
}

// Column strips of the items of the last, partial round: the number (1, 2 or 4) that makes it shortest.  A strip takes the
// tensor pipe 512 / strips cycles per k-block, or its operands at 72 bytes per cycle.
__device__ __forceinline__ int moe_pair_strips(int items, int clusters) {
  const int rest = items % clusters;
  if (items < clusters || rest == 0) return 1;
  const int two = (2 * rest + clusters - 1) / clusters * 341, four = (4 * rest + clusters - 1) / clusters * 284;
  return four < two && four < 512 ? 4 : two < 512 ? 2 : 1;
}

template <int KIND, int STAGE, int OUTMODE, bool ACCUM>
__global__ void __launch_bounds__(moe_rows_threads(STAGE), 1)
moe_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ MoePairWeights tmW, const MoeParams p) {
  static_assert(STAGE == 2 || !ACCUM, "only the down projection accumulates");
  using L = MoePairSmem;
  using KT = KindTraits<KIND>;
  constexpr int STAGES = MOE_PAIR_STAGES;
  constexpr int BN = MOE_ROWS_BN;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t smem_base = smem_u32(smem_raw);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_raw + L::OFF_MISC + 4);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + L::OFF_MISC);
  int* tile_count = reinterpret_cast<int*>(smem_raw + L::OFF_MISC + 12);
  uint16_t* list = reinterpret_cast<uint16_t*>(smem_raw + L::OFF_LIST);
  const int warp = threadIdx.x >> 5;
  const int role = warp_index();  // for the loops that issue
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_rank());  // 0 = leader
  const uint32_t bar_full = smem_base + L::OFF_BAR;
  const uint32_t bar_empty = bar_full + 8 * STAGES;
  const uint32_t bar_tfull = bar_empty + 8 * STAGES;
  const uint32_t bar_tempty = bar_tfull + 16;

  if ((smem_base & 1023u) != 0) {  // same answer in every CTA of the grid
    if (threadIdx.x == 0) atomicCAS(p.status, 0, ST_SMEM_ALIGN);
    return;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar_full + 8 * s, 1);   // leader: its own expect_tx arrival; bytes come from both CTAs
      mbar_init(bar_empty + 8 * s, 1);  // one tcgen05.commit from the leader
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_tfull + 8 * s, 1);
      mbar_init(bar_tempty + 8 * s, 2 * moe_rows_epilogue_warps(STAGE));  // both CTAs' warps (used in the leader only)
    }
    abort_flag[0] = 0;
    abort_flag[1] = 0;
    fence_mbar_init();
    prefetch_tensormap(&tmA);
    prefetch_tensormap(&tmW.box[0]);
  }
  constexpr uint32_t TMEM_COLS = 512;
  if (warp == 1) {
    tmem_alloc_2sm(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish_2sm();
  }
  // Launched as a programmatic dependent: what the kernel before it writes is touched only after the wait.  After a gather
  // pass (p.pdl) that is everything but the routing table, which then comes from a kernel further back.
  const int* num_valid = p.num_valid;
  const int* expert_ids = p.expert_ids;
  if (!p.pdl) pdl_wait(num_valid, expert_ids);
  const int n_rows = __ldg(num_valid);
  const int per = PAIR_ROWS / p.tile_m;  // routing blocks of a tile
  if (warp == 2) {
    const int n = moe_pair_tile_list(expert_ids, p.experts, min((n_rows + p.tile_m - 1) / p.tile_m, MOE_PAIR_MAX_BLOCKS), per, list, lane);
    if (lane == 0) *tile_count = n;
  }
  if (p.pdl) pdl_wait<>();
  tc_fence_before();
  cluster_barrier_all();  // barriers of both CTAs initialised, TMEM of the pair allocated, tiles listed
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // Work items: (tile, channel pair), tiles fastest, in groups whose activation rows stay in L2 while the group walks all
  // channel pairs; clusters working side by side share the weight tiles of an expert.  Those of the last, partial round
  // go in column strips.
  const int tiles = *tile_count;
  const int pairs = STAGE == 1 ? (p.n_out + BLOCK_ROWS - 1) / BLOCK_ROWS : (p.n_out + BN - 1) / BN;
  const int num_kb = p.K_bytes / KBLOCK_BYTES;
  const int first_item = static_cast<int>(cluster_id_x());
  const int step = static_cast<int>(num_clusters_x());
  const int strips = moe_pair_strips(tiles * pairs, step);
  const int whole = strips > 1 ? tiles * pairs - tiles * pairs % step : tiles * pairs;
  const int items = whole + (tiles * pairs - whole) * strips;
  struct Item {
    int expert, row0, rows;  // first sorted row and number of rows (at most 256)
    int pair, c0, width;     // channel pair, first channel and number of channels of each of its tiles
  };
  auto item_of = [&](int t) {
    Item it;
    const bool cut = t >= whole;
    const int u = cut ? whole + (t - whole) / strips : t;
    it.width = cut ? BLOCK_ROWS / strips : BLOCK_ROWS;
    it.c0 = cut ? (t - whole) % strips * it.width : 0;
    const int per_group = MOE_PAIR_GROUP * pairs;
    const int g = u / per_group;
    const int first = g * MOE_PAIR_GROUP;
    const int gm = min(MOE_PAIR_GROUP, tiles - first);
    const int r = u - g * per_group;
    it.pair = r / gm;
    const int b = list[first + r % gm];
    it.expert = __ldg(expert_ids + b);
    it.row0 = b * p.tile_m;
    it.rows = p.tile_m;
    for (int i = 1; i < per; ++i) {
      const int next = it.row0 + i * p.tile_m;
      if (it.rows == i * p.tile_m && next < n_rows && __ldg(expert_ids + b + i) == it.expert) it.rows += p.tile_m;
    }
    it.rows = min(it.rows, n_rows - it.row0);
    return it;
  };

  if (role == 0) {
    // ---------------- producer (both CTAs): own rows, own weight tile ----------------
    const bool issuer = elect_one();
    const uint64_t pol = l2_policy_evict_last();
    // weights that a tile or two read leave L2 first: 800 tokens x top-4, 32 experts, 3072 x 1536 83.5 -> 79.6 us
    const uint64_t pol_w = tiles <= 2 * p.experts ? l2_policy_evict_first() : pol;
    const uint32_t full_leader = mapa_u32(bar_full, 0);
    int stage = 0;
    uint32_t phase = 0;
    int issued = 0;
    bool ok = true;
    for (int t = first_item; t < items && ok; t += step) {
      const Item it = item_of(t);
      int w_row[2], n_valid[2];
      moe_pair_tiles<STAGE>(p, it.pair, w_row, n_valid);
      const int expert = __shfl_sync(0xffffffffu, it.expert, 0);
      const int row0 = __shfl_sync(0xffffffffu, it.row0, 0) + rank * BLOCK_ROWS;
      const bool second = __shfl_sync(0xffffffffu, it.rows, 0) > BLOCK_ROWS;  // else the follower has no rows: whatever its ring holds
      const bool load_a = rank == 0 || second;
      const int width = it.width;
      const int w0 = (rank == 0 ? w_row[0] : w_row[1]) + it.c0;
      const CUtensorMap* mapW = &tmW.box[width == BLOCK_ROWS ? 0 : width == 64 ? 1 : 2];
      // the boxes count in full where they reach past the last row
      const uint32_t bytes = static_cast<uint32_t>((second ? 2 : 1) * BLOCK_ROWS + 2 * width) * KBLOCK_BYTES;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait_warp(bar_empty + 8 * stage, phase ^ 1u, abort_flag)) {
          report_failure(p.status, ST_TIMEOUT, abort_flag);
          ok = false;
          break;
        }
        if (issuer) {
          if (rank == 0) mbar_expect_tx(bar_full + 8 * stage, bytes);
          if (load_a) tma_load_2d_2sm(smem_base + L::OFF_A + stage * L::OPERAND, &tmA, full_leader + 8 * stage, kb * KBLOCK_BYTES, row0, pol);
          tma_load_3d_2sm(smem_base + L::OFF_B + stage * L::OPERAND, mapW, full_leader + 8 * stage, 0, w0, expert * num_kb + kb, pol_w);
        }
        ++issued;
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    pdl_trigger();  // the last loads are on their way: the next kernel may be scheduled as the CTAs finish
    if (!ok || *abort_flag) {
      // Wait (bounded) for the copies in flight.  The leader's barriers count the bytes of both CTAs; the follower
      // cannot wait on them and gives its own copies a millisecond.
      const int pending = rank == 0 ? min(issued, STAGES) : 0;
      for (int i = 0; i < pending; ++i) {
        int s = stage - 1 - i;
        uint32_t ph = phase;
        if (s < 0) {
          s += STAGES;
          ph ^= 1u;
        }
        mbar_wait(bar_full + 8 * s, ph, abort_flag + 1);
      }
      if (rank != 0) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 1000000) __nanosleep(1000);
      }
    }
    __syncwarp();
  } else if (role == 1) {
    // ---------------- MMA issue (leader only) ----------------
    if (rank == 0) {
      const bool issuer = elect_one();
      const uint64_t adesc0 = umma_desc_sw128_kmajor(smem_base + L::OFF_A), bdesc0 = umma_desc_sw128_kmajor(smem_base + L::OFF_B);
      const uint32_t peer_empty = mapa_u32(bar_empty, 1), peer_tfull = mapa_u32(bar_tfull, 1);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int t = first_item; t < items && ok; t += step) {
        if (!mbar_wait_warp(bar_tempty + 8 * acc, acc_phase ^ 1u, abort_flag)) {
          report_failure(p.status, ST_TIMEOUT, abort_flag);
          break;
        }
        tc_fence_after();
        const uint32_t idesc = umma_idesc(KT::dfmt, KT::abfmt, PAIR_ROWS, t < whole ? BN : BN / strips);
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_warp(bar_full + 8 * stage, phase, abort_flag)) {
            report_failure(p.status, ST_TIMEOUT, abort_flag);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t adesc = adesc0 + static_cast<uint32_t>(stage * (L::OPERAND >> 4));
          const uint64_t bdesc = bdesc0 + static_cast<uint32_t>(stage * (L::OPERAND >> 4));
          if (issuer) {
            umma_ss_2sm<KIND>(d_tmem, adesc, bdesc, idesc, kb != 0 ? 1u : 0u);
#pragma unroll
            for (int k = 1; k < KBLOCK_BYTES / UMMA_K_BYTES; ++k)
              umma_ss_2sm<KIND>(d_tmem, adesc + static_cast<uint64_t>(k * (UMMA_K_BYTES >> 4)),
                                bdesc + static_cast<uint64_t>(k * (UMMA_K_BYTES >> 4)), idesc, 1u);
            umma_commit_2sm(bar_empty + 8 * stage);
            umma_commit_2sm(peer_empty + 8 * stage);
            if (kb == num_kb - 1) {
              umma_commit_2sm(bar_tfull + 8 * acc);
              umma_commit_2sm(peer_tfull + 8 * acc);
            }
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue (both CTAs): own 128 rows ----------------
    const int q = warp & 3;  // TMEM lane quadrant this warp may read
    MoeRowsEpilogue<KIND, STAGE, OUTMODE, ACCUM> ep{p, reinterpret_cast<float*>(smem_raw + L::OFF_SW) + (warp - 2) * moe_rows_scales(STAGE),
                                                    smem_base + L::OFF_C + (warp - 2) * STORE_STAGE, (warp - 2) >> 2, lane};
    auto fetch = [&](int t) {
      if (t >= items) return;
      const Item it = item_of(t);
      const int trow = rank * BLOCK_ROWS + q * 32 + lane;  // this thread's row of the tile
      ep.fetch(it.expert, it.row0 + trow, trow < it.rows, it.pair, it.c0, it.width);
    };
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    fetch(first_item);
    for (int t = first_item; t < items && ok; t += step) {
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * BN);
      const uint32_t tempty_leader = mapa_u32(bar_tempty + 8 * acc, 0);
      ok = ep.run(t_row, [&]() { fetch(t + step); }, [&]() { return mbar_wait(bar_tfull + 8 * acc, acc_phase, abort_flag); },
                  [&]() { mbar_arrive_cluster(tempty_leader); });
      if (!ok && lane == 0) report_failure(p.status, ST_TIMEOUT, abort_flag);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
    __syncwarp();
  }

  // Nobody leaves while the peer may still signal one of its barriers or the leader's MMAs may still read its shared
  // memory.  All waits above are bounded, so every thread of both CTAs arrives here.
  tc_fence_before();
  cluster_barrier_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_2sm(tmem_base, TMEM_COLS);
  }
}

}  // namespace flyb200
