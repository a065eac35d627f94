// Large-M kernel, pair form: a cluster of two CTAs owns a tile of 256 rows x bn columns and drives it with
// tcgen05.mma.cta_group::2 (UMMA M = 256, N = bn).  CTA r of the pair holds rows [128 r, 128 r + 128): per k-block it
// loads those rows of A (16 KiB) and half of the tile's weight rows (16 KiB at bn = 256; the 128-row form takes 48 KiB
// for the same product), keeps a 128 x bn accumulator in its own TMEM and stores its own rows of C.  Only the leader
// CTA issues MMAs.  Two accumulators: the epilogue of a tile overlaps the mainloop of the next.
//
// What bounds it: the board's power.  A k-block of a 256 x 256 tile takes 523..540 cycles of the 512 that its four
// MMAs need, at the 1.1..1.3 GHz the 1 kW cap leaves; fewer bytes moved per product are a higher clock.  Next to the
// 128-row form it is 4..17 % faster where it is the choice (large_form in flyb200.cu lists both), in turn on one GPU fp8 16384 x 57344 x 8192
// 5926 us against 6170, 8192 x 28672 x 8192 1476 against 1554, 16384 x 8192 x 8192 867 against 903; bf16 8192 x 8192 x 8192 777..820
// against 847 (cuBLAS 786).  Tiles of 512 rows (half of the weight traffic again, all of TMEM in one tile) were built and
// were slower, 1454 against 1412 us on fp8 8192 x 28672 x 8192, as nothing overlaps their epilogue.
//
// Cross-CTA signalling, all without multicast:
//   * both CTAs' TMA loads complete their bytes on the LEADER's full barrier
//     (the .cta_group::2 form of the load allows the barrier to live in the
//     peer CTA);
//   * the leader frees a stage / publishes an accumulator with two
//     tcgen05.commit, one per CTA's barrier;
//   * the follower's epilogue warps hand the accumulator back with a remote
//     mbarrier.arrive on the leader's barrier.
#pragma once
#include "gemm_kernels.cuh"

namespace flyb200 {

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_id_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t num_clusters_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t mapa_u32(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_barrier_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// arrive on an mbarrier that may live in the peer CTA (shared::cluster address)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_alloc_2sm(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_2sm() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_2sm(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// TMA loads whose completion bytes are credited to a barrier given as a
// shared::cluster address (the leader's), no multicast.
__device__ __forceinline__ void tma_load_2d_2sm(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster, int x, int y,
                                                uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(dst),
      "l"(map), "r"(bar_cluster), "r"(x), "r"(y), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_2sm(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster, int x, int y,
                                                int z, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4, %5}], [%2], %6;" ::"r"(dst),
      "l"(map), "r"(bar_cluster), "r"(x), "r"(y), "r"(z), "l"(policy)
      : "memory");
}
template <int KIND>
__device__ __forceinline__ void umma_ss_2sm(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  if constexpr (KIND == KIND_F8) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  } else if constexpr (KIND == KIND_I8) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}
// completion of all MMAs issued so far by this thread -> one arrival on the
// barrier at `bar_cluster` (own CTA or the peer)
__device__ __forceinline__ void umma_commit_2sm(uint32_t bar_cluster) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster)
               : "memory");
}

constexpr int PAIR_ROWS = 2 * BLOCK_ROWS;  // rows of a pair's tile (UMMA M)

// Shared-memory carve-up of one CTA for a tile width and a ring depth (identical on host and device).
__host__ __device__ inline RowsLayout pair_layout(int bn, int stages) {
  RowsLayout l;
  l.a_stage = BLOCK_ROWS * KBLOCK_BYTES;  // this CTA's rows of A
  l.b_stage = bn / 2 * KBLOCK_BYTES;      // this CTA's half of the tile's weight rows
  l.off_b = stages * l.a_stage;
  l.off_c = l.off_b + stages * l.b_stage;  // eight buffers: one per epilogue warp, or two for each of four
  l.off_bar = l.off_c + 8 * ROWS_C_BUF;    // full[S], empty[S], tfull[2], tempty[2]
  l.off_misc = l.off_bar + 8 * (2 * stages + 4);
  l.total = l.off_misc + 16;
  return l;
}

struct PairMaps {
  CUtensorMap a;
  CUtensorMap w, w_strip;  // boxes of a CTA's weight rows: of a whole tile, and of a column strip
  CUtensorMap c;
};

template <int KIND, int OUTMODE>
__global__ void __launch_bounds__(ROWS_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ PairMaps maps, const GemmParams p) {
  using KT = KindTraits<KIND>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t smem_base = smem_u32(smem_raw);
  const int BN = p.bn;
  const int STAGES = p.rows_stages;
  const RowsLayout L = pair_layout(BN, STAGES);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_raw + L.off_misc + 4);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + L.off_misc);

  const int warp = threadIdx.x >> 5;
  const int role = warp_index();  // for the loops that issue
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();  // 0 = leader
  const uint32_t bar_full = smem_base + L.off_bar;
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
      mbar_init(bar_tfull + 8 * s, 1);                              // one tcgen05.commit from the leader
      mbar_init(bar_tempty + 8 * s, 2 * ((blockDim.x - 64) >> 5));  // every epilogue warp of both CTAs (used in the leader only)
    }
    abort_flag[0] = 0;
    abort_flag[1] = 0;  // stays zero: lets the drain below wait on time alone
    fence_mbar_init();
    prefetch_tensormap(&maps.a);
    prefetch_tensormap(&maps.w);
    if (OUTMODE != OUT_RAW32) prefetch_tensormap(&maps.c);
  }
  constexpr uint32_t TMEM_COLS = 512;
  if (warp == 1) {
    tmem_alloc_2sm(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish_2sm();
  }
  tc_fence_before();
  cluster_barrier_all();  // barriers of both CTAs initialised, TMEM of the pair allocated
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (p.pdl) {  // no global memory is read or written before this
    asm volatile("griddepcontrol.wait;" ::: "memory");
    pdl_trigger();
  }

  const int num_m = (p.M + PAIR_ROWS - 1) / PAIR_ROWS;
  const int num_n = (p.N + BN - 1) / BN;
  const int num_tiles = num_m * num_n;
  const int num_kb = p.K_bytes / KBLOCK_BYTES;
  const int gm_full = p.group_m;
  const int first_item = static_cast<int>(cluster_id_x());
  const int step = static_cast<int>(num_clusters_x());

  // Groups of row tiles; the row tile changes fastest, every second group walks the channels backwards.
  auto tile_coords = [&](int t, int& m_blk, int& n_blk) {
    const int per_group = gm_full * num_n;
    const int g = t / per_group;
    const int first_m = g * gm_full;
    const int gm = min(gm_full, num_m - first_m);
    const int r = t - g * per_group;
    m_blk = first_m + r % gm;
    n_blk = r / gm;
    if (g & 1) n_blk = num_n - 1 - n_blk;
  };

  // Work items: the tiles of the whole rounds, then those of the last, partial round in `parts` column strips
  // each (host: pair_tail_parts).
  const int parts = p.tail_parts;
  const int whole = parts > 1 ? num_tiles - num_tiles % step : num_tiles;
  const int items = whole + (num_tiles - whole) * parts;
  const int strip = BN / parts;
  // item -> first row of the pair, first column and width; false where the strip lies past the last column
  auto item_coords = [&](int i, int& m0, int& n0, int& width) {
    int m_blk, n_blk;
    const int j = i - whole;
    tile_coords(j < 0 ? i : whole + j / parts, m_blk, n_blk);
    m0 = m_blk * PAIR_ROWS;
    n0 = n_blk * BN + (j < 0 ? 0 : j % parts * strip);
    width = j < 0 ? BN : strip;
    return n0 < p.N;
  };

  if (role == 0) {
    // ---------------- producer (both CTAs): own A rows, own half of the weight rows ----------------
    // The whole warp runs the loop and one lane issues, as in the MMA warp.
    const bool issuer = elect_one();
    const uint64_t pol = l2_policy_evict_last();
    const uint32_t full_leader = mapa_u32(bar_full, 0);
    int stage = 0;
    uint32_t phase = 0;
    int issued = 0;
    bool ok = true;
    for (int t = first_item; t < items && ok; t += step) {
      int m0, n0, width;
      if (!item_coords(t, m0, n0, width)) continue;
      m0 += static_cast<int>(rank) * BLOCK_ROWS;
      n0 += static_cast<int>(rank) * (width / 2);
      // the boxes count in full where they reach past the last row
      const uint32_t bytes = 2 * static_cast<uint32_t>(BLOCK_ROWS + width / 2) * KBLOCK_BYTES;
      // One box per operand: with the weight rows in two boxes of 64 the kernel took 780 instead of 690 cycles per k-block.
      const CUtensorMap* mapW = width == BN ? &maps.w : &maps.w_strip;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait_warp(bar_empty + 8 * stage, phase ^ 1u, abort_flag)) {
          report_failure(p.status, ST_TIMEOUT, abort_flag);
          ok = false;
          break;
        }
        if (issuer) {
          if (rank == 0) mbar_expect_tx(bar_full + 8 * stage, bytes);
          tma_load_2d_2sm(smem_base + stage * L.a_stage, &maps.a, full_leader + 8 * stage, kb * KBLOCK_BYTES, m0, pol);
          tma_load_3d_2sm(smem_base + L.off_b + stage * L.b_stage, mapW, full_leader + 8 * stage, 0, n0, kb, pol);
        }
        ++issued;
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (lane == 0) {
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
    }
    __syncwarp();
  } else if (role == 1) {
    // ---------------- MMA issue (leader only) ----------------
    // The whole warp runs the loop and one lane issues, so that addresses and descriptors stay uniform over the warp; the
    // same loop in one thread took 779 cycles per k-block, this way 537 (bf16 8192 x 8192 x 8192).
    if (rank == 0) {
      const bool issuer = elect_one();
      const uint64_t adesc0 = umma_desc_sw128_kmajor(smem_base);
      const uint64_t bdesc0 = umma_desc_sw128_kmajor(smem_base + L.off_b);
      const uint32_t peer_empty = mapa_u32(bar_empty, 1), peer_tfull = mapa_u32(bar_tfull, 1);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int t = first_item; t < items && ok; t += step) {
        int m0, n0, width;
        if (!item_coords(t, m0, n0, width)) continue;
        const uint32_t idesc = umma_idesc(KT::dfmt, KT::abfmt, PAIR_ROWS, static_cast<uint32_t>(width));
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * ROWS_ACC_COLS);
        if (!mbar_wait_warp(bar_tempty + 8 * acc, acc_phase ^ 1u, abort_flag)) {
          report_failure(p.status, ST_TIMEOUT, abort_flag);
          break;
        }
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_warp(bar_full + 8 * stage, phase, abort_flag)) {
            report_failure(p.status, ST_TIMEOUT, abort_flag);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t adesc = adesc0 + static_cast<uint32_t>(stage * (L.a_stage >> 4));
          const uint64_t bdesc = bdesc0 + static_cast<uint32_t>(stage * (L.b_stage >> 4));
          if (issuer) {
            umma_ss_2sm<KIND>(d_tmem, adesc, bdesc, idesc, kb != 0 ? 1u : 0u);
#pragma unroll
            for (int k = 1; k < KBLOCK_BYTES / UMMA_K_BYTES; ++k)
              umma_ss_2sm<KIND>(d_tmem, adesc + static_cast<uint64_t>(k * (UMMA_K_BYTES >> 4)),
                                bdesc + static_cast<uint64_t>(k * (UMMA_K_BYTES >> 4)), idesc, 1u);
            // the stage is free in both CTAs once these MMAs have read it
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
    const int q = warp & 3;
    const int ew = warp - 2;
    const int share = (static_cast<int>(blockDim.x) - 64) >> 7;  // epilogue warps per 32 rows (host: rows_epilogue_warps)
    const int cbufs = 2 / share;
    const uint32_t stage_c = smem_base + L.off_c + ew * cbufs * ROWS_C_BUF;
    int acc = 0;
    uint32_t acc_phase = 0;
    int cbuf = 0;
    for (int t = first_item; t < items; t += step) {
      int m0, n0, width;
      if (!item_coords(t, m0, n0, width)) continue;
      m0 += static_cast<int>(rank) * BLOCK_ROWS + q * 32;
      if (!mbar_wait(bar_tfull + 8 * acc, acc_phase, abort_flag)) {
        if (lane == 0) report_failure(p.status, ST_TIMEOUT, abort_flag);
        break;
      }
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * ROWS_ACC_COLS);
      const uint32_t tempty_leader = mapa_u32(bar_tempty + 8 * acc, 0);
      epilogue_warp_tile<KIND, OUTMODE>(p, &maps.c, 1, 0, t_row, m0, n0, width, lane, stage_c, cbuf, [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(tempty_leader);
      }, cbufs, share, ew >> 2);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
    if (lane == 0) bulk_wait_group<0>();
    __syncwarp();
  }

  // Nobody leaves while the peer may still signal one of its barriers or the
  // leader's MMAs may still read its shared memory.  All waits above are
  // bounded, so every thread of both CTAs arrives here.
  tc_fence_before();
  cluster_barrier_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_2sm(tmem_base, TMEM_COLS);
  }
}

}  // namespace flyb200
