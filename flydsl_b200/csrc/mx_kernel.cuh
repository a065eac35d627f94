// MXFP8 GEMM: E4M3 codes with one E8M0 (power-of-two) scale per 32 elements
// of K on BOTH operands, multiplied with the block-scaled tensor-core
// instruction
//
//   tcgen05.mma.kind::mxf8f6f4.block_scale   D[tmem] (+)= (A . sfA) x (B . sfB)^T
//
// which reads the scale factors from tensor memory.  c[M, N] = bf16/fp16 of
// sum_k a[m, k] 2^(sa[m, k/32] - 127) w[n, k] 2^(sw[n, k/32] - 127).
//
// Data layout.  Codes: activations row-major [M, K]; weights in the same
// preshuffled image as the per-channel-scaled GEMM ([K/128][N][128 B swizzled]).
// Scales: "scale image" [K/128][rows/128][512 B]: one 512-byte atom per 128 rows
// and 128-element k-block, byte (r % 32) * 16 + (r / 32) * 4 + j = scale of row r
// of the tile for the j-th 32-element block.  An atom is what one
// tcgen05.cp.32x128b.warpx4 moves from shared memory into four TMEM columns
// (lane r % 32 of every 32-lane quarter, column r / 32, byte j), the arrangement
// the instruction expects; j is selected per instruction by the scale-factor id
// fields of the instruction descriptor.
//
// Kernel: persistent, tokens on the UMMA M side (128 per tile), BN output
// channels on the N side, a ring of {A tile, W tile, scale atom of A, scale
// atoms of W}, a rotating set of TMEM columns for the scale atoms of the stages
// in flight.  Two shapes: BN = 128 with two TMEM accumulators (the epilogue of
// tile i overlaps the mainloop of tile i + 1; 6 stages), and BN = 256 with one
// accumulator (the wider MMA needs fewer operand bytes per flop, but 2 x 256
// accumulator columns plus scale columns exceed the 512 columns of TMEM, so the
// epilogue is exposed; 4 stages) for long K, where the epilogue is a small part
// of a tile.  Threads as in the large-M kernel: warp 0 producer, warp 1 MMA
// (copies the two scale atoms to TMEM, then issues the four MMAs of a k-block),
// warps 2..9 epilogue (thread = token row, two warps per 32 rows; stores turned in shared memory, store_rows32).
//
// SPLIT: where the 128 x 128 tiles leave at least half of the SMs idle, a cluster of two, four or eight
// CTAs shares a tile, each with a part of K.  Every CTA parks its fp32 partial tile in its shared memory
// and, after a cluster barrier, sums a share of the columns over the peers in rank order (deterministic).
// Bound by the k-blocks a CTA walks (0.36 us each at 6 stages) plus about 5 us of launch, reduction and
// exit; a workspace and a second kernel would add a launch to that.  Measured, see mx_split.
#pragma once
#include "moe_kernel.cuh"

namespace flyb200 {


constexpr int MX_THREADS = 64 + 8 * 32;  // producer, MMA issuer, eight epilogue warps

struct MxParams {
  const uint8_t* w;    // weight codes, preshuffled image
  const uint8_t* sfa;  // scale image of the activations, [K/128][ceil(M/128)][512]
  const uint8_t* sfw;  // scale image of the weights, [K/128][N/128][512]
  void* c;
  int M, N, K_bytes;
  int group_m;
  int split;           // SPLIT: CTAs per cluster, K parts of a tile
  uint32_t fmt_bits;   // operand formats of kind::mxf8f6f4 as instruction-descriptor bits: (A format << 7) | (B format << 10)
  int* status;
};

// FP4: the codes are E2M1, two per byte.  A 128-byte k-block then holds 256
// elements = eight scale blocks per row: two scale atoms per 128 rows instead of
// one (atom h covers elements [128 h, 128 h + 128) of the k-block), everything
// else - operand tiles, ring, swizzle - is the same bytes as for 8-bit codes.
template <int BN, bool FP4 = false>
struct MxSmem {
  static constexpr int STAGES = BN == 128 ? 6 : 4;
  static constexpr int NACC = BN == 128 ? 2 : 1;          // TMEM accumulators
  static constexpr int HALVES = FP4 ? 2 : 1;              // scale atoms per 128 rows and k-block
  static constexpr int SFB_ATOMS = BN / 128;
  static constexpr int A_STAGE = BLOCK_ROWS * KBLOCK_BYTES;
  static constexpr int B_STAGE = BN * KBLOCK_BYTES;
  static constexpr int SFA_STAGE = HALVES * MX_SF_ATOM;
  static constexpr int SFB_HALF = SFB_ATOMS * MX_SF_ATOM;
  static constexpr int SFB_STAGE = HALVES * SFB_HALF;
  static constexpr int OFF_A = 0;
  static constexpr int OFF_B = OFF_A + STAGES * A_STAGE;
  static constexpr int OFF_SFA = OFF_B + STAGES * B_STAGE;
  static constexpr int OFF_SFB = OFF_SFA + STAGES * SFA_STAGE;
  static constexpr int OFF_C = OFF_SFB + STAGES * SFB_STAGE;    // 8 warps x one store stage
  static constexpr int OFF_BAR = OFF_C + 8 * STORE_STAGE;       // full[S], empty[S], tfull[2], tempty[2]
  static constexpr int OFF_MISC = OFF_BAR + 8 * (2 * STAGES + 4);
  static constexpr int TOTAL = OFF_MISC + 16;
};

template <int OUTMODE, int BN, bool FP4 = false, bool SPLIT = false>
__global__ void __launch_bounds__(MX_THREADS, 1) mx_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const MxParams p) {
  using L = MxSmem<BN, FP4>;
  constexpr int STAGES = L::STAGES;
  constexpr int NACC = L::NACC;
  constexpr int HALVES = L::HALVES;
  // TMEM columns of the scale atoms of one stage: per half, 4 for A then 4 per 128 channels for W
  constexpr int SFA_COLS = 4 * HALVES;
  constexpr int SF_COLS = SFA_COLS + 4 * L::SFB_ATOMS * HALVES;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t smem_base = smem_u32(smem_raw);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_raw + L::OFF_MISC + 4);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + L::OFF_MISC);
  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const uint32_t bar_full = smem_base + L::OFF_BAR;
  const uint32_t bar_empty = bar_full + 8 * STAGES;
  const uint32_t bar_tfull = bar_empty + 8 * STAGES;
  const uint32_t bar_tempty = bar_tfull + 16;

  if ((smem_base & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(p.status, 0, ST_SMEM_ALIGN);
    return;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_tfull + 8 * s, 1);
      mbar_init(bar_tempty + 8 * s, 8);
    }
    abort_flag[0] = 0;
    abort_flag[1] = 0;
    fence_mbar_init();
    prefetch_tensormap(&tmA);
  }
  // TMEM: columns [0, 256) the accumulator(s), then per stage in flight the scale
  // atoms (4 columns for A, 4 per 128 channels for W)
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t SF_COL0 = NACC * BN;
  static_assert(SF_COL0 + STAGES * SF_COLS <= TMEM_COLS, "accumulators and scale columns must fit TMEM");
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait<>();  // launched as a programmatic dependent: nothing in global memory is touched before this

  const int num_m = (p.M + BLOCK_ROWS - 1) / BLOCK_ROWS;
  const int num_n = p.N / BN;
  const int num_tiles = num_m * num_n;
  const int all_kb = p.K_bytes / KBLOCK_BYTES;
  // this CTA's k-blocks, first tile and step to the next one (SPLIT: one tile per cluster)
  const int rank = SPLIT ? static_cast<int>(cluster_ctarank()) : 0;
  const int kb0 = SPLIT ? rank * all_kb / p.split : 0;
  const int kb1 = SPLIT ? (rank + 1) * all_kb / p.split : all_kb;
  const int tile0 = SPLIT ? static_cast<int>(blockIdx.x) / p.split : static_cast<int>(blockIdx.x);
  const int tile_step = SPLIT ? num_tiles : static_cast<int>(gridDim.x);
  auto tile_coords = [&](int t, int& m_blk, int& n_blk) {
    const int per_group = p.group_m * num_n;
    const int g = t / per_group;
    const int first_m = g * p.group_m;
    const int gm = min(p.group_m, num_m - first_m);
    const int r = t - g * per_group;
    m_blk = first_m + r % gm;
    n_blk = r / gm;
  };

  if (warp == 0) {
    // ------------------------------ producer ------------------------------
    // The whole warp runs the loop, here and in the MMA warp, and one lane issues (ptx.cuh).  By themselves the issuing
    // threads bound this kernel, eleven instructions per k-block in the MMA loop: one lane / whole warp, us, MXFP8 384 x 4096 x 14336
    // 41.6 / 31.7, 256 x 8192 x 8192 26.4 / 20.1, MXFP4 1024 x 8192 x 8192 36.4 / 29.4, 384 x 4096 x 14336 24.8 / 17.4, MXFP6 256 x 8192 x 8192 26.2 / 20.0.
    const bool issuer = elect_one();
    const uint64_t pol = l2_policy_evict_last();
    int stage = 0;
    uint32_t phase = 0;
    int issued = 0;
    bool ok = true;
    for (int t = tile0; t < num_tiles && ok; t += tile_step) {
      int m_blk, n_blk;
      tile_coords(t, m_blk, n_blk);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_warp(bar_empty + 8 * stage, phase ^ 1u, abort_flag)) {
          report_failure(p.status, ST_TIMEOUT, abort_flag);
          ok = false;
          break;
        }
        const uint32_t fb = bar_full + 8 * stage;
        if (issuer) {
          mbar_expect_tx(fb, L::A_STAGE + L::B_STAGE + L::SFA_STAGE + L::SFB_STAGE);
          tma_load_2d(smem_base + L::OFF_A + stage * L::A_STAGE, &tmA, fb, kb * KBLOCK_BYTES, m_blk * BLOCK_ROWS, pol);
          bulk_load_1d(smem_base + L::OFF_B + stage * L::B_STAGE,
                       p.w + (static_cast<size_t>(kb) * p.N + n_blk * BN) * KBLOCK_BYTES, L::B_STAGE, fb, pol);
          // the scale images are indexed by 128-ELEMENT k-blocks: HALVES of them per 128-byte k-block
#pragma unroll
          for (int h = 0; h < HALVES; ++h) {
            const size_t ekb = static_cast<size_t>(kb) * HALVES + h;
            bulk_load_1d(smem_base + L::OFF_SFA + stage * L::SFA_STAGE + h * MX_SF_ATOM,
                         p.sfa + (ekb * num_m + m_blk) * MX_SF_ATOM, MX_SF_ATOM, fb, pol);
            bulk_load_1d(smem_base + L::OFF_SFB + stage * L::SFB_STAGE + h * L::SFB_HALF,
                         p.sfw + (ekb * (p.N / 128) + n_blk * L::SFB_ATOMS) * MX_SF_ATOM, L::SFB_HALF, fb, pol);
          }
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
      const int pending = min(issued, STAGES);
      for (int i = 0; i < pending; ++i) {
        int s = stage - 1 - i;
        uint32_t ph = phase;
        if (s < 0) {
          s += STAGES;
          ph ^= 1u;
        }
        mbar_wait(bar_full + 8 * s, ph, abort_flag + 1);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issue -----------------------------
    const bool issuer = elect_one();
    // 8-bit containers: E4M3 unless the caller names other formats (E2M3 / E2M1 codes padded to a byte)
    const uint32_t idesc = FP4 ? umma_idesc_mxf4(BLOCK_ROWS, BN) : (umma_idesc_mxf8(BLOCK_ROWS, BN) | p.fmt_bits);
    const uint64_t adesc0 = umma_desc_sw128_kmajor(smem_base + L::OFF_A), bdesc0 = umma_desc_sw128_kmajor(smem_base + L::OFF_B);
    const uint64_t sfa_desc0 = sf_smem_desc(smem_base + L::OFF_SFA), sfb_desc0 = sf_smem_desc(smem_base + L::OFF_SFB);
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int t = tile0; t < num_tiles && ok; t += tile_step) {
      if (!mbar_wait_warp(bar_tempty + 8 * acc, acc_phase ^ 1u, abort_flag)) {
        report_failure(p.status, ST_TIMEOUT, abort_flag);
        break;
      }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_warp(bar_full + 8 * stage, phase, abort_flag)) {
          report_failure(p.status, ST_TIMEOUT, abort_flag);
          ok = false;
          break;
        }
        tc_fence_after();
        // scale atoms of this stage: shared memory -> their TMEM columns
        const uint32_t sfa_t = tmem_base + SF_COL0 + static_cast<uint32_t>(stage * SF_COLS);
        const uint32_t sfb_t = sfa_t + SFA_COLS;
        const uint64_t adesc = adesc0 + static_cast<uint32_t>(stage * (L::A_STAGE >> 4));
        const uint64_t bdesc = bdesc0 + static_cast<uint32_t>(stage * (L::B_STAGE >> 4));
        const uint64_t sfa_desc = sfa_desc0 + static_cast<uint32_t>(stage * (L::SFA_STAGE >> 4));
        const uint64_t sfb_desc = sfb_desc0 + static_cast<uint32_t>(stage * (L::SFB_STAGE >> 4));
        if (issuer) {
#pragma unroll
          for (int h = 0; h < HALVES; ++h) {
            tmem_cp_sf(sfa_t + 4 * h, sfa_desc + h * (MX_SF_ATOM >> 4));
#pragma unroll
            for (int at = 0; at < L::SFB_ATOMS; ++at)
              tmem_cp_sf(sfb_t + 4 * (h * L::SFB_ATOMS + at), sfb_desc + ((h * L::SFB_HALF + at * MX_SF_ATOM) >> 4));
          }
#pragma unroll
          for (int k = 0; k < KBLOCK_BYTES / UMMA_K_BYTES; ++k) {
            if constexpr (FP4) {
              // 32 bytes = 64 elements = scale blocks 2k and 2k+1 of the k-block: atom k/2, bytes 2(k%2) and 2(k%2)+1
              const uint32_t sf_id = static_cast<uint32_t>((k & 1) * 2);
              const uint32_t id = idesc | (sf_id << 4) | (sf_id << 29);
              umma_mxf4(d_tmem, adesc + static_cast<uint64_t>(k * (UMMA_K_BYTES >> 4)),
                        bdesc + static_cast<uint64_t>(k * (UMMA_K_BYTES >> 4)), id, sfa_t + 4 * (k >> 1),
                        sfb_t + 4 * L::SFB_ATOMS * (k >> 1), (kb != kb0 || k != 0) ? 1u : 0u);
            } else {
              // the k-th 32-element block uses byte k of the scale columns: scale-factor id k for both operands
              const uint32_t id = idesc | (static_cast<uint32_t>(k) << 4) | (static_cast<uint32_t>(k) << 29);
              umma_mxf8(d_tmem, adesc + static_cast<uint64_t>(k * (UMMA_K_BYTES >> 4)),
                        bdesc + static_cast<uint64_t>(k * (UMMA_K_BYTES >> 4)), id, sfa_t, sfb_t, (kb != kb0 || k != 0) ? 1u : 0u);
            }
          }
          umma_commit(bar_empty + 8 * stage);
          if (kb == kb1 - 1) umma_commit(bar_tfull + 8 * acc);
        }
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
      acc = (acc + 1) % NACC;
      if (acc == 0) acc_phase ^= 1u;
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    // eight warps: two per TMEM lane quadrant, each with one half of the columns
    const int q = warp & 3;
    const int first_col = ((warp - 2) >> 2) * (BN / 2);
    const uint32_t stage_c = smem_base + L::OFF_C + (warp - 2) * STORE_STAGE;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int t = tile0; t < num_tiles && ok; t += tile_step) {
      int m_blk, n_blk;
      tile_coords(t, m_blk, n_blk);
      if (!mbar_wait(bar_tfull + 8 * acc, acc_phase, abort_flag)) {
        if (lane == 0) report_failure(p.status, ST_TIMEOUT, abort_flag);
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * BN);
      if constexpr (SPLIT) {
        // Park the partial tile at the start of the ring (the barrier above came after the last MMA has
        // read it): sixteen bytes of row r, columns 4 c ..., at (c * 128 + r) * 16, conflict-free.
        static_assert(BLOCK_ROWS * BN * 4 <= L::OFF_SFA, "the partial tile must fit into the ring");
#pragma unroll 1
        for (int c0 = first_col; c0 < first_col + BN / 2; c0 += 64) {
          uint32_t r0[32], r1[32];
          tmem_ld_x32(t_row + c0, r0);
          tmem_ld_x32(t_row + c0 + 32, r1);
          tmem_ld_wait();
          const uint32_t dst = smem_base + static_cast<uint32_t>(((c0 / 4) * BLOCK_ROWS + q * 32 + lane) * 16);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            st_smem_v4(dst + j * BLOCK_ROWS * 16, r0[4 * j], r0[4 * j + 1], r0[4 * j + 2], r0[4 * j + 3]);
            st_smem_v4(dst + (j + 8) * BLOCK_ROWS * 16, r1[4 * j], r1[4 * j + 1], r1[4 * j + 2], r1[4 * j + 3]);
          }
        }
      } else {
        long long rows[4];  // output rows this lane stores pieces of
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int r = m_blk * BLOCK_ROWS + q * 32 + 8 * k + (lane >> 2);
          rows[k] = r < p.M ? r : -1;
        }
        const bool any = m_blk * BLOCK_ROWS + q * 32 < p.M;  // few tokens: most warps have no row and nothing to read
        if (!any && lane == 0) mbar_arrive(bar_tempty + 8 * acc);
#pragma unroll 1
        for (int c0 = any ? first_col : BN; c0 < first_col + BN / 2; c0 += 64) {  // 64 columns per TMEM wait
          uint32_t r0[32], r1[32];
          tmem_ld_x32(t_row + c0, r0);
          tmem_ld_x32(t_row + c0 + 32, r1);
          tmem_ld_wait();
          if (c0 + 64 >= first_col + BN / 2) {  // last read of this accumulator: hand it back to the MMA warp
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_tempty + 8 * acc);
          }
          float y[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) y[j] = __uint_as_float(r0[j]);
          store_rows32<OUTMODE, false>(p.c, rows, p.N, n_blk * BN + c0, y, 32, stage_c, lane);
#pragma unroll
          for (int j = 0; j < 32; ++j) y[j] = __uint_as_float(r1[j]);
          store_rows32<OUTMODE, false>(p.c, rows, p.N, n_blk * BN + c0 + 32, y, 32, stage_c, lane);
        }
      }
      acc = (acc + 1) % NACC;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  if constexpr (SPLIT) {
    // Every thread of every CTA of the cluster comes here, also after a failed wait (all are bounded).
    __syncwarp();
    cluster_sync_all();
    if (warp >= 2) {
      const int q = warp & 3;
      const uint32_t stage_c = smem_base + L::OFF_C + (warp - 2) * STORE_STAGE;
      int m_blk, n_blk;
      tile_coords(tile0, m_blk, n_blk);
      long long rows[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int r = m_blk * BLOCK_ROWS + q * 32 + 8 * k + (lane >> 2);
        rows[k] = r < p.M ? r : -1;
      }
      // columns summed and stored by this CTA (64, 32 or 16), half of them by each of a quadrant's two warps
      const int share = BN / p.split / 2;
      const int c0 = rank * 2 * share + ((warp - 2) >> 2) * share;
      float y[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) y[j] = 0.0f;
      for (int part = 0; part < p.split; ++part) {
        const uint32_t src = map_to_cta(smem_base + static_cast<uint32_t>(((c0 / 4) * BLOCK_ROWS + q * 32 + lane) * 16), part);
        uint4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = 4 * j < share ? ld_dsmem_v4(src + j * BLOCK_ROWS * 16) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          y[4 * j] += __uint_as_float(v[j].x);
          y[4 * j + 1] += __uint_as_float(v[j].y);
          y[4 * j + 2] += __uint_as_float(v[j].z);
          y[4 * j + 3] += __uint_as_float(v[j].w);
        }
      }
      store_rows32<OUTMODE, false>(p.c, rows, p.N, n_blk * BN + c0, y, share, stage_c, lane);
    }
    __syncwarp();
    cluster_sync_all();  // nobody leaves while a peer may still read its shared memory
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// Scale image from row-major scales [rows, K/32] (uint8): see the layout above; rows past `rows` read
// as zero.  A thread moves the four scales of one row and 128-element k-block, a 4-byte word on both
// sides (byte by byte on a side whose base is not a multiple of four).  A call of 1 to 1024
// rows of K = 8192 takes 2.0 to 2.4 us, the floor of a launch.
static __global__ void mx_scale_image_kernel(uint8_t* __restrict__ dst, const uint8_t* __restrict__ src, int rows, int kb32,
                                      int row_tiles) {
  pdl_wait(dst, src);
  pdl_trigger();
  const long long total = static_cast<long long>(kb32 / 4) * row_tiles * (MX_SF_ATOM / 4);
  const bool aligned = (reinterpret_cast<uintptr_t>(src) & 3u) == 0;  // rows of kb32 bytes, a multiple of four
  const bool dst_aligned = (reinterpret_cast<uintptr_t>(dst) & 3u) == 0;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int w = static_cast<int>(i % (MX_SF_ATOM / 4));  // (r % 32) * 4 + r / 32
    const long long atom = i / (MX_SF_ATOM / 4);
    const int tile = static_cast<int>(atom % row_tiles);
    const int kblk = static_cast<int>(atom / row_tiles);
    const int r = tile * 128 + (w >> 2) + 32 * (w & 3);
    uint32_t v = 0;
    if (r < rows) {
      const uint8_t* s = src + static_cast<size_t>(r) * kb32 + kblk * 4;
      v = aligned ? __ldg(reinterpret_cast<const uint32_t*>(s))
                  : (__ldg(s) | (__ldg(s + 1) << 8) | (__ldg(s + 2) << 16) | (static_cast<uint32_t>(__ldg(s + 3)) << 24));
    }
    if (dst_aligned) {
      reinterpret_cast<uint32_t*>(dst)[i] = v;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) dst[4 * i + j] = static_cast<uint8_t>(v >> (8 * j));
    }
  }
}

}  // namespace flyb200
