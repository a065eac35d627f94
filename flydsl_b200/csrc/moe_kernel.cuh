// Grouped (mixture-of-experts) A8W8 GEMMs on the preshuffled weight image.
//
// The routing step has sorted the (token, top-k slot) pairs by expert and padded
// every expert's list to a multiple of tile_m, so that "routing block" b (rows
// [b * tile_m, (b + 1) * tile_m) of the sorted list) belongs to one expert,
// expert_ids[b].  Both stages run the same kernel:
//
//   stage 1 (gate-up):  out[token, slot, n] = silu(g) * u  with
//                       g = x . Wgate[e, n, :], u = x . Wup[e, n, :]
//   stage 2 (down):     out[token, :] (+)= (a2[token, slot, :] . W2[e, :, :]^T) * routed weight
//
// Layout of one CTA: a routing block on the UMMA N side (BN >= tile_m token
// rows, read with one TMA box from the activation rows gathered into sorted
// order), two 128-channel weight tiles of the block's expert on the UMMA M side
// (stage 1: the gate tile and the matching up tile; stage 2: two neighbouring
// tiles), each tile with its own MMA-issuing warp and its own TMEM accumulator.
// Every expert has its own weight image [K/128][rows_per_expert][128 B], one
// after the other, so a tile of any expert is one contiguous 16 KiB burst per
// k-block.
//
// Threads: warp 0 producer (TMA), warp 1 MMA issuer of tile A, warps 2..5
// epilogue, warp 6 MMA issuer of tile B.  Every wait is bounded.
#pragma once
#include "gemm_kernels.cuh"
#include "quant_kernel.cuh"
#include <type_traits>

namespace flyb200 {

enum : int { MOE_OUT_BF16 = 0, MOE_OUT_FP16 = 1, MOE_OUT_F32 = 2 };
constexpr int MOE_THREADS = 224;

struct MoeParams {
  const uint8_t* w;        // weight images, one per expert, back to back
  const float* sa;         // [P] activation scale per sorted row (0 on padding rows)
  const float* sw;         // [experts * n_expert] weight scale per channel
  const int* sorted_ids;   // [P] (slot << 24) | token; padding rows hold token >= tokens
  const int* expert_ids;   // [blocks] expert of each routing block
  const float* sorted_w;   // [P] routed weight per sorted row
  const int* num_valid;    // [1] rows of the sorted list in use (a multiple of tile_m)
  void* out;
  int tokens, topk, experts;
  int n_expert;            // weight rows per expert (stage 1: 2 * inter_dim, stage 2: model_dim)
  int n_out;               // length of an output row (stage 1: inter_dim, stage 2: model_dim)
  int K_bytes;
  int tile_m;              // routing block size (<= BN)
  int stages;              // ring depth
  int doweight;            // multiply by the routed weight in this stage
  int pdl;                 // launched as a programmatic dependent of the gather pass that writes a_sorted and sa
  int* status;
};

struct MoeLayout {
  int off_w, off_a, off_bar, off_misc, off_row, off_sa, off_tw, total;
};
__host__ __device__ inline MoeLayout moe_layout(int bn, int stages) {
  MoeLayout l;
  l.off_w = 0;  // per stage: tile A (16 KiB), tile B (16 KiB)
  l.off_a = stages * 2 * BLOCK_ROWS * KBLOCK_BYTES;
  l.off_bar = l.off_a + stages * bn * KBLOCK_BYTES;
  l.off_misc = (l.off_bar + 8 * (2 * stages + 1) + 15) & ~15;
  l.off_row = l.off_misc + 32;
  l.off_sa = l.off_row + bn * 4;
  l.off_tw = l.off_sa + bn * 4;
  l.total = l.off_tw + bn * 4;
  return l;
}

// x * sigmoid(x), with the fast exponential and reciprocal as in the reference's
// epilogue (exp2 and rcp, kernels/moe/moe_gemm_2stage/layout_helpers.py:247-248)
__device__ __forceinline__ float silu_f32(float x) { return __fdividef(x, 1.0f + __expf(-x)); }

// Two neighbouring channels (lo at `col`, hi at `col + 1`) of one output row.
template <int OUTMODE, bool ACCUM>
__device__ __forceinline__ void moe_store_pair(void* out, size_t elem, float lo, float hi) {
  if constexpr (OUTMODE == MOE_OUT_BF16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    __nv_bfloat162* dst = reinterpret_cast<__nv_bfloat162*>(static_cast<__nv_bfloat16*>(out) + elem);
    if constexpr (ACCUM) {
      atomicAdd(dst, v);
    } else {
      *dst = v;
    }
  } else if constexpr (OUTMODE == MOE_OUT_FP16) {
    __half2 v = __floats2half2_rn(lo, hi);
    __half2* dst = reinterpret_cast<__half2*>(static_cast<__half*>(out) + elem);
    if constexpr (ACCUM) {
      atomicAdd(dst, v);
    } else {
      *dst = v;
    }
  } else {
    float* dst = static_cast<float*>(out) + elem;
    if constexpr (ACCUM) {
      atomicAdd(dst, lo);
      atomicAdd(dst + 1, hi);
    } else {
      *reinterpret_cast<float2*>(dst) = make_float2(lo, hi);
    }
  }
}

// Sixteen tokens (registers) of one channel (this lane) -> memory.  Neighbouring
// lanes swap every other token so that a lane holds two neighbouring channels of
// one token and writes them as one packed element: even lanes take the even
// tokens of the pair of channels, odd lanes the odd tokens.
// `ch`: this lane's channel inside the tile; `n_valid`: channels of the tile that exist (even).
template <int OUTMODE, bool ACCUM>
__device__ __forceinline__ void moe_emit16(void* out, const float (&v)[16], const int* row_s, int c0, int tile_m, int ch,
                                           int n_valid, int col0, int n_out) {
  const bool odd = (ch & 1) != 0;
  const int col = col0 + (ch & ~1);
#pragma unroll
  for (int j = 0; j < 16; j += 2) {
    const float send = odd ? v[j] : v[j + 1];
    const float recv = __shfl_xor_sync(0xffffffffu, send, 1);
    const int t = c0 + j + (odd ? 1 : 0);
    const float lo = odd ? recv : v[j];
    const float hi = odd ? v[j + 1] : recv;
    if (t < tile_m && ch < n_valid) {
      const int row = row_s[t];
      if (row >= 0) moe_store_pair<OUTMODE, ACCUM>(out, static_cast<size_t>(row) * n_out + col, lo, hi);
    }
  }
}

// STAGE 1: gate-up with silu; STAGE 2: down projection.
template <int KIND, int BN, int STAGE, int OUTMODE, bool ACCUM>
__global__ void __launch_bounds__(MOE_THREADS) moe_gemm_kernel(const __grid_constant__ CUtensorMap tmA,
                                                            const MoeParams p) {
  static_assert(STAGE == 1 || STAGE == 2, "two stages");
  static_assert(STAGE == 2 || !ACCUM, "only the down projection accumulates");
  using KT = KindTraits<KIND>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t smem_base = smem_u32(smem_raw);
  const int stages = p.stages;
  const MoeLayout L = moe_layout(BN, stages);
  constexpr int W_TILE = BLOCK_ROWS * KBLOCK_BYTES;
  constexpr int W_STAGE = 2 * W_TILE;
  constexpr int A_STAGE = BN * KBLOCK_BYTES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + L.off_misc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_raw + L.off_misc + 4);
  int* row_s = reinterpret_cast<int*>(smem_raw + L.off_row);
  float* sa_s = reinterpret_cast<float*>(smem_raw + L.off_sa);
  float* tw_s = reinterpret_cast<float*>(smem_raw + L.off_tw);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const uint32_t bar_full = smem_base + L.off_bar;
  const uint32_t bar_empty = bar_full + 8 * stages;
  const uint32_t bar_tfull = bar_empty + 8 * stages;

  // Blocks past the end of the sorted list, and blocks without an expert, have no work.
  const int blk = blockIdx.x;
  const int row0 = blk * p.tile_m;  // first sorted row of the block
  // They leave at once, so that CTAs with work get their SMs - but for the first CTA: a grid of nothing else must
  // not complete before the kernel it depends on.
  const int expert = row0 >= __ldg(p.num_valid) ? -1 : __ldg(p.expert_ids + blk);
  if (expert < 0 || expert >= p.experts) {
    if (p.pdl && blockIdx.x == 0 && blockIdx.y == 0) pdl_wait<>();
    return;
  }
  if ((smem_base & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(p.status, 0, ST_SMEM_ALIGN);
    return;
  }

  // The two weight tiles of this CTA: first row in the expert's image, channels that exist, output column.
  int w_row[2], n_valid[2], col0[2];
  if constexpr (STAGE == 1) {
    const int inter = p.n_out;
    const int c = blockIdx.y * BLOCK_ROWS;
    w_row[0] = c;
    w_row[1] = inter + c;
    n_valid[0] = n_valid[1] = min(BLOCK_ROWS, inter - c);
    col0[0] = col0[1] = c;
  } else {
    const int c = blockIdx.y * 2 * BLOCK_ROWS;
    w_row[0] = c;
    w_row[1] = c + BLOCK_ROWS;
    n_valid[0] = min(BLOCK_ROWS, p.n_out - c);
    n_valid[1] = max(0, min(BLOCK_ROWS, p.n_out - c - BLOCK_ROWS));
    col0[0] = c;
    col0[1] = c + BLOCK_ROWS;
  }
  const bool has_b = n_valid[1] > 0;
  const int num_kb = p.K_bytes / KBLOCK_BYTES;
  const uint8_t* w_expert = p.w + static_cast<size_t>(expert) * p.n_expert * p.K_bytes;
  const float* sw_expert = p.sw + static_cast<size_t>(expert) * p.n_expert;
  const uint32_t w_bytes0 = static_cast<uint32_t>(n_valid[0]) * KBLOCK_BYTES;
  const uint32_t w_bytes1 = static_cast<uint32_t>(n_valid[1]) * KBLOCK_BYTES;
  bool ok = true;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, has_b ? 2 : 1);  // one commit per issuer
    }
    mbar_init(bar_tfull, has_b ? 2 : 1);
    abort_flag[0] = 0;
    abort_flag[1] = 0;  // stays zero: lets the drain below wait on time alone
    fence_mbar_init();
    prefetch_tensormap(&tmA);
  }
  constexpr uint32_t TMEM_COLS = 2 * BN < 32 ? 32 : 2 * BN;
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------ producer ------------------------------
    const bool issuer = elect_one();  // the whole warp runs the loop, here and in the MMA warps, and one lane issues (ptx.cuh)
    const uint64_t pol_a = l2_policy_evict_last();
    const uint64_t pol_w = l2_policy_evict_normal();  // other blocks of the same expert read the same tiles
    int stage = 0;
    uint32_t phase = 0;
    int issued = 0;
    auto load_weights = [&](int kb, int st, uint32_t fb) {
      mbar_expect_tx(fb, A_STAGE + w_bytes0 + w_bytes1);
      const uint32_t wdst = smem_base + L.off_w + st * W_STAGE;
      bulk_load_1d(wdst, w_expert + (static_cast<size_t>(kb) * p.n_expert + w_row[0]) * KBLOCK_BYTES, w_bytes0, fb,
                   pol_w);
      if (has_b)
        bulk_load_1d(wdst + W_TILE, w_expert + (static_cast<size_t>(kb) * p.n_expert + w_row[1]) * KBLOCK_BYTES,
                     w_bytes1, fb, pol_w);
    };
    // As a programmatic dependent of the gather pass the kernel may run before
    // the gathered activations exist.  The weights are model state: the ring is
    // filled with them first; everything the gather pass writes is touched only
    // after griddepcontrol.wait.
    const int pre = p.pdl ? min(stages, num_kb) : 0;
    if (issuer)
      for (int i = 0; i < pre; ++i) load_weights(i, i, bar_full + 8 * i);
    if (p.pdl) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (issuer)
      for (int i = 0; i < pre; ++i)
        tma_load_2d(smem_base + L.off_a + i * A_STAGE, &tmA, bar_full + 8 * i, i * KBLOCK_BYTES, row0, pol_a);
    issued = pre;
    if (pre == stages) phase = 1u; else stage = pre;
    for (int kb = pre; kb < num_kb; ++kb) {
      if (!mbar_wait_warp(bar_empty + 8 * stage, phase ^ 1u, abort_flag)) {
        report_failure(p.status, ST_TIMEOUT, abort_flag);
        ok = false;
        break;
      }
      const uint32_t fb = bar_full + 8 * stage;
      if (issuer) {
        load_weights(kb, stage, fb);
        tma_load_2d(smem_base + L.off_a + stage * A_STAGE, &tmA, fb, kb * KBLOCK_BYTES, row0, pol_a);
      }
      ++issued;
      if (++stage == stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if (p.pdl) pdl_trigger();  // after its wait: the next kernel may be scheduled as the CTAs finish
    if (!ok || *abort_flag) {
      // wait (bounded) for copies still in flight so none lands after the CTA is gone
      const int pending = min(issued, stages);
      for (int i = 0; i < pending; ++i) {
        int s = stage - 1 - i;
        uint32_t ph = phase;
        if (s < 0) {
          s += stages;
          ph ^= 1u;
        }
        mbar_wait(bar_full + 8 * s, ph, abort_flag + 1);
      }
    }
    __syncwarp();
  } else if (warp == 1 || warp == 6) {
    // ------------------------------ MMA issue -----------------------------
    const int which = warp == 1 ? 0 : 1;  // tile A / tile B
    if (which == 0 || has_b) {
      const bool issuer = elect_one();
      constexpr uint32_t idesc = umma_idesc(KT::dfmt, KT::abfmt, BLOCK_ROWS, BN);
      const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(which * BN);
      const uint64_t wdesc0 = umma_desc_sw128_kmajor(smem_base + L.off_w + which * W_TILE);
      const uint64_t adesc0 = umma_desc_sw128_kmajor(smem_base + L.off_a);
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait_warp(bar_full + 8 * stage, phase, abort_flag)) {
          report_failure(p.status, ST_TIMEOUT, abort_flag);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t wdesc = wdesc0 + static_cast<uint32_t>(stage * (W_STAGE >> 4));
        const uint64_t adesc = adesc0 + static_cast<uint32_t>(stage * (A_STAGE >> 4));
        if (issuer) {
#pragma unroll
          for (int k = 0; k < KBLOCK_BYTES / UMMA_K_BYTES; ++k) {
            umma_ss<KIND>(d_tmem, wdesc + static_cast<uint64_t>(k * (UMMA_K_BYTES >> 4)),
                          adesc + static_cast<uint64_t>(k * (UMMA_K_BYTES >> 4)), idesc, (kb != 0 || k != 0) ? 1u : 0u);
          }
          umma_commit(bar_empty + 8 * stage);
          if (kb == num_kb - 1) umma_commit(bar_tfull);
        }
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------ epilogue -------------------------------
    // thread <-> channel (TMEM lane), registers <-> tokens of the block
    const int q = warp & 3;
    const int ch = q * 32 + lane;
    const int et = threadIdx.x - 64;
    const int n_rows = __ldg(p.num_valid);
    if (p.pdl) asm volatile("griddepcontrol.wait;" ::: "memory");  // p.sa is written by the gather pass
    for (int i = et; i < BN; i += 128) {
      int row = -1;
      float sa = 0.0f, tw = 1.0f;
      if (i < p.tile_m && row0 + i < n_rows) {
        const int id = __ldg(p.sorted_ids + row0 + i);
        const int tok = id & 0xFFFFFF;
        const int slot = static_cast<int>(static_cast<uint32_t>(id) >> 24);
        if (tok < p.tokens && slot < p.topk) {
          row = (STAGE == 2 && ACCUM) ? tok : tok * p.topk + slot;
          sa = __ldg(p.sa + row0 + i);
          if (p.doweight) tw = __ldg(p.sorted_w + row0 + i);
        }
      }
      row_s[i] = row;
      sa_s[i] = sa;
      tw_s[i] = tw;
    }
    const float sw0 = ch < n_valid[0] ? __ldg(sw_expert + w_row[0] + ch) : 0.0f;
    const float sw1 = ch < n_valid[1] ? __ldg(sw_expert + w_row[1] + ch) : 0.0f;
    named_bar_sync(1, 128);

    ok = mbar_wait(bar_tfull, 0, abort_flag);
    if (!ok && lane == 0) report_failure(p.status, ST_TIMEOUT, abort_flag);
    ok = named_bar_and(1, 128, ok);
    if (ok) {
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += 16) {
        if (c0 >= p.tile_m) break;
        uint32_t ra[16], rb[16];
        tmem_ld_x16(t_row + c0, ra);
        if (has_b) tmem_ld_x16(t_row + BN + c0, rb);
        tmem_ld_wait();
        float va[16], vb[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float sa = sa_s[c0 + j];
          const float a = KT::is_int ? static_cast<float>(static_cast<int32_t>(ra[j])) : __uint_as_float(ra[j]);
          const float b = !has_b ? 0.0f : KT::is_int ? static_cast<float>(static_cast<int32_t>(rb[j])) : __uint_as_float(rb[j]);
          // the reference's order: accumulator times weight scale, then times activation scale
          const float fa = (a * sw0) * sa;
          const float fb = (b * sw1) * sa;
          if constexpr (STAGE == 1) {
            float y = silu_f32(fa) * fb;
            if (p.doweight) y *= tw_s[c0 + j];
            va[j] = y;
          } else {
            const float tw = tw_s[c0 + j];
            va[j] = p.doweight ? fa * tw : fa;
            vb[j] = p.doweight ? fb * tw : fb;
          }
        }
        moe_emit16<OUTMODE, ACCUM>(p.out, va, row_s, c0, p.tile_m, ch, n_valid[0], col0[0], p.n_out);
        if constexpr (STAGE == 2) {
          if (has_b) moe_emit16<OUTMODE, ACCUM>(p.out, vb, row_s, c0, p.tile_m, ch, n_valid[1], col0[1], p.n_out);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------
// Large routing blocks (tile_m a multiple of 128, or 64): persistent form
// ---------------------------------------------------------------------------
// Tokens on the UMMA M side (128 sorted rows per work item), the two weight
// tiles side by side on the N side (256 channels: stage 1 gate | up, stage 2 two
// neighbouring tiles), one CTA per SM walking the (row block, channel pair)
// items, a shared-memory ring that keeps streaming across items and two TMEM
// accumulators so that the epilogue of an item overlaps the mainloop of the
// next.  A thread of the epilogue owns one token row (stage 2: two warps per 32 rows): it
// reads the gate and up columns of the same channel from its own TMEM lane; the
// outputs leave through store_rows32.
constexpr int MOE_ROWS_STAGES = 4;
constexpr int MOE_ROWS_BN = 2 * BLOCK_ROWS;
constexpr int MOE_ROWS_GROUP = 32;  // row blocks per rasterisation group (16 MiB of activations at K = 4096)

constexpr int STORE_STAGE = 32 * 64;  // shared memory of a warp for store_rows32, bytes
// Producer, MMA issuer and epilogue warps: eight where the epilogue is as long as the mainloop it overlaps (the down
// projection), four for the gate-up stage, whose K is longer: eight / four, us, gather included, 4096 tokens x top-2 x 4096 x
// 2048 136.0 / 132.8, 515 x top-4 x 2048 x 1408 29.0 / 28.5, 1024 x top-2 x 4096 x 2048 51.5 / 51.2.
__host__ __device__ constexpr int moe_rows_epilogue_warps(int stage) { return stage == 1 ? 4 : 8; }
__host__ __device__ constexpr int moe_rows_threads(int stage) { return 64 + 32 * moe_rows_epilogue_warps(stage); }
struct MoeRowsSmem {
  static constexpr int A_STAGE = BLOCK_ROWS * KBLOCK_BYTES;
  static constexpr int B_STAGE = MOE_ROWS_BN * KBLOCK_BYTES;
  static constexpr int OFF_A = 0;
  static constexpr int OFF_B = OFF_A + MOE_ROWS_STAGES * A_STAGE;
  static constexpr int OFF_C = OFF_B + MOE_ROWS_STAGES * B_STAGE;    // 8 warps x one store stage
  static constexpr int OFF_SW = OFF_C + 8 * STORE_STAGE;             // 1024 weight scales: 8 warps x 128 or 4 x 256
  static constexpr int OFF_BAR = OFF_SW + 8 * BLOCK_ROWS * 4;        // full[S], empty[S], tfull[2], tempty[2]
  static constexpr int OFF_MISC = OFF_BAR + 8 * (2 * MOE_ROWS_STAGES + 4);
  static constexpr int TOTAL = OFF_MISC + 16;
};

// 16 bytes of an output row added in place: one reduction instead of four (packed halves) or eight
// (single floats of a pair) that each occupy an L2 slice for a whole 32-byte sector.
template <int OUTMODE>
__device__ __forceinline__ void moe_red16(void* dst, const uint32_t (&v)[4]) {
  if constexpr (OUTMODE == MOE_OUT_BF16) {
    asm volatile("red.relaxed.gpu.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(dst), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3])
                 : "memory");
  } else if constexpr (OUTMODE == MOE_OUT_FP16) {
    asm volatile("red.relaxed.gpu.global.add.noftz.v4.f16x2 [%0], {%1, %2, %3, %4};" ::"l"(dst), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3])
                 : "memory");
  } else {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(__uint_as_float(v[0])),
                 "f"(__uint_as_float(v[1])), "f"(__uint_as_float(v[2])), "f"(__uint_as_float(v[3]))
                 : "memory");
  }
}

// 32 rows (one per lane) x 32 consecutive channels of output, n_ok (a multiple of 8) of them existing,
// in 16-byte accesses.  The lanes' rows lie apart in memory, so a lane that wrote its own row would touch a
// line of its own with every access; the chunk is turned in 2 KiB of shared memory instead (swizzled, no bank
// conflicts) and four lanes write 64 contiguous bytes of a row: with that and eight epilogue warps instead of
// four the down projection of 4096 tokens x top-2 (K = 2048) goes from 70.9 to 67.0 us, the layer from 277 to 274,
// MXFP8 600 x 1792 x 2048 from 9.6 to 8.2, 384 x 1024 x 4096 from 10.1 to 9.1, 256 x 4096 x 14336 from 25.9 to 24.5.  `rows[k]`: output row of lane 8 k + lane / 4, or
// negative for none.  Rows are multiples of 16 channels, so every access is 16-byte aligned.  Accumulating one
// packed pair at a time bound the down projection (515 tokens x top-4 x 2048 fp16, int8, K = 1408: 94.4 us).
template <int OUTMODE, bool ACCUM>
__device__ __forceinline__ void store_rows32(void* out, const long long (&rows)[4], int n_out, int col, const float (&y)[32], int n_ok,
                                             uint32_t stage, int lane) {
  constexpr int PER = OUTMODE == MOE_OUT_F32 ? 4 : 8;  // channels per 16 bytes
  constexpr int COLS = 4 * PER;                        // channels turned at a time: 64 bytes per row
  const int piece = lane & 3;
  const uint32_t mine = stage + static_cast<uint32_t>(lane * 64);
#pragma unroll
  for (int c0 = 0; c0 < 32; c0 += COLS) {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      uint32_t v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int e = c0 + g * PER;
        if constexpr (OUTMODE == MOE_OUT_F32) {
          v[i] = __float_as_uint(y[e + i]);
        } else if constexpr (OUTMODE == MOE_OUT_BF16) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(y[e + 2 * i], y[e + 2 * i + 1]);
          v[i] = *reinterpret_cast<const uint32_t*>(&h);
        } else {
          const __half2 h = __floats2half2_rn(y[e + 2 * i], y[e + 2 * i + 1]);
          v[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
      }
      st_smem_v4(mine + static_cast<uint32_t>((g ^ ((lane >> 1) & 3)) << 4), v[0], v[1], v[2], v[3]);
    }
    __syncwarp();
    const bool exists = c0 + piece * PER < n_ok;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int r = 8 * k + (lane >> 2);
      const uint4 q = ld_smem_v4(stage + static_cast<uint32_t>(r * 64 + ((piece ^ ((r >> 1) & 3)) << 4)));
      if (!exists || rows[k] < 0) continue;
      unsigned char* dst = static_cast<unsigned char*>(out) + (rows[k] * n_out + col + c0 + piece * PER) * (16 / PER);
      if constexpr (ACCUM) {
        const uint32_t v[4] = {q.x, q.y, q.z, q.w};
        moe_red16<OUTMODE>(dst, v);
      } else {
        *reinterpret_cast<uint4*>(dst) = q;
      }
    }
    __syncwarp();  // the stage is free again
  }
}

// First rows in the expert's image of the two tiles of a channel pair, and the channels of each that exist.
template <int STAGE>
__device__ __forceinline__ void moe_pair_tiles(const MoeParams& p, int pair, int (&w_row)[2], int (&n_valid)[2]) {
  if constexpr (STAGE == 1) {
    const int c = pair * BLOCK_ROWS;
    w_row[0] = c;
    w_row[1] = p.n_out + c;
    n_valid[0] = n_valid[1] = min(BLOCK_ROWS, p.n_out - c);
  } else {
    const int c = pair * MOE_ROWS_BN;
    w_row[0] = c;
    w_row[1] = c + BLOCK_ROWS;
    n_valid[0] = min(BLOCK_ROWS, p.n_out - c);
    n_valid[1] = max(0, min(BLOCK_ROWS, p.n_out - c - BLOCK_ROWS));
  }
}

// What one epilogue warp does with the 128-row accumulator tiles of its items: stage 1 both tiles of a channel pair, stage 2
// one of them.  The factors of the next item (routing id, activation scale, routed weight, weight scales) are asked for
// before the current one is converted.
__host__ __device__ constexpr int moe_rows_scales(int stage) { return stage == 1 ? 2 * BLOCK_ROWS : BLOCK_ROWS; }  // of a warp
template <int KIND, int STAGE, int OUTMODE, bool ACCUM>
struct MoeRowsEpilogue {
  static constexpr int SCALES = moe_rows_scales(STAGE);
  const MoeParams& p;
  float* sw_s;       // shared memory of the warp for the weight scales of its columns
  uint32_t stage_c;  // ... and for store_rows32
  int half;          // stage 2: which of the two tiles of a channel pair
  int lane;
  // of the item asked for last: this lane's row, its share of the weight scales, output column, channels and tile width
  int id;
  float sa, tw, sw[SCALES / 32];
  int col0_next, cols_next, width_next;

  // This lane's sorted row `srow` (`row_ok`: it belongs to the item) and `width` channels (a multiple of 32) of every tile
  // of channel pair `pair` from the `c0`-th on.
  __device__ __forceinline__ void fetch(int expert, int srow, bool row_ok, int pair, int c0, int width) {
    int w_row[2], n_valid[2];
    moe_pair_tiles<STAGE>(p, pair, w_row, n_valid);
    width_next = width;
    cols_next = (STAGE == 2 && half ? n_valid[1] : n_valid[0]) - c0;
    col0_next = (STAGE == 1 ? pair * BLOCK_ROWS : pair * MOE_ROWS_BN + half * BLOCK_ROWS) + c0;
    id = -1;  // token 0xFFFFFF of slot 255: no row
    sa = 0.0f;
    tw = 1.0f;
    if (row_ok) {
      id = __ldg(p.sorted_ids + srow);
      sa = __ldg(p.sa + srow);
      if (p.doweight) tw = __ldg(p.sorted_w + srow);
    }
    const float* sw_expert = p.sw + static_cast<size_t>(expert) * p.n_expert + c0;
#pragma unroll
    for (int i = 0; i < SCALES / 32; ++i) {
      const bool second = STAGE == 1 ? i >= BLOCK_ROWS / 32 : half == 1;
      const int c = (i * 32 + lane) & (BLOCK_ROWS - 1);
      sw[i] = c < cols_next ? __ldg(sw_expert + (second ? w_row[1] : w_row[0]) + c) : 0.0f;
    }
  }

  // The item asked for last.  `next` asks for the one after it; `wait` blocks until the accumulator at `t_row` is complete
  // (`width` columns of the first tile, then those of the second); `release` (one lane) hands it back after the last
  // read.  False if the wait failed.
  template <typename NextFn, typename WaitFn, typename ReleaseFn>
  __device__ __forceinline__ bool run(uint32_t t_row, NextFn next, WaitFn wait, ReleaseFn release) {
    const int tok = id & 0xFFFFFF;
    const int slot = static_cast<int>(static_cast<uint32_t>(id) >> 24);
    const bool exists = tok < p.tokens && slot < p.topk;
    const long long orow = !exists ? -1 : (STAGE == 2 && ACCUM) ? tok : static_cast<long long>(tok) * p.topk + slot;
    const float row_scale = exists ? sa : 0.0f, row_weight = tw;
    long long rows[4];  // output rows this lane stores pieces of
#pragma unroll
    for (int k = 0; k < 4; ++k) rows[k] = __shfl_sync(0xffffffffu, orow, 8 * k + (lane >> 2));
    __syncwarp();  // the scales of the item before have been read
#pragma unroll
    for (int i = 0; i < SCALES / 32; ++i) sw_s[i * 32 + lane] = sw[i];
    __syncwarp();
    const int cols = cols_next, col0 = col0_next, width = width_next;
    next();
    if (!wait()) return false;
    tc_fence_after();
    constexpr bool IS_INT = KindTraits<KIND>::is_int;
    auto to_f = [](uint32_t r) { return IS_INT ? static_cast<float>(static_cast<int32_t>(r)) : __uint_as_float(r); };
    auto last_read = [&]() {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) release();
    };
    if constexpr (STAGE == 1) {
      // Not unrolled, here and below, and no accumulators asked for ahead: four times this code was slower, in the gate-up
      // stage 5.3 us a tile instead of 3.65.
#pragma unroll 1
      for (int c = 0; c < width; c += 32) {
        uint32_t rg[32], ru[32];
        tmem_ld_x32(t_row + c, rg);
        tmem_ld_x32(t_row + width + c, ru);
        tmem_ld_wait();
        if (c + 32 >= width) last_read();
        float y[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float g = (to_f(rg[j]) * sw_s[c + j]) * row_scale;
          const float u = (to_f(ru[j]) * sw_s[BLOCK_ROWS + c + j]) * row_scale;
          float v = silu_f32(g) * u;
          if (p.doweight) v *= row_weight;
          y[j] = v;
        }
        const int n_ok = min(32, cols - c);
        if (n_ok > 0) store_rows32<OUTMODE, ACCUM>(p.out, rows, p.n_out, col0 + c, y, n_ok, stage_c, lane);
      }
    } else {
#pragma unroll 1
      for (int c = 0; c < width; c += 32) {
        uint32_t r[32];
        tmem_ld_x32(t_row + half * width + c, r);
        tmem_ld_wait();
        if (c + 32 >= width) last_read();
        float y[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float v = (to_f(r[j]) * sw_s[c + j]) * row_scale;
          y[j] = p.doweight ? v * row_weight : v;
        }
        const int n_ok = min(32, cols - c);
        if (n_ok > 0) store_rows32<OUTMODE, ACCUM>(p.out, rows, p.n_out, col0 + c, y, n_ok, stage_c, lane);
      }
    }
    return true;
  }
};

template <int KIND, int STAGE, int OUTMODE, bool ACCUM>
__global__ void __launch_bounds__(moe_rows_threads(STAGE), 1) moe_rows_kernel(const __grid_constant__ CUtensorMap tmA,
                                                                  const MoeParams p) {
  static_assert(STAGE == 2 || !ACCUM, "only the down projection accumulates");
  using L = MoeRowsSmem;
  using KT = KindTraits<KIND>;
  constexpr int STAGES = MOE_ROWS_STAGES;
  constexpr int BN = MOE_ROWS_BN;
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
      mbar_init(bar_tempty + 8 * s, moe_rows_epilogue_warps(STAGE));
    }
    abort_flag[0] = 0;
    abort_flag[1] = 0;
    fence_mbar_init();
    prefetch_tensormap(&tmA);
  }
  constexpr uint32_t TMEM_COLS = 512;
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int* num_valid = p.num_valid;
  pdl_wait(num_valid);  // launched as a programmatic dependent: nothing in global memory is touched before this

  // Work items: (row block of 128 sorted rows, channel pair).  Row blocks run
  // fastest, so CTAs working side by side share the weight tiles of an expert,
  // and they are taken in groups of MOE_ROWS_GROUP whose activation rows stay in
  // L2 while the group walks all channel pairs.
  const int n_rows = __ldg(num_valid);
  const int row_blocks = (n_rows + BLOCK_ROWS - 1) / BLOCK_ROWS;
  const int pairs = STAGE == 1 ? (p.n_out + BLOCK_ROWS - 1) / BLOCK_ROWS : (p.n_out + BN - 1) / BN;
  // Routing blocks of 64 rows: a 128-row block holds two of them.  Where both have
  // the same expert they are one item; where the expert changes inside the 128
  // rows the block is worked on twice ("passes"), once per expert, each pass
  // storing only its own 64 rows.  That happens once per expert boundary.
  const int passes = p.tile_m == 64 ? 2 : 1;
  const int items = row_blocks * pairs * passes;
  const int num_kb = p.K_bytes / KBLOCK_BYTES;
  auto item_coords = [&](int t, int& rb, int& pair) {
    const int per_group = MOE_ROWS_GROUP * pairs;
    const int g = t / per_group;
    const int first = g * MOE_ROWS_GROUP;
    const int gm = min(MOE_ROWS_GROUP, row_blocks - first);
    const int r = t - g * per_group;
    rb = first + r % gm;
    pair = r / gm;
  };
  // expert of the routing block that starts at sorted row `row`, or -1 when there is none
  auto expert_at = [&](int row) {
    if (row >= n_rows) return -1;
    const int e = __ldg(p.expert_ids + row / p.tile_m);
    return (e < 0 || e >= p.experts) ? -1 : e;
  };
  // Item t -> row block, channel pair, expert (-1: nothing to do) and the rows [lo, hi) it stores.
  auto item_of = [&](int t, int& rb, int& pair, int& lo, int& hi) {
    // all first passes come before the (few) second passes, so that the CTAs share the real work evenly
    const int base = row_blocks * pairs;
    item_coords(t % base, rb, pair);
    lo = 0;
    hi = BLOCK_ROWS;
    if (passes == 1) return expert_at(rb * BLOCK_ROWS);
    const int ea = expert_at(rb * BLOCK_ROWS), eb = expert_at(rb * BLOCK_ROWS + 64);
    if (t < base) {
      if (eb != ea) hi = 64;
      return ea;
    }
    lo = 64;
    return eb == ea ? -1 : eb;
  };
  if (warp == 0) {
    // ------------------------------ producer ------------------------------
    const bool issuer = elect_one();
    const uint64_t pol = l2_policy_evict_last();
    int stage = 0;
    uint32_t phase = 0;
    int issued = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
      int rb, pair, lo, hi;
      const int expert = __shfl_sync(0xffffffffu, item_of(t, rb, pair, lo, hi), 0);
      if (expert < 0) continue;
      int w_row[2], n_valid[2];
      moe_pair_tiles<STAGE>(p, pair, w_row, n_valid);
      const uint8_t* w_expert = p.w + static_cast<size_t>(expert) * p.n_expert * p.K_bytes;
      const uint32_t b0 = static_cast<uint32_t>(n_valid[0]) * KBLOCK_BYTES, b1 = static_cast<uint32_t>(n_valid[1]) * KBLOCK_BYTES;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait_warp(bar_empty + 8 * stage, phase ^ 1u, abort_flag)) {
          report_failure(p.status, ST_TIMEOUT, abort_flag);
          ok = false;
          break;
        }
        const uint32_t fb = bar_full + 8 * stage;
        const uint32_t bdst = smem_base + L::OFF_B + stage * L::B_STAGE;
        if (issuer) {
          mbar_expect_tx(fb, L::A_STAGE + b0 + b1);
          tma_load_2d(smem_base + L::OFF_A + stage * L::A_STAGE, &tmA, fb, kb * KBLOCK_BYTES, rb * BLOCK_ROWS, pol);
          bulk_load_1d(bdst, w_expert + (static_cast<size_t>(kb) * p.n_expert + w_row[0]) * KBLOCK_BYTES, b0, fb, pol);
          if (b1)
            bulk_load_1d(bdst + BLOCK_ROWS * KBLOCK_BYTES,
                         w_expert + (static_cast<size_t>(kb) * p.n_expert + w_row[1]) * KBLOCK_BYTES, b1, fb, pol);
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
    constexpr uint32_t idesc = umma_idesc(KT::dfmt, KT::abfmt, BLOCK_ROWS, BN);
    const uint64_t adesc0 = umma_desc_sw128_kmajor(smem_base + L::OFF_A), bdesc0 = umma_desc_sw128_kmajor(smem_base + L::OFF_B);
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
      int rb, pair, lo, hi;
      if (__shfl_sync(0xffffffffu, item_of(t, rb, pair, lo, hi), 0) < 0) continue;
      if (!mbar_wait_warp(bar_tempty + 8 * acc, acc_phase ^ 1u, abort_flag)) {
        report_failure(p.status, ST_TIMEOUT, abort_flag);
        break;
      }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait_warp(bar_full + 8 * stage, phase, abort_flag)) {
          report_failure(p.status, ST_TIMEOUT, abort_flag);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t adesc = adesc0 + static_cast<uint32_t>(stage * (L::A_STAGE >> 4));
        const uint64_t bdesc = bdesc0 + static_cast<uint32_t>(stage * (L::B_STAGE >> 4));
        if (issuer) {
#pragma unroll
          for (int k = 0; k < KBLOCK_BYTES / UMMA_K_BYTES; ++k) {
            umma_ss<KIND>(d_tmem, adesc + static_cast<uint64_t>(k * (UMMA_K_BYTES >> 4)),
                          bdesc + static_cast<uint64_t>(k * (UMMA_K_BYTES >> 4)), idesc, (kb | k) != 0 ? 1u : 0u);
          }
          umma_commit(bar_empty + 8 * stage);
          if (kb == num_kb - 1) umma_commit(bar_tfull + 8 * acc);
        }
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    // Stage 1: one warp per TMEM lane quadrant, all 128 channels of the gate and of the up tile.  Stage 2: two, each
    // with the 128 channels of one of the two tiles.
    const int q = warp & 3;  // TMEM lane quadrant this warp may read
    MoeRowsEpilogue<KIND, STAGE, OUTMODE, ACCUM> ep{p, reinterpret_cast<float*>(smem_raw + L::OFF_SW) + (warp - 2) * moe_rows_scales(STAGE),
                                                    smem_base + L::OFF_C + (warp - 2) * STORE_STAGE, (warp - 2) >> 2, lane};
    // asks for the first item from t on that has work; the item's number, or `items` and more
    auto fetch_from = [&](int t) {
      for (; t < items; t += gridDim.x) {
        int rb, pair, lo, hi;
        const int expert = item_of(t, rb, pair, lo, hi);
        if (expert < 0) continue;
        const int trow = q * 32 + lane;  // this thread's token row
        const int srow = rb * BLOCK_ROWS + trow;
        ep.fetch(expert, srow, srow < n_rows && trow >= lo && trow < hi, pair, 0, BLOCK_ROWS);
        break;
      }
      return t;
    };
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int t = fetch_from(blockIdx.x); t < items && ok;) {
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * BN);
      ok = ep.run(t_row, [&]() { t = fetch_from(t + gridDim.x); }, [&]() { return mbar_wait(bar_tfull + 8 * acc, acc_phase, abort_flag); },
                  [&]() { mbar_arrive(bar_tempty + 8 * acc); });
      if (!ok && lane == 0) report_failure(p.status, ST_TIMEOUT, abort_flag);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// Gather the activation rows (and their scales) into sorted order:
//   dst[p, :] = src[row(p), :], dst_scale[p] = src_scale[row(p)]
// with row(p) = token (by_slot == 0, stage 1), token * topk + slot (by_slot == 1,
// stage 2) or slot * tokens + token (by_slot == 2: slot-major activations, the
// reference's "int8smooth" stage 1); rows that are padding, or past num_valid,
// become zero with scale zero.
// One warp per row, 16 bytes per lane and step.
static __global__ void moe_gather_rows_kernel(uint8_t* __restrict__ dst, float* __restrict__ dst_scale,
                                       const uint8_t* __restrict__ src, const float* __restrict__ src_scale,
                                       const int* __restrict__ sorted_ids, const int* __restrict__ num_valid, int tokens,
                                       int topk, int by_slot, int K_bytes, int rows) {
  pdl_wait(dst, dst_scale, src, src_scale, sorted_ids, num_valid);
  pdl_trigger();  // a GEMM launched as programmatic dependent may start its weight stream now
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_valid = __ldg(num_valid);
  for (int r = blockIdx.x * warps_per_block + (threadIdx.x >> 5); r < rows; r += gridDim.x * warps_per_block) {
    long long srow = -1;
    if (r < n_valid) {
      const int id = __ldg(sorted_ids + r);
      const int tok = id & 0xFFFFFF;
      const int slot = static_cast<int>(static_cast<uint32_t>(id) >> 24);
      if (tok < tokens && slot < topk)
        srow = by_slot == 1 ? static_cast<long long>(tok) * topk + slot
                            : by_slot == 2 ? static_cast<long long>(slot) * tokens + tok : tok;
    }
    uint4* d = reinterpret_cast<uint4*>(dst + static_cast<size_t>(r) * K_bytes);
    if (srow >= 0) {
      const uint4* s = reinterpret_cast<const uint4*>(src + static_cast<size_t>(srow) * K_bytes);
      for (int i = lane; i < K_bytes / 16; i += 32) d[i] = __ldg(s + i);
      if (lane == 0) dst_scale[r] = __ldg(src_scale + srow);
    } else {
      for (int i = lane; i < K_bytes / 16; i += 32) d[i] = make_uint4(0, 0, 0, 0);
      if (lane == 0) dst_scale[r] = 0.0f;
    }
  }
}

// The per-token quantiser and the gather of stage 2 as one pass: sorted row p takes the 16-bit row
// token * topk + slot of `x`, quantises it (quant_kernel.cuh) and writes codes and scale where the down
// projection reads them; padding rows, and rows past num_valid, become zero with scale zero.  Saves the
// write and the read of the codes in between and a launch, and rows of routes that nobody sorted are never
// read.  Bound by memory: alone, 8192 routes x 2048 12.0 us against 12.0 (quantiser) + 8.6 (gather); the layer of 4096
// tokens x top-2 x 4096 x 2048 goes from 295 to 284 us, of 32 tokens from 115 to 88 (a launch and two allocations).
template <bool FP8, int NV, int WPR>
__global__ void __launch_bounds__(256)
moe_quant_sorted_kernel(uint8_t* __restrict__ y, float* __restrict__ scale, const __nv_bfloat16* __restrict__ x,
                        const int* __restrict__ sorted_ids, const int* __restrict__ num_valid, int tokens, int topk, int K, int rows) {
  constexpr int VEC = 8, TPR = 32 * WPR;
  __shared__ uint32_t red[8];
  pdl_wait(y, scale, x, sorted_ids, num_valid);
  pdl_trigger();  // a GEMM launched as programmatic dependent may start its weight stream now
  const int group = threadIdx.x / TPR, tid = threadIdx.x % TPR;
  const int r = blockIdx.x * (8 / WPR) + group;
  if (r >= rows) return;
  long long srow = -1;
  if (r < __ldg(num_valid)) {
    const int id = __ldg(sorted_ids + r);
    const int tok = id & 0xFFFFFF;
    const int slot = static_cast<int>(static_cast<uint32_t>(id) >> 24);
    if (tok < tokens && slot < topk) srow = static_cast<long long>(tok) * topk + slot;
  }
  uint8_t* yr = y + static_cast<size_t>(r) * K;
  if (srow < 0) {  // the same for all threads of the row
    for (int k = tid * VEC; k < K; k += TPR * VEC) *reinterpret_cast<uint2*>(yr + k) = make_uint2(0u, 0u);
    if (tid == 0) scale[r] = 0.0f;
    return;
  }
  const __nv_bfloat16* xr = x + srow * K;
  uint4 raw[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int k = (i * TPR + tid) * VEC;
    raw[i] = k < K ? __ldg(reinterpret_cast<const uint4*>(xr + k)) : make_uint4(0u, 0u, 0u, 0u);
  }
  quant_row_from_registers<__nv_bfloat16, FP8, NV, WPR>(raw, yr, scale + r, K, tid, red, group * WPR, 1 + group);
}

// ---------------------------------------------------------------------------
// Routing table (the layout tests/kernels/test_moe_gemm_2stage.py:99-137 of the
// reference describes): counting sort of the (token, slot) pairs by expert,
// stable, every expert's run padded to a multiple of block_size.
// ---------------------------------------------------------------------------
// One launch, one CTA per expert, no scratch.  Every CTA counts all pairs into a
// shared-memory histogram (so it knows where its run starts and where the list ends
// without talking to the others), then walks the pairs once more and writes its own
// run, its padding and its share of the tail behind the last run.  Latency-bound: a
// chunk is four pairs per thread, one barrier, so 4096 pairs cost about a microsecond.
// Measured alone (pairs / experts, one kernel against memset + count + a walk of 256 pairs at
// a time, us): 64 / 8 4.4 against 5.0, 2060 / 16 5.4 against 11.5, 8192 / 8 9.5 against 29.  (In a chain of
// programmatic dependents it starts early and waits, which a profile counts to it: 17.5 us for the last.)
constexpr int MOE_SORT_MAX_THREADS = 1024;
constexpr int MOE_SORT_BINS = 4096;  // experts counted per pass over the pairs

// ids of the four pairs at `i` (a multiple of four), -1 past the end; made relative to `first_expert`.  Of an
// 8-byte id the low half counts, as in torch's conversion to int32, so that the table and the masked top-k sum
// (which reads 4-byte ids) agree on every route.
template <typename ID>
__device__ __forceinline__ void moe_load_ids(const ID* __restrict__ ids, long long i, long long n_pairs, long long first_expert,
                                             int experts, bool vec, int (&e)[4]) {
  int v[4];
  if (vec && i + 3 < n_pairs) {
    if constexpr (sizeof(ID) == 4) {
      const int4 q = __ldg(reinterpret_cast<const int4*>(ids + i));
      v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
    } else {
      const longlong2 q0 = __ldg(reinterpret_cast<const longlong2*>(ids + i)), q1 = __ldg(reinterpret_cast<const longlong2*>(ids + i + 2));
      v[0] = static_cast<int>(q0.x), v[1] = static_cast<int>(q0.y), v[2] = static_cast<int>(q1.x), v[3] = static_cast<int>(q1.y);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = i + j < n_pairs ? static_cast<int>(__ldg(ids + i + j)) : -1;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const long long local = v[j] - first_expert;
    e[j] = v[j] >= 0 && local >= 0 && local < experts ? static_cast<int>(local) : -1;
  }
}

template <typename ID>
__global__ void __launch_bounds__(MOE_SORT_MAX_THREADS)
moe_sort_kernel(const ID* __restrict__ topk_ids, const float* __restrict__ topk_weights, int n_pairs, int topk, int tokens,
                int experts, long long first_expert, int block_size, int* __restrict__ sorted_ids,
                float* __restrict__ sorted_weights, int* __restrict__ sorted_expert_ids, int* __restrict__ post_pad,
                int max_padded, int max_blocks) {
  __shared__ int bins[MOE_SORT_BINS];
  __shared__ int warp_sums[2][32];
  __shared__ int s_start, s_total, s_mine;
  pdl_wait(topk_ids, topk_weights, sorted_ids, sorted_weights, sorted_expert_ids, post_pad);
  pdl_trigger();
  const int me = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int threads = blockDim.x, warps = threads >> 5;
  const bool vec = (reinterpret_cast<uintptr_t>(topk_ids) & 15u) == 0;
  if (tid == 0) s_start = s_total = s_mine = 0;
  for (int b0 = 0; b0 < experts; b0 += MOE_SORT_BINS) {
    const int nb = min(MOE_SORT_BINS, experts - b0);
    __syncthreads();  // the previous pass has been read
    for (int i = tid; i < nb; i += threads) bins[i] = 0;
    __syncthreads();
    for (long long i = 4 * tid; i < n_pairs; i += 4 * threads) {
      int e[4];
      moe_load_ids(topk_ids, i, n_pairs, first_expert, experts, vec, e);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (e[j] >= b0 && e[j] < b0 + nb) atomicAdd(&bins[e[j] - b0], 1);
    }
    __syncthreads();
    int before = 0, all = 0;
    for (int i = tid; i < nb; i += threads) {
      const int c = bins[i];
      const int padded = (c + block_size - 1) / block_size * block_size;
      all += padded;
      if (b0 + i < me) before += padded;
      if (b0 + i == me) s_mine = c;
    }
    for (int o = 16; o > 0; o >>= 1) {
      before += __shfl_xor_sync(0xffffffffu, before, o);
      all += __shfl_xor_sync(0xffffffffu, all, o);
    }
    if (lane == 0) {
      atomicAdd(&s_start, before);
      atomicAdd(&s_total, all);
    }
  }
  __syncthreads();
  const int start = s_start, mine = s_mine, total = s_total;
  const int padded = (mine + block_size - 1) / block_size * block_size;
  const int sentinel = (topk << 24) | tokens;
  for (int i = tid; i < padded / block_size; i += threads) sorted_expert_ids[start / block_size + i] = me;
  for (int i = start + mine + tid; i < start + padded; i += threads) {
    sorted_ids[i] = sentinel;
    sorted_weights[i] = 0.0f;
  }
  const long long tail0 = static_cast<long long>(me) * threads + tid, tail_step = static_cast<long long>(experts) * threads;
  for (long long i = total + tail0; i < max_padded; i += tail_step) {
    sorted_ids[i] = sentinel;
    sorted_weights[i] = 0.0f;
  }
  for (long long i = total / block_size + tail0; i < max_blocks; i += tail_step) sorted_expert_ids[i] = -1;
  if (me == experts - 1 && tid == 0) {
    post_pad[0] = total;
    post_pad[1] = tokens;
  }
  int base = 0;  // pairs of this expert seen so far
  int buf = 0;
  for (long long c0 = 0; c0 < n_pairs && base < mine; c0 += 4 * threads) {
    const long long i = c0 + 4 * tid;
    int e[4];
    moe_load_ids(topk_ids, i, n_pairs, first_expert, experts, vec, e);
    int hits = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) hits += e[j] == me ? 1 : 0;
    int scan = hits;  // inclusive over the warp
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, scan, o);
      if (lane >= o) scan += up;
    }
    if (lane == 31) warp_sums[buf][warp] = scan;
    __syncthreads();  // two buffers: the next chunk writes the other one
    int ws = lane < warps ? warp_sums[buf][lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, ws, o);
      if (lane >= o) ws += up;
    }
    const int before_warp = warp == 0 ? 0 : __shfl_sync(0xffffffffu, ws, warp - 1);
    const int in_chunk = __shfl_sync(0xffffffffu, ws, 31);
    int dst = start + base + before_warp + scan - hits;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (e[j] == me) {
        const int pair = static_cast<int>(i) + j;
        sorted_ids[dst] = ((pair % topk) << 24) | (pair / topk);
        sorted_weights[dst] = __ldg(topk_weights + pair);
        ++dst;
      }
    }
    base += in_chunk;
    buf ^= 1;
  }
}

// y[t, :] = sum over the top-k slots of x[t, slot, :] (fp32 sum in slot order, one rounding).
// With a mask, slot k of token t counts only if expert_mask[topk_ids[t, k]] != 0
// (the expert-parallel validity mask of kernels/moe/moe_gemm_2stage/moe_reduce.py:3-7
// in the reference): rows of routes that another rank serves are never read.
//
// Memory-bound: the loads of up to four slots of all vectors of a thread are in flight together.  VEC = 8 (16-byte
// accesses) wherever `dim` and the bases allow it, else pairs; UNROLL = 2 where a row holds enough vectors, which
// halves the blocks.  WHOLE: blockIdx.x is the token, a thread owns UNROLL x VEC columns (vectors 256 apart), no division and
// no run-time stride.  Otherwise 2^log2_cols threads share a token, so that rows of a few vectors leave no warp idle,
// and rows past the grid's limit take further passes.  Measured, us, 4096 tokens x top-2 x 4096 bf16 (101 MB) as WHOLE 15.6 = 6.4 TB/s,
// in the other form 25.8, one pair per thread with a 64-bit division each 59; 20000 x top-2 x 256 WHOLE 25.5, other form 7.6, pairs 19.3.
template <typename T, int VEC, int UNROLL, typename I>
__device__ __forceinline__ void moe_reduce_columns(T* __restrict__ y, const T* __restrict__ x, long long t, int topk, int dim, I first, int step,
                                                   const int* __restrict__ expert_mask, const int* __restrict__ topk_ids, int num_experts) {
  float sum[UNROLL][VEC];
#pragma unroll
  for (int u = 0; u < UNROLL; ++u) {
#pragma unroll
    for (int i = 0; i < VEC; ++i) sum[u][i] = 0.0f;
  }
  constexpr int W = VEC / 2;  // 32-bit words of a vector
  for (int s0 = 0; s0 < topk; s0 += 4) {
    uint32_t v[4][UNROLL][W];
    bool on[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int s = s0 + j;
      on[j] = s < topk;
      if (on[j] && expert_mask != nullptr) {
        const int e = __ldg(topk_ids + t * topk + s);
        on[j] = e >= 0 && e < num_experts && __ldg(expert_mask + e) != 0;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (!on[j]) continue;
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        if (first + u * step >= dim) continue;
        const T* src = x + (t * topk + s0 + j) * dim + first + u * step;
        if constexpr (VEC == 8) {
          const uint4 q = __ldg(reinterpret_cast<const uint4*>(src));
          v[j][u][0] = q.x, v[j][u][1] = q.y, v[j][u][2] = q.z, v[j][u][3] = q.w;
        } else {
          v[j][u][0] = __ldg(reinterpret_cast<const uint32_t*>(src));
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (!on[j]) continue;
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
#pragma unroll
        for (int i = 0; i < W; ++i) {
          float2 f;
          if constexpr (std::is_same<T, __nv_bfloat16>::value) {
            f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v[j][u][i]));
          } else {
            f = __half22float2(*reinterpret_cast<const __half2*>(&v[j][u][i]));
          }
          sum[u][2 * i] += f.x;
          sum[u][2 * i + 1] += f.y;
        }
      }
    }
  }
#pragma unroll
  for (int u = 0; u < UNROLL; ++u) {
    const I c = first + u * step;
    if (c >= dim) break;
    uint32_t out[W];
#pragma unroll
    for (int i = 0; i < W; ++i) {
      if constexpr (std::is_same<T, __nv_bfloat16>::value) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(sum[u][2 * i], sum[u][2 * i + 1]);
        out[i] = *reinterpret_cast<const uint32_t*>(&h);
      } else {
        const __half2 h = __floats2half2_rn(sum[u][2 * i], sum[u][2 * i + 1]);
        out[i] = *reinterpret_cast<const uint32_t*>(&h);
      }
    }
    T* dst = y + t * dim + c;
    if constexpr (VEC == 8) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(out[0], out[1], out[2], out[3]);
    } else {
      *reinterpret_cast<uint32_t*>(dst) = out[0];
    }
  }
}
template <typename T, int VEC, int UNROLL, bool WHOLE>
__global__ void __launch_bounds__(256) moe_reduce_kernel(T* __restrict__ y, const T* __restrict__ x, int tokens, int topk, int dim,
                                                         int log2_cols, const int* __restrict__ expert_mask,
                                                         const int* __restrict__ topk_ids, int num_experts) {
  static_assert(VEC == 2 || VEC == 8, "pairs or 16-byte vectors");
  pdl_wait(y, x, expert_mask, topk_ids);
  pdl_trigger();
  if constexpr (WHOLE) {
    moe_reduce_columns<T, VEC, UNROLL, int>(y, x, blockIdx.x, topk, dim, (blockIdx.y * UNROLL * 256 + threadIdx.x) * VEC, 256 * VEC, expert_mask,
                                            topk_ids, num_experts);
  } else {
    const long long t = (static_cast<long long>(blockIdx.x) << (8 - log2_cols)) + (threadIdx.x >> log2_cols);
    if (t >= tokens) return;
    const int step = VEC << log2_cols;
    long long first = static_cast<long long>(blockIdx.y) * UNROLL * step + (threadIdx.x & ((1 << log2_cols) - 1)) * VEC;
    for (; first < dim; first += static_cast<long long>(gridDim.y) * UNROLL * step)
      moe_reduce_columns<T, VEC, UNROLL, long long>(y, x, t, topk, dim, first, step, expert_mask, topk_ids, num_experts);
  }
}

}  // namespace flyb200
