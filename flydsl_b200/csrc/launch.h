// Kernel launchers of libflyb200, one translation unit per kernel family so
// that the families compile in parallel (not part of the C ABI).
#pragma once
#include "decode_kernel.cuh"
#include "host_common.h"
#include "rows2_kernel.cuh"

#include <atomic>
#include <cstdlib>

namespace flyb200 {
namespace host {

constexpr int SMEM_LIMIT = 232448;  // 227 KiB of dynamic shared memory per CTA
constexpr int MAX_DEVICES = 64;
constexpr int ROWS_MAX_STAGES = 8;

#define FLYB200_CUDA_TRY(expr)                                                          \
  do {                                                                                  \
    cudaError_t _e = (expr);                                                            \
    if (_e != cudaSuccess) return ::flyb200::host::record_cuda_error(_e, #expr);        \
  } while (0)

// One-time (per device) opt-in to large dynamic shared memory for a kernel.
template <typename KernelT>
int ensure_smem(KernelT kernel, int bytes, std::atomic<uint64_t>& done) {
  int dev = 0;
  FLYB200_CUDA_TRY(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << dev;
  if (done.load(std::memory_order_acquire) & bit) return 0;
  FLYB200_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  done.fetch_or(bit, std::memory_order_release);
  return 0;
}

// Deepest ring (at most ROWS_MAX_STAGES) of the large-M kernel that fits shared memory for a tile width.
inline int rows_stages_for(int bn) {
  int s = ROWS_MAX_STAGES;
  while (s > 2 && rows_layout(bn, s).total > SMEM_LIMIT) --s;
  return s;
}

// Column strips of the tiles of the large-M kernel's last round, where that is at most half full (1: none): two or
// four strips per tile while every SM gets at most one; strips are multiples of 64 columns (the stores' box).  At one
// width the gain is small, as the round is short of power rather than of time (fewer busy SMs clock higher): whole tiles /
// strips, us, fp16 4096 x 4096 x 4096 (3.46 rounds of tiles) 104.1 / 102.8, fp8 55.4 / 54.2.  But strips also make 256-column tiles
// of a little more than whole rounds pay, which the planner then prefers to narrower ones in whole rounds: 96 shapes
// (512..8192 x 3584..28672, K = 2048..8192, fp8 and bf16) whose width changed from 192 or 224 to 256 take 0.85..1.07 of the time
// (median 0.96; fp8 4096 x 6144 x 2048 55.7 -> 47.2, bf16 3000 x 3584 x 4096 84.1 -> 89.7).
inline int rows_tail_parts(int bn, long long tiles, int sms) {
  const long long rest = tiles % sms;
  if (tiles < sms || rest == 0 || bn % 128 != 0) return 1;
  if (bn == 256 && 4 * rest <= sms) return 4;
  return 2 * rest <= sms ? 2 : 1;
}

// Pair form: ring depth for a tile width, and the number of 256 x bn tiles.
inline int pair_stages_for(int bn) {
  int s = ROWS_MAX_STAGES;
  while (s > 2 && pair_layout(bn, s).total > SMEM_LIMIT) --s;
  return s;
}
inline long long pair_tiles(int M, int N, int bn) {
  return static_cast<long long>((M + PAIR_ROWS - 1) / PAIR_ROWS) * ((N + bn - 1) / bn);
}
// Cycles a pair spends on one k-block of a tile or strip: the tensor pipe, or the bytes each SM takes in.
inline long long pair_kb_cycles(int width) {
  const long long mma = 2LL * width, load = (BLOCK_ROWS + width / 2) * KBLOCK_BYTES / 72;
  return mma > load ? mma : load;
}
// Column strips of the tiles of the last, partial round: the number that makes it shortest.
inline int pair_tail_parts(int bn, long long tiles, int clusters) {
  const long long rest = tiles % clusters;
  if (tiles < clusters || rest == 0) return 1;
  int best = 1;
  long long best_cycles = pair_kb_cycles(bn);
  for (int parts = 2; parts <= 4 && bn % (64 * parts) == 0; parts *= 2) {
    const long long c = (rest * parts + clusters - 1) / clusters * pair_kb_cycles(bn / parts);
    if (c < best_cycles) {
      best_cycles = c;
      best = parts;
    }
  }
  return best;
}

// Epilogue warps of the large-M kernel.  With few k-blocks a tile's epilogue is as long as the mainloop that it overlaps,
// and in a launch of few rounds the last one is exposed: eight warps.  In long launches over 32 k-blocks and more the
// epilogue is hidden either way and four warps leave more power to the tensor cores.  Eight / four, us, fp8:
// K = 1024 4096 x 14336 74.5 / 108, K = 2048 with silu 2048 x 8192 46.5 / 58.8; K = 8192 (at the power cap) 8192 x 28672 1539 / 1519, with gelu 1587 / 1431,
// 16384 x 57344 6081 / 5989.
// FLYB200_ROWS_EPI = 4 or 8 forces the number (tuning and tests).
inline int rows_epilogue_warps(int kb, long long tiles, int sms) {
  if (const char* e = getenv("FLYB200_ROWS_EPI"))
    if (e[0] == '4' || e[0] == '8') return e[0] - '0';
  return kb >= 32 && tiles >= 8LL * sms ? 4 : 8;
}

// Large-M kernel (p.bn, p.rows_stages, p.tail_parts set): one CTA per 128 x bn tile, or per 256 x bn tile (tmA with boxes of 256
// rows, three stages).  `kind` is KIND_*, `outmode` OUT_*.
enum : int { ROWS_FORM_ONE = 0, ROWS_FORM_TALL = 2 };
constexpr int ROWS_TALL_STAGES = 3;
int launch_rows_kind(int kind, int outmode, int form, const CUtensorMap& tmA, const CUtensorMap& tmC, const GemmParams& p,
                     int sms, cudaStream_t s);
// Large-M kernel, CTA pairs on 256 x bn tiles (p.bn, p.rows_stages, p.tail_parts set).
int launch_pair_kind(int kind, int outmode, const PairMaps& maps, const GemmParams& p, int sms, cudaStream_t s);
// Large-M kernel storing every tile through p.n_dst output maps.
int launch_rows_scatter_kind(int kind, int outmode, const CUtensorMap& tmA, const OutputMaps& outs, const GemmParams& p,
                             int sms, cudaStream_t s);
// Small-M kernel for a token block of `bn` and weight tiles of `w_rows` channels.
int launch_decode_kind(int kind, int outmode, int bn, int w_rows, const CUtensorMap& tmA, const GemmParams& p,
                       cudaStream_t s);

// Small-M kernel as CTA pairs (256 channels x `bn` tokens per pair, `bn` = 64, 128 or 256); `tmA` has boxes of bn / 2
// tokens.  Needs an even number of channel tiles and an even ring depth.
int launch_decode2_kind(int kind, int outmode, int bn, const CUtensorMap& tmA, const GemmParams& p, cudaStream_t s);

}  // namespace host
}  // namespace flyb200
