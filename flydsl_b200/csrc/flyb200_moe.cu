// libflyb200: host side of the grouped (mixture-of-experts) entry points of
// include/flyb200.h — argument checks, tensor map, kernel selection, launch.
#include "../../include/flyb200.h"
#include "host_common.h"
#include "moe_pair_kernel.cuh"

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <type_traits>

using namespace flyb200;

namespace {

#define CUDA_TRY(expr)                                                  \
  do {                                                                  \
    cudaError_t _e = (expr);                                            \
    if (_e != cudaSuccess) return host::record_cuda_error(_e, #expr);   \
  } while (0)

constexpr int SMEM_LIMIT = 232448;  // 227 KiB of dynamic shared memory per CTA

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Ring depth.  Up to 128 tokens per block two CTAs share an SM (half of its
// shared memory and of its 512 TMEM columns each), so that one CTA's set-up and
// epilogue overlap the other's mainloop and a grid of up to 296 CTAs runs as one
// wave; 256-token blocks need all TMEM columns and get the whole SM.
inline int moe_stages(int bn) {
  const int stage = 2 * BLOCK_ROWS * KBLOCK_BYTES + bn * KBLOCK_BYTES;
  const int budget = bn <= 128 ? (SMEM_LIMIT + 1024) / 2 - 1024 : SMEM_LIMIT;
  int n = (budget - 1024 - 12 * bn) / stage;
  return n > 8 ? 8 : n;
}

template <int KIND, int BN, int STAGE, int OUTMODE, bool ACCUM>
int launch_moe(const CUtensorMap& tmA, MoeParams p, int blocks, cudaStream_t s) {
  static std::atomic<uint64_t> done{0};
  auto kernel = moe_gemm_kernel<KIND, BN, STAGE, OUTMODE, ACCUM>;
  int dev = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << dev;
  if (!(done.load(std::memory_order_acquire) & bit)) {
    CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT));
    done.fetch_or(bit, std::memory_order_release);
  }
  p.stages = moe_stages(BN);
  const MoeLayout L = moe_layout(BN, p.stages);
  if (p.stages < 2 || L.total > SMEM_LIMIT) return FLYB200_E_UNSUPPORTED;
  const int tiles = STAGE == 1 ? (p.n_out + BLOCK_ROWS - 1) / BLOCK_ROWS : (p.n_out + 2 * BLOCK_ROWS - 1) / (2 * BLOCK_ROWS);
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(blocks, tiles, 1);
  cfg.blockDim = dim3(MOE_THREADS, 1, 1);
  cfg.dynamicSmemBytes = L.total;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = p.pdl ? 1 : 0;
  CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, tmA, p));
  return FLYB200_OK;
}

int sm_count(int* out) {
  static std::atomic<int> cached[64];
  int dev = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return FLYB200_E_UNSUPPORTED;
  int n = cached[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    CUDA_TRY(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    cached[dev].store(n, std::memory_order_relaxed);
  }
  *out = n;
  return FLYB200_OK;
}

// CTA pairs on up to 256 rows of an expert.
template <int KIND, int STAGE, int OUTMODE, bool ACCUM>
int launch_moe_pair(const CUtensorMap& tmA, const MoePairWeights& tmW, const MoeParams& p, int blocks, int sms, cudaStream_t s) {
  static std::atomic<uint64_t> done{0};
  auto kernel = moe_pair_kernel<KIND, STAGE, OUTMODE, ACCUM>;
  int dev = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << dev;
  if (!(done.load(std::memory_order_acquire) & bit)) {
    CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MoePairSmem::TOTAL));
    done.fetch_or(bit, std::memory_order_release);
  }
  const int pairs = STAGE == 1 ? (p.n_out + BLOCK_ROWS - 1) / BLOCK_ROWS : (p.n_out + MOE_ROWS_BN - 1) / MOE_ROWS_BN;
  const long long items = static_cast<long long>(blocks) * pairs;  // at most: a tile holds a routing block or more
  const int clusters = static_cast<int>(items < sms / 2 ? items : sms / 2);
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(2 * clusters, 1, 1);
  cfg.blockDim = dim3(moe_rows_threads(STAGE), 1, 1);
  cfg.dynamicSmemBytes = MoePairSmem::TOTAL;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = host::pdl_default() != 0 ? 2 : 1;
  CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, tmA, tmW, p));
  return FLYB200_OK;
}

// Persistent form for routing blocks that are a multiple of 128 rows.
template <int KIND, int STAGE, int OUTMODE, bool ACCUM>
int launch_moe_rows(const CUtensorMap& tmA, const MoeParams& p, int blocks, int sms, cudaStream_t s) {
  static std::atomic<uint64_t> done{0};
  auto kernel = moe_rows_kernel<KIND, STAGE, OUTMODE, ACCUM>;
  int dev = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << dev;
  if (!(done.load(std::memory_order_acquire) & bit)) {
    CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MoeRowsSmem::TOTAL));
    done.fetch_or(bit, std::memory_order_release);
  }
  const long long row_blocks = (static_cast<long long>(blocks) * p.tile_m + BLOCK_ROWS - 1) / BLOCK_ROWS;
  const int pairs = STAGE == 1 ? (p.n_out + BLOCK_ROWS - 1) / BLOCK_ROWS : (p.n_out + MOE_ROWS_BN - 1) / MOE_ROWS_BN;
  const long long items = row_blocks * pairs;
  const int grid = static_cast<int>(items < sms ? items : sms);
  CUDA_TRY(host::launch_dependent(kernel, dim3(grid), moe_rows_threads(STAGE), MoeRowsSmem::TOTAL, s, tmA, p));
  return FLYB200_OK;
}

// tmW: the weight images' maps for CTA pairs, or null for one CTA per item.
template <int KIND, int STAGE, int OUTMODE, bool ACCUM>
int launch_moe_large(const CUtensorMap& tmA, const MoePairWeights* tmW, const MoeParams& p, int blocks, int sms, cudaStream_t s) {
  return tmW ? launch_moe_pair<KIND, STAGE, OUTMODE, ACCUM>(tmA, *tmW, p, blocks, sms, s)
             : launch_moe_rows<KIND, STAGE, OUTMODE, ACCUM>(tmA, p, blocks, sms, s);
}
template <int KIND>
int launch_moe_large_variant(int stage, int out_dtype, bool accumulate, const CUtensorMap& tmA, const MoePairWeights* tmW, const MoeParams& p,
                             int blocks, int sms, cudaStream_t s) {
  if (stage == 1) {
    if (out_dtype == FLYB200_OUT_BF16) return launch_moe_large<KIND, 1, MOE_OUT_BF16, false>(tmA, tmW, p, blocks, sms, s);
    if (out_dtype == FLYB200_OUT_FP16) return launch_moe_large<KIND, 1, MOE_OUT_FP16, false>(tmA, tmW, p, blocks, sms, s);
    return FLYB200_E_UNSUPPORTED;
  }
  if (accumulate) {
    if (out_dtype == FLYB200_OUT_BF16) return launch_moe_large<KIND, 2, MOE_OUT_BF16, true>(tmA, tmW, p, blocks, sms, s);
    if (out_dtype == FLYB200_OUT_FP16) return launch_moe_large<KIND, 2, MOE_OUT_FP16, true>(tmA, tmW, p, blocks, sms, s);
    if (out_dtype == FLYB200_OUT_F32) return launch_moe_large<KIND, 2, MOE_OUT_F32, true>(tmA, tmW, p, blocks, sms, s);
    return FLYB200_E_UNSUPPORTED;
  }
  if (out_dtype == FLYB200_OUT_BF16) return launch_moe_large<KIND, 2, MOE_OUT_BF16, false>(tmA, tmW, p, blocks, sms, s);
  if (out_dtype == FLYB200_OUT_FP16) return launch_moe_large<KIND, 2, MOE_OUT_FP16, false>(tmA, tmW, p, blocks, sms, s);
  return FLYB200_E_UNSUPPORTED;
}

// Estimated time (us, the gather pass left out) of a stage on CTA pairs, or with one CTA per 128-row item.  How the routes fall on the
// experts is known on the device only, so the estimate spreads `routes` evenly: 128-row items (routing blocks of 64 make one more
// pass where the expert changes inside an item) or 256-row tiles per expert, rounds of them over the SMs with a part of a
// last one, per k-block and per item a time, at least the weights at 6.5 TB/s.
// Fitted to 5038 drawn layers (16..8192 tokens, top-1..8, 8..128 experts of which a rank serves all, a half, a quarter or an eighth, 1024..7168 x
// 512..4096, routing blocks of 64..256, graph replay, weights rotated past L2).  The form with the smaller estimate is on average 1.0 / 1.0 %
// (gate-up / down) behind the better one where all experts are served and 1.5 / 1.2 % on a rank's share, 53 % at worst; always
// pairs 3.8 / 10.0 and 6.8 / 12.2 %, always one CTA 7.9 / 5.0 and 5.2 / 2.9 %.  With all ranks' routes counted on a share 2.6 / 1.9 %.  One
// CTA / pairs, us, gather included: 4096 tokens x top-2, 8 experts, 4096 x 2048 128 / 122 and 74 / 67 (gate-up, down), 800 x top-4, 32
// experts, 3072 x 1536 91 / 65 and 48 / 41, 515 x top-4, 16 experts, 2048 x 1408 32.6 / 30.7 and 24.4 / 21.0; where items are few and the
// weights fit L2, or K is short, it is the other way round: 1024 x top-4, 8 experts, 2048 x 1024, down 19.2 / 20.0, 4096 x top-4, 32 experts, 2048 x
// 768, down 43.0 / 51.2.
double moe_form_us(bool pairs, int stage, double routes, int experts, int n_out, int num_kb, int tile_m, int sms) {
  const bool up = stage == 1;
  const double used = routes < 1.0 ? 1.0 : routes < experts ? routes : experts, rows = routes / used;
  const int columns = up ? (n_out + 127) / 128 : (n_out + 255) / 256;
  const double weights = used * n_out * (up ? 2 : 1) * num_kb * KBLOCK_BYTES / 6.5e6;
  double rounds, item, fixed;
  if (pairs) {
    const double tiles = rows / 256 + (up ? 0.6 : 0.55);
    rounds = used * (tiles < 1.0 ? 1.0 : tiles) * columns / (sms / 2) + 0.45;
    item = up ? num_kb * 0.26 + 1.9 : num_kb * 0.28 + 3.1;
    fixed = up ? 7.8 : 5.7;
  } else {
    const double more = tile_m == 64 ? (up ? 1.55 : 1.35) : tile_m == 128 ? (up ? 1.0 : 0.95) : (up ? 1.5 : 1.0);
    rounds = used * (rows / 128 + more) * columns / sms + (up ? 0.85 : 0.5);
    item = up ? num_kb * 0.39 + 0.4 : num_kb * 0.45 + 1.6;
    fixed = 3.7;
  }
  const double work = (rounds < 1.0 ? 1.0 : rounds) * item;
  return fixed + (work > weights ? work : weights);
}

// Kernel for routing blocks of tile_m rows when nothing forces one, numbered as in FLYB200_MOE_KERNEL: 1 two weight tiles per CTA,
// 2 one CTA per 128-row item, 3 CTA pairs (while the list of their tiles fits shared memory).  `all_experts`: of which the
// `experts` of this call get their share of the routes.
int moe_form(int stage, int tokens, int topk, int experts, int all_experts, int model_dim, int inter_dim, int tile_m, int blocks, int sms) {
  if (tile_m % BLOCK_ROWS != 0 && tile_m != 64) return 1;
  if (blocks > MOE_PAIR_MAX_BLOCKS || sms < 2) return 2;
  const double routes = static_cast<double>(tokens) * topk * experts / all_experts;
  const int n_out = stage == 1 ? inter_dim : model_dim, num_kb = (stage == 1 ? model_dim : inter_dim) / KBLOCK_BYTES;
  auto us = [&](bool pairs) { return moe_form_us(pairs, stage, routes, experts, n_out, num_kb, tile_m, sms); };
  return us(true) < us(false) ? 3 : 2;
}

template <int KIND, int BN>
int launch_moe_variant(int stage, int out_dtype, bool accumulate, const CUtensorMap& tmA, const MoeParams& p, int blocks,
                       cudaStream_t s) {
  if (stage == 1) {
    if (out_dtype == FLYB200_OUT_BF16) return launch_moe<KIND, BN, 1, MOE_OUT_BF16, false>(tmA, p, blocks, s);
    if (out_dtype == FLYB200_OUT_FP16) return launch_moe<KIND, BN, 1, MOE_OUT_FP16, false>(tmA, p, blocks, s);
    return FLYB200_E_UNSUPPORTED;
  }
  if (accumulate) {
    if (out_dtype == FLYB200_OUT_BF16) return launch_moe<KIND, BN, 2, MOE_OUT_BF16, true>(tmA, p, blocks, s);
    if (out_dtype == FLYB200_OUT_FP16) return launch_moe<KIND, BN, 2, MOE_OUT_FP16, true>(tmA, p, blocks, s);
    if (out_dtype == FLYB200_OUT_F32) return launch_moe<KIND, BN, 2, MOE_OUT_F32, true>(tmA, p, blocks, s);
    return FLYB200_E_UNSUPPORTED;
  }
  if (out_dtype == FLYB200_OUT_BF16) return launch_moe<KIND, BN, 2, MOE_OUT_BF16, false>(tmA, p, blocks, s);
  if (out_dtype == FLYB200_OUT_FP16) return launch_moe<KIND, BN, 2, MOE_OUT_FP16, false>(tmA, p, blocks, s);
  return FLYB200_E_UNSUPPORTED;  // per-slot partials are 16-bit only, as in the reference
}

template <int KIND>
int launch_moe_bn(int bn, int stage, int out_dtype, bool accumulate, const CUtensorMap& tmA, const MoeParams& p,
                  int blocks, cudaStream_t s) {
  switch (bn) {
    case 16: return launch_moe_variant<KIND, 16>(stage, out_dtype, accumulate, tmA, p, blocks, s);
    case 32: return launch_moe_variant<KIND, 32>(stage, out_dtype, accumulate, tmA, p, blocks, s);
    case 64: return launch_moe_variant<KIND, 64>(stage, out_dtype, accumulate, tmA, p, blocks, s);
    case 128: return launch_moe_variant<KIND, 128>(stage, out_dtype, accumulate, tmA, p, blocks, s);
    case 256: return launch_moe_variant<KIND, 256>(stage, out_dtype, accumulate, tmA, p, blocks, s);
  }
  return FLYB200_E_UNSUPPORTED;
}

// Vectors of eight where every row starts on a 16-byte boundary, else pairs; a block per token where its threads have
// work for half a block and more and the grid holds the columns.
template <typename T, int VEC, int UNROLL>
cudaError_t launch_moe_reduce_form(T* y, const T* x, int tokens, int topk, int dim, const int* expert_mask, const int* topk_ids, int num_experts,
                                   cudaStream_t s) {
  const int vecs = dim / VEC;
  int log2_cols = 8;
  while (log2_cols > 0 && vecs <= (128 >> (8 - log2_cols))) --log2_cols;  // threads per token: vecs rounded up to a power of two
  const int per_block = 256 >> log2_cols;                                 // tokens
  const int column_blocks = (vecs - 1) / (UNROLL << log2_cols) + 1;
  const dim3 grid((tokens - 1) / per_block + 1, column_blocks < 65535 ? column_blocks : 65535);
  auto kernel = log2_cols == 8 && column_blocks <= 65535 ? moe_reduce_kernel<T, VEC, UNROLL, true> : moe_reduce_kernel<T, VEC, UNROLL, false>;
  return host::launch_dependent(kernel, grid, 256, 0, s, y, x, tokens, topk, dim, log2_cols, expert_mask, topk_ids, num_experts);
}
template <typename T>
cudaError_t launch_moe_reduce(void* y, const void* x, int tokens, int topk, int dim, const int* expert_mask, const int* topk_ids,
                              int num_experts, cudaStream_t s) {
  T* yt = static_cast<T*>(y);
  const T* xt = static_cast<const T*>(x);
  auto launch = [&](auto form) { return form(yt, xt, tokens, topk, dim, expert_mask, topk_ids, num_experts, s); };
  if (dim % 8 != 0 || !aligned16(y) || !aligned16(x)) return launch(launch_moe_reduce_form<T, 2, 1>);
  return dim > 8 * 256 && tokens > 256 ? launch(launch_moe_reduce_form<T, 8, 2>) : launch(launch_moe_reduce_form<T, 8, 1>);
}

}  // namespace

extern "C" {

int flyb200_moe_gather_rows(void* dst, float* dst_scale, const void* src, const float* src_scale, const int* sorted_ids,
                            const int* num_valid_ids, int tokens, int topk, int by_slot, int row_bytes, int rows,
                            void* stream) {
  if (!dst || !dst_scale || !src || !src_scale || !sorted_ids || !num_valid_ids) return FLYB200_E_BAD_ARG;
  if (tokens < 0 || topk <= 0 || topk > 255 || row_bytes <= 0 || rows < 0 || by_slot < 0 || by_slot > 2)
    return FLYB200_E_BAD_ARG;
  if (row_bytes % 16 != 0) return FLYB200_E_UNSUPPORTED;
  if (!aligned16(dst) || !aligned16(src)) return FLYB200_E_BAD_ALIGN;
  if (rows == 0) return FLYB200_OK;
  const int warps = 8;
  int grid = (rows + warps - 1) / warps;
  if (grid > 148 * 8) grid = 148 * 8;
  CUDA_TRY(host::launch_dependent(moe_gather_rows_kernel, dim3(grid), warps * 32, 0, static_cast<cudaStream_t>(stream),
                                  static_cast<uint8_t*>(dst), dst_scale, static_cast<const uint8_t*>(src), src_scale, sorted_ids,
                                  num_valid_ids, tokens, topk, by_slot, row_bytes, rows));
  return FLYB200_OK;
}

int flyb200_moe_quant_sorted(void* dst, float* dst_scale, const void* src, const int* sorted_ids, const int* num_valid_ids,
                             int tokens, int topk, int K, int rows, int quant_dtype, void* stream) {
  if (!dst || !dst_scale || !src || !sorted_ids || !num_valid_ids) return FLYB200_E_BAD_ARG;
  if (tokens < 0 || topk <= 0 || topk > 255 || K <= 0 || rows < 0) return FLYB200_E_BAD_ARG;
  if (quant_dtype != FLYB200_DT_FP8 && quant_dtype != FLYB200_DT_INT8) return FLYB200_E_BAD_ARG;
  if (K % 16 != 0 || K > FLYB200_MOE_QUANT_MAX_K) return FLYB200_E_UNSUPPORTED;
  if (!aligned16(dst) || !aligned16(src)) return FLYB200_E_BAD_ALIGN;
  if (rows == 0) return FLYB200_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t err = cudaSuccess;
  quant_row_dispatch(rows, K / 8, [&](auto nv, auto wpr) {
    constexpr int NV = decltype(nv)::value, WPR = decltype(wpr)::value;
    const int grid = (rows + 8 / WPR - 1) / (8 / WPR);
    const __nv_bfloat16* x = static_cast<const __nv_bfloat16*>(src);
    uint8_t* y = static_cast<uint8_t*>(dst);
    err = host::launch_dependent(quant_dtype == FLYB200_DT_FP8 ? moe_quant_sorted_kernel<true, NV, WPR> : moe_quant_sorted_kernel<false, NV, WPR>,
                                 dim3(grid), 256, 0, s, y, dst_scale, x, sorted_ids, num_valid_ids, tokens, topk, K, rows);
  });
  CUDA_TRY(err);
  return FLYB200_OK;
}

int flyb200_moe_form(int stage, int tokens, int topk, int experts, int all_experts, int model_dim, int inter_dim, int tile_m,
                     int blocks, int sm_count) {
  if ((stage != 1 && stage != 2) || tokens <= 0 || topk <= 0 || experts <= 0 || all_experts < experts || model_dim <= 0 || inter_dim <= 0 ||
      tile_m < 16 || tile_m > 256 || tile_m % 16 != 0 || blocks <= 0 || sm_count <= 0)
    return 0;
  return moe_form(stage, tokens, topk, experts, all_experts, model_dim, inter_dim, tile_m, blocks, sm_count);
}

int flyb200_moe_gemm(int stage, void* out, const void* a_sorted, const void* w_shuf, const float* scale_a_sorted,
                     const float* scale_w, const int* sorted_ids, const int* expert_ids, const float* sorted_weights,
                     const int* num_valid_ids, int tokens, int topk, int experts, int model_dim, int inter_dim,
                     int tile_m, int blocks, int in_dtype, int out_dtype, int doweight, int accumulate, int after_gather,
                     void* stream) {
  return flyb200_moe_gemm_shard(stage, out, a_sorted, w_shuf, scale_a_sorted, scale_w, sorted_ids, expert_ids, sorted_weights, num_valid_ids,
                                tokens, topk, experts, experts, model_dim, inter_dim, tile_m, blocks, in_dtype, out_dtype, doweight,
                                accumulate, after_gather, stream);
}

int flyb200_moe_gemm_shard(int stage, void* out, const void* a_sorted, const void* w_shuf, const float* scale_a_sorted,
                           const float* scale_w, const int* sorted_ids, const int* expert_ids, const float* sorted_weights,
                           const int* num_valid_ids, int tokens, int topk, int experts, int all_experts, int model_dim, int inter_dim,
                           int tile_m, int blocks, int in_dtype, int out_dtype, int doweight, int accumulate, int after_gather,
                           void* stream) {
  if (stage != 1 && stage != 2) return FLYB200_E_BAD_ARG;
  if (!out || !a_sorted || !w_shuf || !scale_a_sorted || !scale_w || !sorted_ids || !expert_ids || !num_valid_ids)
    return FLYB200_E_BAD_ARG;
  if (doweight && !sorted_weights) return FLYB200_E_BAD_ARG;
  if (tokens < 0 || topk <= 0 || topk > 255 || experts <= 0 || all_experts < experts || model_dim <= 0 || inter_dim <= 0 || blocks < 0)
    return FLYB200_E_BAD_ARG;
  if (tokens >= (1 << 24)) return FLYB200_E_UNSUPPORTED;  // a sorted id keeps the token in 24 bits
  if (in_dtype != FLYB200_DT_FP8 && in_dtype != FLYB200_DT_INT8) return FLYB200_E_UNSUPPORTED;
  if (tile_m < 16 || tile_m > 256 || tile_m % 16 != 0) return FLYB200_E_BAD_ARG;
  if (stage == 1 && accumulate) return FLYB200_E_BAD_ARG;
  const int K = stage == 1 ? model_dim : inter_dim;
  const int n_out = stage == 1 ? inter_dim : model_dim;
  if (K % KBLOCK_BYTES != 0 || n_out % 16 != 0) return FLYB200_E_UNSUPPORTED;
  if (!aligned16(out) || !aligned16(a_sorted) || !aligned16(w_shuf)) return FLYB200_E_BAD_ALIGN;
  if (blocks == 0 || tokens == 0) return FLYB200_OK;

  MoeParams p;
  memset(&p, 0, sizeof(p));
  p.w = static_cast<const uint8_t*>(w_shuf);
  p.sa = scale_a_sorted;
  p.sw = scale_w;
  p.sorted_ids = sorted_ids;
  p.expert_ids = expert_ids;
  p.sorted_w = sorted_weights;
  p.num_valid = num_valid_ids;
  p.out = out;
  p.tokens = tokens;
  p.topk = topk;
  p.experts = experts;
  p.n_expert = stage == 1 ? 2 * inter_dim : model_dim;
  p.n_out = n_out;
  p.K_bytes = K;
  p.tile_m = tile_m;
  p.doweight = doweight ? 1 : 0;
  p.pdl = 0;
  int rc = host::status_word(&p.status);
  if (rc) return rc;

  cudaStream_t s = static_cast<cudaStream_t>(stream);
  CUtensorMap tmA;
  // Routing blocks of 64, 128 or 256 rows: persistent kernel with the tokens on the
  // UMMA M side (FLYB200_MOE_KERNEL=1 in the environment forces the other form, 2 one CTA per item, 3 CTA pairs, for
  // tests and tuning).
  const char* force = getenv("FLYB200_MOE_KERNEL");
  const bool rows_form = (tile_m % BLOCK_ROWS == 0 || tile_m == 64) && !(force && force[0] == '1');
  if (rows_form) {
    int sms = 0;
    if ((rc = sm_count(&sms))) return rc;
    rc = host::byte_matrix_map(&tmA, a_sorted, static_cast<uint64_t>(K), static_cast<uint64_t>(blocks) * tile_m, BLOCK_ROWS);
    if (rc) return rc;
    const int form = moe_form(stage, tokens, topk, experts, all_experts, model_dim, inter_dim, tile_m, blocks, sms);
    const bool pair = force && (force[0] == '2' || force[0] == '3') ? force[0] == '3' && blocks <= MOE_PAIR_MAX_BLOCKS && sms > 1 : form == 3;
    MoePairWeights tmW;
    for (int i = 0; pair && i < 3; ++i) {
      rc = host::weight_image_map(&tmW.box[i], w_shuf, static_cast<uint64_t>(p.n_expert), static_cast<uint64_t>(experts) * (K / KBLOCK_BYTES), BLOCK_ROWS >> i);
      if (rc) return rc;
    }
    p.pdl = pair && after_gather && host::pdl_default() != 0 ? 1 : 0;
    const MoePairWeights* w_map = pair ? &tmW : nullptr;
    if (in_dtype == FLYB200_DT_FP8) return launch_moe_large_variant<KIND_F8>(stage, out_dtype, accumulate != 0, tmA, w_map, p, blocks, sms, s);
    return launch_moe_large_variant<KIND_I8>(stage, out_dtype, accumulate != 0, tmA, w_map, p, blocks, sms, s);
  }
  int bn = 16;
  while (bn < tile_m) bn *= 2;
  p.pdl = after_gather && host::pdl_default() != 0 ? 1 : 0;
  rc = host::byte_matrix_map(&tmA, a_sorted, static_cast<uint64_t>(K), static_cast<uint64_t>(blocks) * tile_m, bn);
  if (rc) return rc;
  if (in_dtype == FLYB200_DT_FP8) return launch_moe_bn<KIND_F8>(bn, stage, out_dtype, accumulate != 0, tmA, p, blocks, s);
  return launch_moe_bn<KIND_I8>(bn, stage, out_dtype, accumulate != 0, tmA, p, blocks, s);
}

int flyb200_moe_sorting_range(const void* topk_ids, int id_bytes, const float* topk_weights, int tokens, int topk, int experts,
                              long long first_expert, int block_size, int* sorted_ids, float* sorted_weights,
                              int* sorted_expert_ids, int* num_tokens_post_pad, void* stream) {
  if (!topk_ids || !topk_weights || !sorted_ids || !sorted_weights || !sorted_expert_ids || !num_tokens_post_pad)
    return FLYB200_E_BAD_ARG;
  if (id_bytes != 4 && id_bytes != 8) return FLYB200_E_BAD_ARG;
  if (tokens < 0 || topk <= 0 || topk > 255 || experts <= 0 || block_size <= 0 || first_expert < 0) return FLYB200_E_BAD_ARG;
  if (tokens >= (1 << 24)) return FLYB200_E_UNSUPPORTED;
  const long long n_pairs = static_cast<long long>(tokens) * topk;
  const long long max_padded = n_pairs + static_cast<long long>(experts) * block_size - topk;
  if (max_padded > 0x7fffffffLL || max_padded <= 0) return FLYB200_E_UNSUPPORTED;
  const int max_blocks = static_cast<int>((max_padded + block_size - 1) / block_size);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // four pairs per thread, and enough threads for the histogram and the padding of small calls
  long long threads = (n_pairs / 4 + 31) / 32 * 32;
  threads = threads < 128 ? 128 : threads > MOE_SORT_MAX_THREADS ? MOE_SORT_MAX_THREADS : threads;
  auto launch = [&](auto* ids) {
    using ID = std::remove_const_t<std::remove_pointer_t<decltype(ids)>>;
    return host::launch_dependent(moe_sort_kernel<ID>, dim3(experts), static_cast<int>(threads), 0, s, ids, topk_weights,
                                  static_cast<int>(n_pairs), topk, tokens, experts, first_expert, block_size, sorted_ids, sorted_weights,
                                  sorted_expert_ids, num_tokens_post_pad, static_cast<int>(max_padded), max_blocks);
  };
  CUDA_TRY(id_bytes == 4 ? launch(static_cast<const int*>(topk_ids)) : launch(static_cast<const long long*>(topk_ids)));
  return FLYB200_OK;
}

int flyb200_moe_sorting(const int* topk_ids, const float* topk_weights, int tokens, int topk, int experts, int block_size,
                        int* sorted_ids, float* sorted_weights, int* sorted_expert_ids, int* num_tokens_post_pad,
                        int* counts_scratch, void* stream) {
  if (!counts_scratch) return FLYB200_E_BAD_ARG;
  return flyb200_moe_sorting_range(topk_ids, 4, topk_weights, tokens, topk, experts, 0, block_size, sorted_ids, sorted_weights,
                                   sorted_expert_ids, num_tokens_post_pad, stream);
}

int flyb200_moe_reduce(void* y, const void* x, int tokens, int topk, int dim, int dtype, const int* expert_mask,
                       const int* topk_ids, int num_experts, void* stream) {
  if (!y || !x || tokens < 0 || topk <= 0 || dim <= 0) return FLYB200_E_BAD_ARG;
  if (expert_mask && (!topk_ids || num_experts <= 0)) return FLYB200_E_BAD_ARG;
  if (dim % 2 != 0) return FLYB200_E_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(y) & 3u) || (reinterpret_cast<uintptr_t>(x) & 3u)) return FLYB200_E_BAD_ALIGN;
  if (tokens == 0) return FLYB200_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype != FLYB200_OUT_BF16 && dtype != FLYB200_OUT_FP16) return FLYB200_E_UNSUPPORTED;
  if (dtype == FLYB200_OUT_BF16) CUDA_TRY(launch_moe_reduce<__nv_bfloat16>(y, x, tokens, topk, dim, expert_mask, topk_ids, num_experts, s));
  else CUDA_TRY(launch_moe_reduce<__half>(y, x, tokens, topk, dim, expert_mask, topk_ids, num_experts, s));
  return FLYB200_OK;
}

}  // extern "C"
