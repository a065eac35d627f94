// libflyb200: host side of the MXFP8 (block-scaled) entry points of
// include/flyb200.h — argument checks, tensor map, launch.
#include "../../include/flyb200.h"
#include "host_common.h"
#include "mx_kernel.cuh"
#include "mx_quant_kernel.cuh"

#include <atomic>
#include <cstdlib>
#include <cstring>

using namespace flyb200;

namespace {

#define CUDA_TRY(expr)                                                  \
  do {                                                                  \
    cudaError_t _e = (expr);                                            \
    if (_e != cudaSuccess) return host::record_cuda_error(_e, #expr);   \
  } while (0)

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <int OUTMODE, int BN, bool FP4, bool SPLIT = false>
int launch_mx(const CUtensorMap& tmA, const MxParams& p, cudaStream_t s) {
  static std::atomic<uint64_t> done{0};
  auto kernel = mx_gemm_kernel<OUTMODE, BN, FP4, SPLIT>;
  using Smem = MxSmem<BN, FP4>;
  int dev = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << dev;
  if (!(done.load(std::memory_order_acquire) & bit)) {
    CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem::TOTAL));
    done.fetch_or(bit, std::memory_order_release);
  }
  int sms = 0;
  int rc = host::sm_count(&sms);
  if (rc) return rc;
  const long long tiles = static_cast<long long>((p.M + BLOCK_ROWS - 1) / BLOCK_ROWS) * (p.N / BN);
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(static_cast<unsigned>(SPLIT ? tiles * p.split : tiles < sms ? tiles : sms), 1, 1);
  cfg.blockDim = dim3(MX_THREADS, 1, 1);
  cfg.dynamicSmemBytes = Smem::TOTAL;
  cfg.stream = s;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_dependent
  attrs[0].val.programmaticStreamSerializationAllowed = 1;
  int na = host::pdl_default() != 0 ? 1 : 0;
  if (SPLIT) {
    attrs[na].id = cudaLaunchAttributeClusterDimension;
    attrs[na].val.clusterDim.x = static_cast<unsigned>(p.split);
    attrs[na].val.clusterDim.y = 1;
    attrs[na].val.clusterDim.z = 1;
    ++na;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = na;
  CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, tmA, p));
  return FLYB200_OK;
}

}  // namespace

template <typename TIn>
cudaError_t launch_mx_quant(uint8_t* codes, uint8_t* scale, uint8_t* raw, const TIn* x, long long units, int fmt, cudaStream_t s) {
  const unsigned grid = static_cast<unsigned>((units + 255) / 256);
  auto kernel = fmt == MXQ_FP8 ? mx_quant_kernel<TIn, MXQ_FP8> : fmt == MXQ_FP4 ? mx_quant_kernel<TIn, MXQ_FP4> : mx_quant_kernel<TIn, MXQ_FP6>;
  return host::launch_dependent(kernel, dim3(grid), 256, 0, s, codes, scale, raw, x, units);
}

namespace {
// Up to 128 tokens are a weight stream for the small-M kernel in its block-scaled kind - as long as its
// CTAs (one per 128 channels) fit one round: on wider outputs its later rounds run part empty and the
// persistent large-M kernel is 20-45 % faster (MXFP8 128 x 28672 x 8192: 43 against 66 us; MXFP4 128 x
// 57344 x 8192: 51 against 90 us).  FLYB200_MX_SMALL=0 / 1 forces the choice.
// With more than half as many channel tiles as SMs the small-M kernel has no K split to balance its token
// tile with, and from 65 tokens up (MXFP4, half the weight bytes: 33) the large-M kernel is ahead: MXFP8 96 x
// 12288 x 4096 16.6 against 20.1 us, 128 x 16384 x 8192 29.0 / 34.7 (64: 16.2 / 16.4, 28 / 28); MXFP4 128 x 12288 x
// 4096 11.5 / 18.3, 64 x 10240 x 8192 16.8 / 18.1 (16: 11.4 / 9.7).
bool mx_small_m(int M, int N, bool fp4 = false) {
  if (M > 128) return false;
  if (const char* e = getenv("FLYB200_MX_SMALL")) {
    if (e[0] == '0') return false;
    if (e[0] == '1') return true;
  }
  int sms = 0;
  if (flyb200::host::sm_count(&sms) != FLYB200_OK) return true;
  const int tiles = (N + 127) / 128;
  return tiles <= sms && (2 * tiles <= sms || M <= (fp4 ? 32 : 64));
}
// The mixed kinds (byte containers; kb 128-byte k-blocks).  Small-M / large-M kernel, us, MXFP6 x MXFP4:
//  * below 12 k-blocks the small-M kernel does not split K and pays about 45 ns a token for its stores: 128 x 2048 x 1024
//    10.9 / 5.6, 16 x 4096 x 1024 6.4 / 4.9, 4 x 8192 x 512 4.3 / 3.7.  Only on outputs of more than half as many channel tiles as
//    SMs, where the large-M kernel cannot split K either, a few tokens are faster: 8 x 14336 x 1024 6.2 / 7.0, 16 x 14336 x 512
//    5.1 / 4.6;
//  * from 12 to 15 its split is small: 16 x 4096 x 1536 5.1 / 6.2, 33 x 4096 x 1536 7.2 / 6.4, 33 x 14336 x 1536 8.1 / 9.0;
//  * above, up to 64 tokens (64 x 4096 x 4096 8.0 / 10.0), on wide outputs 48 (48 x 14336 x 2048 9.2 / 11.0, 64 x 14336 x 2048 9.7 / 8.8),
//    and 128 where the large-M kernel can split K in four: 100 x 2048 x 4096 8.0 / 8.8.
bool mx_mixed_small_m(int M, int N, int kb) {
  if (!mx_small_m(M, N)) return false;
  int sms = 0;
  if (getenv("FLYB200_MX_SMALL") || flyb200::host::sm_count(&sms) != FLYB200_OK) return true;
  const int tiles = (N + 127) / 128;
  const bool wide = 2 * tiles > sms;
  if (kb < 12) return wide && M <= kb;
  if (kb < 16) return M <= (wide ? 48 : 16);
  if (wide) return M <= 48;
  return M <= 64 || 4 * tiles <= sms;
}
// Tile shape of the large-M kernel: 128 x 256 tiles (one accumulator, exposed epilogue) win once a
// tile's mainloop is a few times longer than its epilogue (2.44-2.47 against 1.82-1.88 PFLOP/s at
// K = 8192, M >= 4096) - unless the 128 x 128 tiles cover the output in one round of CTAs: then
// they put twice as many SMs to work (MXFP8 256 x 8192 x 8192: 27.9 against 31.4 us; MXFP4:
// 18.4 against 20.9 us).  `k_bytes`: bytes of codes per row.
bool mx_wide_tiles(int M, int N, int k_bytes) {
  if (N % 256 != 0 || k_bytes < 1024) return false;
  int sms = 0;
  if (flyb200::host::sm_count(&sms) != FLYB200_OK) return true;
  const long long tiles128 = static_cast<long long>((M + 127) / 128) * (N / 128);
  return tiles128 > sms;
}
// K parts of a tile (CTAs of a cluster), 1 = none: the largest of eight, four and two that fits one round of
// CTAs with at least eight k-blocks each.  Clusters of eight have to find eight free SMs inside one GPC
// and are placed without delay only while they cover at most half of the SMs.  Measured, split 1 / 2 / 4 /
// 8, us: MXFP6 x MXFP4 256 x 4096 x 14336 (64 tiles) 46.2 / 27.7 / 36.0 / 66, 128 x 4096 x 14336 (32) 46.2 /
// 27.0 / 19.9 / 41, 64 x 1024 x 8192 (8) 27.8 / 17.1 / 13.1 / 11.2; MXFP8 200 x 1024 x 14336 (16) 44.0 / 23.9 /
// 16.5 / 22.5, 600 x 1792 x 2048 (70, 16 k-blocks) 11.4 / 9.6 / 23 / 41, 256 x 4096 x 1024 (64, 8 k-blocks)
// 7.2 / 8.0 / 16 / 40; MXFP4 256 x 4096 x 14336 27.9 / 18.1 / 26.4 / 54.
// FLYB200_MX_SPLIT = 1, 2, 4 or 8 forces the factor (tuning and tests), halved until every part has a k-block:
// a CTA without one would add an accumulator that no MMA has written.
int mx_split(int M, int N, int k_bytes) {
  const int kb = k_bytes / KBLOCK_BYTES;
  if (const char* e = getenv("FLYB200_MX_SPLIT"))
    if (e[0] == '1' || e[0] == '2' || e[0] == '4' || e[0] == '8') {
      int split = e[0] - '0';
      while (split > kb) split /= 2;
      return split;
    }
  int sms = 0;
  if (flyb200::host::sm_count(&sms) != FLYB200_OK) return 1;
  const long long tiles = static_cast<long long>((M + 127) / 128) * (N / 128);
  if (16 * tiles <= sms && kb >= 64) return 8;
  if (4 * tiles <= sms && kb >= 32) return 4;
  if (2 * tiles <= sms && kb >= 16) return 2;
  return 1;
}

template <int OUTMODE, bool FP4>
int launch_mx_large(const void* a, MxParams& p, cudaStream_t s) {
  int rc = host::status_word(&p.status);
  if (rc) return rc;
  CUtensorMap tmA;
  rc = host::byte_matrix_map(&tmA, a, static_cast<uint64_t>(p.K_bytes), static_cast<uint64_t>(p.M), BLOCK_ROWS);
  if (rc) return rc;
  // FLYB200_MX_BN forces a tile shape without a K split (tuning and tests)
  bool wide = mx_wide_tiles(p.M, p.N, p.K_bytes);
  p.split = wide ? 1 : mx_split(p.M, p.N, p.K_bytes);
  if (const char* e = getenv("FLYB200_MX_BN")) {
    if (e[0] == '1') wide = false, p.split = 1;
    if (e[0] == '2' && p.N % 256 == 0) wide = true;
  }
  if (wide) return launch_mx<OUTMODE, 256, FP4>(tmA, p, s);
  if (p.split > 1) return launch_mx<OUTMODE, 128, FP4, true>(tmA, p, s);
  return launch_mx<OUTMODE, 128, FP4>(tmA, p, s);
}
template <bool FP4>
int launch_mx_large(const void* a, MxParams& p, int out_dtype, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return out_dtype == FLYB200_OUT_BF16 ? launch_mx_large<MOE_OUT_BF16, FP4>(a, p, s) : launch_mx_large<MOE_OUT_FP16, FP4>(a, p, s);
}
}  // namespace

extern "C" {

size_t flyb200_mx_scale_image_bytes(int rows, int K) {
  if (rows <= 0 || K <= 0 || K % KBLOCK_BYTES != 0) return 0;
  return static_cast<size_t>(K / KBLOCK_BYTES) * ((rows + 127) / 128) * MX_SF_ATOM;
}

int flyb200_mx_quant(void* codes, void* scale, void* raw, const void* x, long long elements, int x_dtype, int format,
                     void* stream) {
  if (!codes || !scale || !x || elements < 0) return FLYB200_E_BAD_ARG;
  if (format != FLYB200_MXFMT_E4M3 && format != FLYB200_MXFMT_E2M3 && format != FLYB200_MXFMT_E2M1) return FLYB200_E_UNSUPPORTED;
  if (format == FLYB200_MXFMT_E2M3 && !raw) return FLYB200_E_BAD_ARG;
  if (x_dtype < 0 || x_dtype > 2) return FLYB200_E_BAD_ARG;
  if (elements % 32 != 0 || elements / MXQ_UNIT > 0x7fffffffll * 256) return FLYB200_E_UNSUPPORTED;
  if (!aligned16(codes) || !aligned16(x) || (raw && !aligned16(raw))) return FLYB200_E_BAD_ALIGN;
  if (elements == 0) return FLYB200_OK;
  const long long units = elements / MXQ_UNIT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  uint8_t *c = static_cast<uint8_t*>(codes), *sc = static_cast<uint8_t*>(scale), *r = static_cast<uint8_t*>(raw);
  if (x_dtype == 0) CUDA_TRY(launch_mx_quant(c, sc, r, static_cast<const float*>(x), units, format, s));
  else if (x_dtype == 1) CUDA_TRY(launch_mx_quant(c, sc, r, static_cast<const __half*>(x), units, format, s));
  else CUDA_TRY(launch_mx_quant(c, sc, r, static_cast<const __nv_bfloat16*>(x), units, format, s));
  return FLYB200_OK;
}

int flyb200_mx_fp6_containers(void* dst, const void* src, long long bytes, void* stream) {
  if (!dst || !src || bytes < 0) return FLYB200_E_BAD_ARG;
  if (bytes % 32 != 0) return FLYB200_E_UNSUPPORTED;
  if (!aligned16(dst) || !aligned16(src)) return FLYB200_E_BAD_ALIGN;
  if (bytes == 0) return FLYB200_OK;
  const long long blocks32 = bytes / 32;
  long long grid = (blocks32 + 255) / 256;
  if (grid > 148 * 16) grid = 148 * 16;
  CUDA_TRY(host::launch_dependent(mx_fp6_containers_kernel, dim3(static_cast<unsigned>(grid)), 256, 0, static_cast<cudaStream_t>(stream),
                                  static_cast<uint4*>(dst), static_cast<const uint4*>(src), blocks32));
  return FLYB200_OK;
}

int flyb200_mx_scale_image(void* dst, const void* src, int rows, int K, void* stream) {
  if (!dst || !src || rows <= 0 || K <= 0) return FLYB200_E_BAD_ARG;
  if (K % KBLOCK_BYTES != 0) return FLYB200_E_UNSUPPORTED;
  const int row_tiles = (rows + 127) / 128;
  const long long total = static_cast<long long>(flyb200_mx_scale_image_bytes(rows, K)) / 4;
  long long blocks = (total + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  CUDA_TRY(host::launch_dependent(mx_scale_image_kernel, dim3(static_cast<unsigned>(blocks)), 256, 0, static_cast<cudaStream_t>(stream),
                                  static_cast<uint8_t*>(dst), static_cast<const uint8_t*>(src), rows, K / 32, row_tiles));
  return FLYB200_OK;
}

int flyb200_gemm_mxfp8(void* c, const void* a, const void* w_shuf, const void* scale_a_image, const void* scale_w_image,
                       int M, int N, int K, int out_dtype, void* stream) {
  if (!c || !a || !w_shuf || !scale_a_image || !scale_w_image || M < 0 || N <= 0 || K <= 0) return FLYB200_E_BAD_ARG;
  if (out_dtype != FLYB200_OUT_BF16 && out_dtype != FLYB200_OUT_FP16) return FLYB200_E_BAD_ARG;
  if (K % KBLOCK_BYTES != 0 || N % 128 != 0) return FLYB200_E_UNSUPPORTED;
  if (!aligned16(c) || !aligned16(a) || !aligned16(w_shuf) || !aligned16(scale_a_image) || !aligned16(scale_w_image))
    return FLYB200_E_BAD_ALIGN;
  if (M == 0) return FLYB200_OK;
  // up to 128 tokens: a weight stream, run by the small-M kernel in its block-scaled kind
  if (mx_small_m(M, N))
    return host::gemm_mx_small(c, a, w_shuf, scale_a_image, scale_w_image, M, N, K, out_dtype == FLYB200_OUT_FP16 ? 1 : 0,
                               false, stream);
  MxParams p;
  memset(&p, 0, sizeof(p));
  p.w = static_cast<const uint8_t*>(w_shuf);
  p.sfa = static_cast<const uint8_t*>(scale_a_image);
  p.sfw = static_cast<const uint8_t*>(scale_w_image);
  p.c = c;
  p.M = M;
  p.N = N;
  p.K_bytes = K;
  p.group_m = 16;
  return launch_mx_large<false>(a, p, out_dtype, stream);
}

int flyb200_gemm_mx_mixed(void* c, const void* a, const void* w_shuf, const void* scale_a_image, const void* scale_w_image,
                          int M, int N, int K, int a_format, int w_format, int out_dtype, void* stream) {
  if (!c || !a || !w_shuf || !scale_a_image || !scale_w_image || M < 0 || N <= 0 || K <= 0) return FLYB200_E_BAD_ARG;
  if (out_dtype != FLYB200_OUT_BF16 && out_dtype != FLYB200_OUT_FP16) return FLYB200_E_BAD_ARG;
  auto known = [](int f) { return f == FLYB200_MXFMT_E4M3 || f == FLYB200_MXFMT_E5M2 || f == FLYB200_MXFMT_E2M3 ||
                                  f == FLYB200_MXFMT_E3M2 || f == FLYB200_MXFMT_E2M1; };
  if (!known(a_format) || !known(w_format)) return FLYB200_E_BAD_ARG;
  if (K % KBLOCK_BYTES != 0 || N % 128 != 0) return FLYB200_E_UNSUPPORTED;
  if (!aligned16(c) || !aligned16(a) || !aligned16(w_shuf) || !aligned16(scale_a_image) || !aligned16(scale_w_image))
    return FLYB200_E_BAD_ALIGN;
  if (M == 0) return FLYB200_OK;
  if (mx_mixed_small_m(M, N, K / KBLOCK_BYTES))
    return host::gemm_mx_small(c, a, w_shuf, scale_a_image, scale_w_image, M, N, K, out_dtype == FLYB200_OUT_FP16 ? 1 : 0,
                               false, stream, a_format, w_format);
  MxParams p;
  memset(&p, 0, sizeof(p));
  p.w = static_cast<const uint8_t*>(w_shuf);
  p.sfa = static_cast<const uint8_t*>(scale_a_image);
  p.sfw = static_cast<const uint8_t*>(scale_w_image);
  p.c = c;
  p.M = M;
  p.N = N;
  p.K_bytes = K;  // one byte per code: sub-byte codes travel in byte containers
  p.group_m = 16;
  p.fmt_bits = (static_cast<uint32_t>(a_format) << 7) | (static_cast<uint32_t>(w_format) << 10);
  return launch_mx_large<false>(a, p, out_dtype, stream);
}

int flyb200_gemm_mxfp4(void* c, const void* a, const void* w_shuf, const void* scale_a_image, const void* scale_w_image,
                       int M, int N, int K, int out_dtype, void* stream) {
  if (!c || !a || !w_shuf || !scale_a_image || !scale_w_image || M < 0 || N <= 0 || K <= 0) return FLYB200_E_BAD_ARG;
  if (out_dtype != FLYB200_OUT_BF16 && out_dtype != FLYB200_OUT_FP16) return FLYB200_E_BAD_ARG;
  if (K % (2 * KBLOCK_BYTES) != 0 || N % 128 != 0) return FLYB200_E_UNSUPPORTED;  // whole 128-byte k-blocks of packed codes
  if (!aligned16(c) || !aligned16(a) || !aligned16(w_shuf) || !aligned16(scale_a_image) || !aligned16(scale_w_image))
    return FLYB200_E_BAD_ALIGN;
  if (M == 0) return FLYB200_OK;
  // up to 128 tokens: a weight stream (half the bytes of 8-bit codes), run by the small-M kernel
  if (mx_small_m(M, N, true))
    return host::gemm_mx_small(c, a, w_shuf, scale_a_image, scale_w_image, M, N, K / 2,
                               out_dtype == FLYB200_OUT_FP16 ? 1 : 0, true, stream);
  MxParams p;
  memset(&p, 0, sizeof(p));
  p.w = static_cast<const uint8_t*>(w_shuf);
  p.sfa = static_cast<const uint8_t*>(scale_a_image);
  p.sfw = static_cast<const uint8_t*>(scale_w_image);
  p.c = c;
  p.M = M;
  p.N = N;
  p.K_bytes = K / 2;
  p.group_m = 16;
  return launch_mx_large<true>(a, p, out_dtype, stream);
}

}  // extern "C"
