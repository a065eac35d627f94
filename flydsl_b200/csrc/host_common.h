// Host helpers shared by the translation units of libflyb200 (not part of the C ABI).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace flyb200 {
namespace host {

// FLYB200_PDL, read once per process: 0 = no programmatic dependent launch, 1 = on, 2 = on and the weights are known to be static.
int pdl_default();

// Launches a kernel whose first statement is pdl_wait (ptx.cuh) as a programmatic dependent: its launch and
// set-up overlap the end of the kernel before it on the stream, one to two us each in a chain of small
// kernels.  Plain stream order / this, us a pass: MoE layer of 32 tokens 57.3 / 49.1, of 4096 282 / 277, its
// stages one by one (515 tokens) 82.0 / 70.2, MXFP6 layer of 256 tokens 41.4 / 33.9, MXFP8 of 1024 83.5 / 80.3.
template <typename... KArgs, typename... Args>
cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, int threads, int smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = pdl_default() != 0 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Tensor map over a row-major byte matrix [rows, row_bytes]: boxes of
// 128 bytes x box_rows rows, 128-byte swizzle, out-of-bounds rows read as zero.
int byte_matrix_map(CUtensorMap* m, const void* base, uint64_t row_bytes, uint64_t rows, uint32_t box_rows);
// Tensor map over preshuffled weights: `k_blocks` images of n_rows x 128 bytes, boxes of box_rows rows of one of them,
// copied as they are (the image is already swizzled); rows past n_rows read as zero.
int weight_image_map(CUtensorMap* m, const void* base, uint64_t n_rows, uint64_t k_blocks, uint32_t box_rows);
// Block-scaled GEMM (MXFP8, or MXFP4 with `fp4`) of up to 128 tokens on the small-M (weight-streaming)
// kernel; K = bytes of codes per row; outmode 0 bf16, 1 fp16.  a_format, w_format: codes in byte containers
// (FLYB200_MXFMT_*; 0 = E4M3, and for `fp4`).
int gemm_mx_small(void* c, const void* a, const void* w, const void* sf_a, const void* sf_w, int M, int N, int K,
                  int outmode, bool fp4, void* stream, int a_format = 0, int w_format = 0);
// Pointer to the current device's status word (first failed bounded wait wins).
int status_word(int** out);
// SM count of the current device.
int sm_count(int* out);
// Remember a CUDA error for flyb200_last_cuda_error(); returns FLYB200_E_CUDA.
int record_cuda_error(cudaError_t e, const char* what);

}  // namespace host
}  // namespace flyb200
