// Per-1x32 quantisers of the block-scaled formats, fp32 / fp16 / bf16 -> codes and
// one E8M0 scale per 32 elements: the step that feeds the activations of the MX
// GEMMs.  One kernel per call; results are bit-identical to the torch statements
// in kernels/gemm/mxfp8_preshuffle.py and mxfp4_preshuffle.py on the same GPU
// tensor.
//
//   m     = max |x| of the block            (MXFP8: at least 1e-30)
//   e     = exponent byte of m / 448 (MXFP8; torch divides a CUDA tensor by a
//           Python scalar by multiplying with its fp32 reciprocal) or of m / 4
//           (MXFP4, MXFP6), one higher when the mantissa is 1.5 or more
//   code  = x / 2^(e - 127) rounded to nearest even, saturating
//
// Dividing by a power of two and multiplying by its inverse round the same real
// number once, so the codes need no division, except for MXFP8 blocks so small
// that the scale is clamped to 1e-30.
//
// Bound: memory (bf16 -> MXFP8 moves 2 B in and 1.03 B out per element).  A thread
// takes 16 elements, i.e. half a block: two or four 16-byte loads in flight, one
// shuffle for the maximum, one 16-byte (MXFP4: 8-byte, MXFP6: 12-byte) store.
// Measured (bf16 in, kernel / the torch statement's kernels): MXFP8 1024 x 8192 6.7 / 187 us
// (3.8 TB/s), MXFP4 64 x 8192 1.9 / 165 us, MXFP6 256 x 14336 4.1 / 1070 us; as calls, with the
// statement's 30 to 250 launches: 1024 x 8192 x 8192 MXFP8 layer 320 -> 82 us, 64 x 8192 x 8192
// MXFP4 561 -> 44 us, 256 x 4096 x 14336 MXFP6 1615 -> 68 us.
#pragma once
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp4.h>
#include <cuda_fp6.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <type_traits>

namespace flyb200 {

enum : int { MXQ_FP8 = 0, MXQ_FP6 = 3, MXQ_FP4 = 5 };  // FLYB200_MXFMT_* of the formats that can be written

constexpr int MXQ_UNIT = 16;  // elements per thread

template <typename TIn>
__device__ __forceinline__ void mxq_load(const TIn* p, float (&v)[MXQ_UNIT]) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
  if constexpr (sizeof(TIn) == 4) {
    uint4 t[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = __ldg(q + i);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[4 * i] = __uint_as_float(t[i].x), v[4 * i + 1] = __uint_as_float(t[i].y);
      v[4 * i + 2] = __uint_as_float(t[i].z), v[4 * i + 3] = __uint_as_float(t[i].w);
    }
  } else {
    uint4 t[2];
    t[0] = __ldg(q), t[1] = __ldg(q + 1);
    const uint32_t w[8] = {t[0].x, t[0].y, t[0].z, t[0].w, t[1].x, t[1].y, t[1].z, t[1].w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if constexpr (std::is_same<TIn, __nv_bfloat16>::value) {
        v[2 * i] = __uint_as_float(w[i] << 16), v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
      } else {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        v[2 * i] = f.x, v[2 * i + 1] = f.y;
      }
    }
  }
}

// Exponent byte of a non-negative fp32 value, one higher when the mantissa is 1.5 or more (of a
// subnormal: when it is above one half).
__device__ __forceinline__ uint32_t e8m0_of(float v) {
  const uint32_t u = __float_as_uint(v);
  const uint32_t e = (u >> 23) & 0xFFu;
  if (e == 0xFFu) return e;
  const bool up = (u & 0x400000u) != 0u && ((u & 0x3FFFFFu) != 0u || e > 0u);
  return up ? e + 1u : e;
}

// codes: MXFP8 [rows, K], MXFP4 [rows, K/2] (even element in the low nibble), MXFP6
// [rows, K] in units of 32 bytes per block: 24 bytes of 6-bit codes (little-endian bit
// stream) and 8 zero bytes.  `raw` (MXFP6 only): the codes one per byte.
template <typename TIn, int FMT>
__global__ void __launch_bounds__(256) mx_quant_kernel(uint8_t* __restrict__ codes, uint8_t* __restrict__ scale,
                                                       uint8_t* __restrict__ raw, const TIn* __restrict__ x,
                                                       long long units) {
  pdl_wait(codes, scale, raw, x);
  pdl_trigger();
  const long long u = blockIdx.x * 256ll + threadIdx.x;
  // units is even (whole blocks of 32), so both lanes of a pair are in or out together; the others of the
  // warp stay for the shuffle
  const bool in = u < units;
  float v[MXQ_UNIT];
  if (in) {
    mxq_load(x + u * MXQ_UNIT, v);
  } else {
#pragma unroll
    for (int i = 0; i < MXQ_UNIT; ++i) v[i] = 0.0f;
  }
  // maximum on the bit patterns: the order of |x| for finite values, Inf and NaN above all of them
  uint32_t mb = 0u;
#pragma unroll
  for (int i = 0; i < MXQ_UNIT; ++i) mb = max(mb, __float_as_uint(v[i]) & 0x7FFFFFFFu);
  mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, 1));
  uint32_t e;
  if constexpr (FMT == MXQ_FP8) {
    const float m = mb > 0x7F800000u ? __uint_as_float(mb) : fmaxf(__uint_as_float(mb), 1e-30f);
    e = e8m0_of(__fmul_rn(m, 1.0f / 448.0f));
  } else {
    e = e8m0_of(__fmul_rn(__uint_as_float(mb), 0.25f));
  }
  if (!in) return;
  if ((u & 1) == 0) scale[u >> 1] = static_cast<uint8_t>(e);
  const bool nan_block = e == 0xFFu;  // the scale is NaN: so is every quotient
  // 1 / 2^(e - 127) for e = 0 .. 254
  const float inv = __uint_as_float(e == 254u ? 0x00400000u : (254u - e) << 23);
  if constexpr (FMT == MXQ_FP8) {
    uint32_t w[4];
    if (nan_block) {
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = 0x7F7F7F7Fu;
    } else {
      const float s = e == 0u ? __uint_as_float(0x00400000u) : __uint_as_float(e << 23);
      const bool tiny = s < 1e-30f;  // the statement divides by at least 1e-30
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float q[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) q[j] = tiny ? __fdiv_rn(v[4 * i + j], 1e-30f) : __fmul_rn(v[4 * i + j], inv);
        const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(q[0], q[1]), __NV_SATFINITE, __NV_E4M3);
        const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(q[2], q[3]), __NV_SATFINITE, __NV_E4M3);
        w[i] = lo | (hi << 16);
      }
    }
    *reinterpret_cast<uint4*>(codes + u * MXQ_UNIT) = make_uint4(w[0], w[1], w[2], w[3]);
  } else if constexpr (FMT == MXQ_FP4) {
    uint32_t w[2] = {0u, 0u};
    if (!nan_block) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 q = make_float2(__fmul_rn(v[2 * i], inv), __fmul_rn(v[2 * i + 1], inv));
        const uint32_t b = __nv_cvt_float2_to_fp4x2(q, __NV_E2M1, cudaRoundNearest);
        w[i >> 2] |= b << (8 * (i & 3));
      }
    }
    *reinterpret_cast<uint2*>(codes + u * (MXQ_UNIT / 2)) = make_uint2(w[0], w[1]);
  } else {
    uint32_t r[4] = {0u, 0u, 0u, 0u};
    if (!nan_block) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 q = make_float2(__fmul_rn(v[2 * i], inv), __fmul_rn(v[2 * i + 1], inv));
        const uint32_t b = __nv_cvt_float2_to_fp6x2(q, __NV_E2M3, cudaRoundNearest);
        r[i >> 1] |= (b & 0xFFFFu) << (16 * (i & 1));
      }
    }
    *reinterpret_cast<uint4*>(raw + u * MXQ_UNIT) = make_uint4(r[0], r[1], r[2], r[3]);
    // four 6-bit codes per byte-packed word -> 24 bits, four of those -> three words
    uint32_t t[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      t[i] = (r[i] & 0x3Fu) | ((r[i] >> 2) & 0xFC0u) | ((r[i] >> 4) & 0x3F000u) | ((r[i] >> 6) & 0xFC0000u);
    uint32_t* dst = reinterpret_cast<uint32_t*>(codes + (u >> 1) * 32);
    const int h = static_cast<int>(u & 1);
    dst[3 * h] = t[0] | (t[1] << 24);
    dst[3 * h + 1] = (t[1] >> 8) | (t[2] << 16);
    dst[3 * h + 2] = (t[2] >> 16) | (t[3] << 8);
    dst[6 + h] = 0u;
  }
}

// The MXFP6 activation layout above -> byte containers for kind::mxf8f6f4: every 16 codes (12 bytes)
// followed by 4 bytes of padding.  One thread per block of 32 codes.
static __global__ void __launch_bounds__(256) mx_fp6_containers_kernel(uint4* __restrict__ dst, const uint4* __restrict__ src,
                                                                       long long blocks) {
  pdl_wait(dst, src);
  pdl_trigger();
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < blocks; i += gridDim.x * 256ll) {
    const uint4 a = __ldg(src + 2 * i);
    const uint2 b = __ldg(reinterpret_cast<const uint2*>(src + 2 * i + 1));
    dst[2 * i] = make_uint4(a.x, a.y, a.z, 0u);
    dst[2 * i + 1] = make_uint4(a.w, b.x, b.y, 0u);
  }
}

}  // namespace flyb200
