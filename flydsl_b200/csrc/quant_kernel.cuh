// Per-token (per-row) symmetric quantisation fp32/fp16/bf16 -> fp8 e4m3 / int8
// with one fp32 scale per row: the step that feeds the GEMM's A operand.
//
//   h     = x with NaN -> 0, +Inf -> qmax, -Inf -> -qmax
//   scale = max_k |h[k]| * (1 / qmax), 0 -> 1      (qmax = 448 or 127)
//   y[k]  = convert(h[k] / scale)                  fp8: round to nearest even,
//                                                  int8: truncate toward zero
//
// The arithmetic follows what the torch statement of the reference helper
// computes on a GPU, operation by operation, so results are bit-identical to
// it: the division of the row maximum by the Python scalar qmax is executed by
// torch's CUDA backend as a multiplication by the fp32 reciprocal, the
// element-wise division is a true IEEE division.
//
// Rows of up to 8192 (fp32) / 16384 (16-bit) elements stay in registers between the
// maximum and the conversion and are read from memory once; longer rows are read
// twice (the second time from L1/L2).
#pragma once
#include <cstdint>
#include <type_traits>
#include "ptx.cuh"
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

namespace flyb200 {

enum : int { QX_F32 = 0, QX_F16 = 1, QX_BF16 = 2 };

template <typename T>
struct QuantIn;
template <>
struct QuantIn<float> {
  static constexpr int VEC = 4;  // elements per 16-byte load
  __device__ static void load(const float* p, float (&v)[4]) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
  }
};
template <>
struct QuantIn<__half> {
  static constexpr int VEC = 8;
  __device__ static void load(const __half* p, float (&v)[8]) {
    const uint4 t = *reinterpret_cast<const uint4*>(p);
    const __half2* h = reinterpret_cast<const __half2*>(&t);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __half22float2(h[i]);
      v[2 * i] = f.x, v[2 * i + 1] = f.y;
    }
  }
};
template <>
struct QuantIn<__nv_bfloat16> {
  static constexpr int VEC = 8;
  __device__ static void load(const __nv_bfloat16* p, float (&v)[8]) {
    const uint4 t = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&t);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      v[2 * i] = f.x, v[2 * i + 1] = f.y;
    }
  }
};

__device__ __forceinline__ float scrub(float v, float qmax) {
  if (v != v) return 0.0f;
  if (v == INFINITY) return qmax;
  if (v == -INFINITY) return -qmax;
  return v;
}

template <bool FP8>
__device__ __forceinline__ uint8_t quant_one(float v, float s) {
  const float q = __fdiv_rn(v, s);
  if constexpr (FP8) {
    return static_cast<uint8_t>(__nv_cvt_float_to_fp8(q, __NV_SATFINITE, __NV_E4M3));
  } else {
    return static_cast<uint8_t>(static_cast<int8_t>(__float2int_rz(q)));
  }
}

// Four finite values -> four packed bytes, bit-identical to four quant_one calls without the IEEE
// divisions: q0 = v * y with y = RN(1 / s), then one correction with the exact residual,
// q = q0 + (v - q0 s) y, which rounds to the IEEE quotient (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000", 1990).  Two values per instruction.  The residual is exact
// where q matters (from half the smallest e4m3 subnormal, 2^-10, or 1 for int8, up) as long as s is not
// below 2^-90; the caller divides there.  fp8: the quotient is carried negated, which keeps the sign of a
// zero (-0 / s = -0) through the correction; the sign bits are flipped back at the end.
__device__ __forceinline__ unsigned long long f32x2(float lo, float hi) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float2 f32x2_parts(unsigned long long d) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(d));
  return f;
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long mul_f32x2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// What the conversion of a row needs of its scale, each twice: fp8 (s, -1 / s), int8 (-s, 1 / s).
struct RowDivisor {
  unsigned long long s, inv;
};
template <bool FP8>
__device__ __forceinline__ RowDivisor row_divisor(float s) {
  const float inv = __frcp_rn(s);
  return FP8 ? RowDivisor{f32x2(s, s), f32x2(-inv, -inv)} : RowDivisor{f32x2(-s, -s), f32x2(inv, inv)};
}
constexpr float QUANT_TINY_SCALE = 1e-27f;  // above 2^-90

template <bool FP8>
__device__ __forceinline__ uint32_t quant_four(unsigned long long v01, unsigned long long v23, const RowDivisor& d) {
  unsigned long long q01 = mul_f32x2(v01, d.inv), q23 = mul_f32x2(v23, d.inv);
  q01 = fma_f32x2(fma_f32x2(q01, d.s, v01), d.inv, q01);
  q23 = fma_f32x2(fma_f32x2(q23, d.s, v23), d.inv, q23);
  const float2 a = f32x2_parts(q01), b = f32x2_parts(q23);
  if constexpr (FP8) {
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(a, __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(b, __NV_SATFINITE, __NV_E4M3);
    return (lo | (hi << 16)) ^ 0x80808080u;
  } else {
    const uint32_t lo = __byte_perm(__float2int_rz(a.x), __float2int_rz(a.y), 0x0040);
    const uint32_t hi = __byte_perm(__float2int_rz(b.x), __float2int_rz(b.y), 0x0040);
    return __byte_perm(lo, hi, 0x5410);
  }
}

// Largest magnitude of a 16-byte vector and what the raw words stand for.  For finite values the order
// of |x| is the order of the bit patterns without their sign, and any Inf / NaN shows up as a maximum of at
// least INF_BITS, so the maximum needs no conversion: two 16-bit values per instruction.
template <typename T>
struct QuantRaw;
template <>
struct QuantRaw<float> {
  static constexpr uint32_t INF_BITS = 0x7F800000u;
  __device__ static uint32_t max_abs(uint32_t m, uint32_t w) { return max(m, w & 0x7FFFFFFFu); }
  __device__ static uint32_t fold(uint32_t m) { return m; }
  __device__ static float value(uint32_t bits) { return __uint_as_float(bits); }
  __device__ static void unpack(const uint4& t, float (&v)[4]) {
    v[0] = __uint_as_float(t.x), v[1] = __uint_as_float(t.y), v[2] = __uint_as_float(t.z), v[3] = __uint_as_float(t.w);
  }
};
template <typename T>
struct QuantRaw16 {
  __device__ static uint32_t max_abs(uint32_t m, uint32_t w) { return __vmaxu2(m, w & 0x7FFF7FFFu); }
  __device__ static uint32_t fold(uint32_t m) { return max(m & 0xFFFFu, m >> 16); }
};
template <>
struct QuantRaw<__half> : QuantRaw16<__half> {
  static constexpr uint32_t INF_BITS = 0x7C00u;
  __device__ static float value(uint32_t bits) { return __half2float(__ushort_as_half(static_cast<unsigned short>(bits))); }
  __device__ static void unpack(const uint4& t, float (&v)[8]) { QuantIn<__half>::load(reinterpret_cast<const __half*>(&t), v); }
};
template <>
struct QuantRaw<__nv_bfloat16> : QuantRaw16<__nv_bfloat16> {
  static constexpr uint32_t INF_BITS = 0x7F80u;
  __device__ static float value(uint32_t bits) { return __uint_as_float(bits << 16); }
  __device__ static void unpack(const uint4& t, float (&v)[8]) {
    const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) v[2 * i] = __uint_as_float(w[i] << 16), v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
};

// Quantises one row held as NV raw vectors per thread by the WPR warps that share it (`tid` inside
// them): vector i covers elements (i * 32 WPR + tid) * VEC.  `red`: 8 words of shared memory of the block,
// `first_warp`: the row's first warp; barriers are per row (`bar_id`), so rows may take different branches.
template <typename TIn, bool FP8, int NV, int WPR>
__device__ __forceinline__ void quant_row_from_registers(const uint4 (&raw)[NV], uint8_t* __restrict__ yr, float* scale_out,
                                                         int K, int tid, uint32_t* red, int first_warp, int bar_id) {
  using R = QuantRaw<TIn>;
  constexpr int VEC = QuantIn<TIn>::VEC;
  constexpr int TPR = 32 * WPR;
  constexpr float QMAX = FP8 ? 448.0f : 127.0f;
  const int lane = tid & 31, warp = tid >> 5;
  auto row_max = [&](uint32_t m) {
    m = __reduce_max_sync(0xffffffffu, m);
    if constexpr (WPR > 1) {
      if (lane == 0) red[first_warp + warp] = m;
      asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "n"(TPR) : "memory");
#pragma unroll
      for (int w = 0; w < WPR; ++w) m = max(m, red[first_warp + w]);
    }
    return m;
  };
  uint32_t m = 0u;
#pragma unroll
  for (int i = 0; i < NV; ++i) m = R::max_abs(R::max_abs(R::max_abs(R::max_abs(m, raw[i].x), raw[i].y), raw[i].z), raw[i].w);
  m = row_max(R::fold(m));

  if (m >= R::INF_BITS) {
    // ---- careful path: the row holds Inf or NaN (the same branch in all of the row's threads) ----
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float v[VEC];
      R::unpack(raw[i], v);
#pragma unroll
      for (int e = 0; e < VEC; ++e) amax = fmaxf(amax, fabsf(scrub(v[e], QMAX)));
    }
    if constexpr (WPR > 1) asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "n"(TPR) : "memory");  // red is reused
    float s = __fmul_rn(__uint_as_float(row_max(__float_as_uint(amax))), __fdiv_rn(1.0f, QMAX));
    if (s == 0.0f) s = 1.0f;
    if (tid == 0) *scale_out = s;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int k = (i * TPR + tid) * VEC;
      if (k >= K) break;
      float v[VEC];
      R::unpack(raw[i], v);
#pragma unroll
      for (int e = 0; e < VEC; ++e) yr[k + e] = quant_one<FP8>(scrub(v[e], QMAX), s);
    }
    return;
  }

  float s = __fmul_rn(R::value(m), __fdiv_rn(1.0f, QMAX));
  if (s == 0.0f) s = 1.0f;
  if (tid == 0) *scale_out = s;
  const bool tiny = s < QUANT_TINY_SCALE;
  const RowDivisor d = row_divisor<FP8>(s);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int k = (i * TPR + tid) * VEC;
    if (k >= K) break;
    float v[VEC];
    R::unpack(raw[i], v);
    uint32_t packed[VEC / 4];
#pragma unroll
    for (int w = 0; w < VEC / 4; ++w) {
      if (!tiny) {
        packed[w] = quant_four<FP8>(f32x2(v[4 * w], v[4 * w + 1]), f32x2(v[4 * w + 2], v[4 * w + 3]), d);
      } else {
        packed[w] = 0u;
#pragma unroll
        for (int e = 0; e < 4; ++e) packed[w] |= static_cast<uint32_t>(quant_one<FP8>(v[4 * w + e], s)) << (8 * e);
      }
    }
    if constexpr (VEC == 4) {
      *reinterpret_cast<uint32_t*>(yr + k) = packed[0];
    } else {
      *reinterpret_cast<uint2*>(yr + k) = make_uint2(packed[0], packed[1]);
    }
  }
}

// Single-pass form for rows of at most 32 * WPR * VEC * NV elements.  WPR warps of a 256-thread block
// share a row; every thread has its NV loads in flight together and keeps the raw vectors in registers
// (half the registers of the converted values, so more rows in flight).  Memory-bound where there are
// rows enough; few rows are spread over more warps (quant_warps_per_row).  One 256-thread block per row, with
// a conversion of every value before the maximum and a test next to every product for a rounding boundary,
// was bound by instruction issue and, on short rows, by blocks of a few loads each.  bf16 -> fp8 / int8, us,
// before and now: 8192 x 8192 51.7 / 49.0 and 39.1 / 44.3 (5.2 / 4.6 TB/s), 8192 x 2048 17.5 / 16.3 and
// 11.4 / 12.9, 4096 x 14336 61.4 / 58.7 and 37.6 / 42.8, 997 x 5120 6.9 / 7.0 and 4.3 / 5.1, 1 x 8192 2.7 and 1.9.
// (int8 trails by its float-to-integer conversions, four to a byte quad.)
template <typename TIn, bool FP8, int NV, int WPR>
__global__ void __launch_bounds__(256) pertoken_quant_row_kernel(uint8_t* __restrict__ y, float* __restrict__ scale,
                                                                 const TIn* __restrict__ x, int rows, int K) {
  constexpr int VEC = QuantIn<TIn>::VEC;
  __shared__ uint32_t red[8];
  pdl_wait(x, y, scale);
  pdl_trigger();
  const int group = threadIdx.x / (32 * WPR), tid = threadIdx.x % (32 * WPR);
  const int r = blockIdx.x * (8 / WPR) + group;
  if (r >= rows) return;
  const TIn* xr = x + static_cast<size_t>(r) * K;
  uint4 raw[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int k = (i * 32 * WPR + tid) * VEC;
    raw[i] = k < K ? __ldg(reinterpret_cast<const uint4*>(xr + k)) : make_uint4(0u, 0u, 0u, 0u);
  }
  quant_row_from_registers<TIn, FP8, NV, WPR>(raw, y + static_cast<size_t>(r) * K, scale + r, K, tid, red, group * WPR, 1 + group);
}

// Warps per row: as few as keep a row in eight vectors per thread (a warp that owns its row needs no
// barrier, and eight loads per thread cover the latency), but at least two blocks per SM: few rows
// take more warps each.  `vecs`: 16-byte vectors of a row.
inline int quant_warps_per_row(int rows, int vecs) {
  int wpr = 1;
  while (wpr < 8 && (vecs > 256 * wpr || static_cast<long long>(rows) * wpr < 2LL * 148 * 8)) wpr *= 2;
  return wpr;
}
// Calls launch(NV, WPR) with integral constants for a row of `vecs` vectors; false where it does not fit registers.
template <typename LaunchFn>
bool quant_row_dispatch(int rows, int vecs, LaunchFn launch) {
  using std::integral_constant;
  const int wpr = quant_warps_per_row(rows, vecs);
  const int nv = (vecs + 32 * wpr - 1) / (32 * wpr);  // vectors per thread
  if (nv > 8) return false;
  const bool four = nv <= 4;
  if (wpr == 1) {
    four ? launch(integral_constant<int, 4>(), integral_constant<int, 1>()) : launch(integral_constant<int, 8>(), integral_constant<int, 1>());
  } else if (wpr == 2) {
    four ? launch(integral_constant<int, 4>(), integral_constant<int, 2>()) : launch(integral_constant<int, 8>(), integral_constant<int, 2>());
  } else if (wpr == 4) {
    four ? launch(integral_constant<int, 4>(), integral_constant<int, 4>()) : launch(integral_constant<int, 8>(), integral_constant<int, 4>());
  } else if (nv <= 1) {
    launch(integral_constant<int, 1>(), integral_constant<int, 8>());
  } else if (nv <= 2) {
    launch(integral_constant<int, 2>(), integral_constant<int, 8>());
  } else {
    four ? launch(integral_constant<int, 4>(), integral_constant<int, 8>()) : launch(integral_constant<int, 8>(), integral_constant<int, 8>());
  }
  return true;
}

// General form (any row length): two passes over the row, the second one from L1/L2.
template <typename TIn, bool FP8>
__global__ void __launch_bounds__(256) pertoken_quant_kernel(uint8_t* __restrict__ y, float* __restrict__ scale,
                                                             const TIn* __restrict__ x, int rows, int K) {
  constexpr int VEC = QuantIn<TIn>::VEC;
  constexpr float QMAX = FP8 ? 448.0f : 127.0f;
  __shared__ float warp_max[8];
  __shared__ float row_scale;
  pdl_wait(x, y, scale);
  pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const TIn* xr = x + static_cast<size_t>(r) * K;
    float amax = 0.0f;
    for (int k = threadIdx.x * VEC; k < K; k += 256 * VEC) {
      float v[VEC];
      QuantIn<TIn>::load(xr + k, v);
#pragma unroll
      for (int i = 0; i < VEC; ++i) amax = fmaxf(amax, fabsf(scrub(v[i], QMAX)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) warp_max[warp] = amax;
    __syncthreads();
    if (warp == 0) {
      float m = lane < 8 ? warp_max[lane] : 0.0f;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (lane == 0) {
        float s = __fmul_rn(m, __fdiv_rn(1.0f, QMAX));
        if (s == 0.0f) s = 1.0f;
        row_scale = s;
        scale[r] = s;
      }
    }
    __syncthreads();
    const float s = row_scale;
    uint8_t* yr = y + static_cast<size_t>(r) * K;
    for (int k = threadIdx.x * VEC; k < K; k += 256 * VEC) {
      float v[VEC];
      QuantIn<TIn>::load(xr + k, v);
      uint32_t packed[VEC / 4];
#pragma unroll
      for (int w = 0; w < VEC / 4; ++w) {
        uint32_t b = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) b |= static_cast<uint32_t>(quant_one<FP8>(scrub(v[4 * w + i], QMAX), s)) << (8 * i);
        packed[w] = b;
      }
      if constexpr (VEC == 4) {
        *reinterpret_cast<uint32_t*>(yr + k) = packed[0];
      } else {
        *reinterpret_cast<uint2*>(yr + k) = make_uint2(packed[0], packed[1]);
      }
    }
    __syncthreads();  // row_scale / warp_max are reused by the next row
  }
}

}  // namespace flyb200
