// A8W8 preshuffle GEMM kernels for sm_100a.
//
//   C[M,N] = epilogue( (A[M,K] . W[N,K]^T) * sa[m] * sb[n] )
//
// A (activations) is row-major 8-bit; W (weights) is in the preshuffled image
// [K/128][N][128 B, 128-byte swizzled]: one k-block of any run of rows is a
// contiguous burst that is already the shared-memory image the tensor core
// wants.  Two kernels share one pipeline skeleton (TMA producer warp -> mbarrier
// ring -> single-thread tcgen05.mma issue -> accumulators in TMEM -> epilogue
// warps):
//
//   gemm_rows_kernel   tokens on the UMMA M side (128 per tile), weights on the
//                      N side (BN per tile).  Persistent, grouped rasterisation,
//                      two TMEM accumulator buffers so the epilogue of tile i
//                      overlaps the mainloop of tile i+1, bf16 tiles leave
//                      through swizzled shared memory and TMA stores.
//   gemm_decode_kernel weights on the UMMA M side (128 channels per CTA), the
//                      few tokens on the N side (BN = 16..256), optional split-K
//                      with a ticket so the last CTA of a channel tile reduces
//                      the partials in a fixed order.  HBM-bound weight stream.
#pragma once
#include "ptx.cuh"
#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace flyb200 {

enum : int { OUT_BF16 = 0, OUT_FP16 = 1, OUT_RAW32 = 2 };
enum : int { EPI_NONE = 0, EPI_BIAS = 1, EPI_BIAS_RELU = 2, EPI_BIAS_SILU = 3, EPI_BIAS_GELU = 4 };

constexpr int BLOCK_ROWS = 128;   // UMMA M
constexpr int KBLOCK_BYTES = 128; // one swizzle row: 128 fp8/int8 or 64 half elements
constexpr int UMMA_K_BYTES = 32;  // bytes of K consumed by one tcgen05.mma

struct GemmParams {
  const uint8_t* w;      // preshuffled weights
  const float* sa;       // [M] per-token scale or nullptr
  const float* sb;       // [N] per-channel scale or nullptr
  const void* bias;      // [N] in the output type or nullptr
  void* c;               // output (bf16/fp16 [M,N], or 32-bit raw accumulators)
  int M, N, K_bytes;     // K in bytes (= elements for 8-bit inputs)
  int epilogue;
  int group_m;           // rasterisation group (row tiles per group)
  int split_k;           // decode kernel: number of K splits
  int kb_per_split;      // decode kernel: k-blocks per split
  int reduce_mode;       // decode kernel: how the K splits are combined (REDUCE_*)
  int stages;            // decode kernel: depth of the shared-memory ring
  int pdl;               // decode kernel: launched with programmatic stream serialisation
  int prefetch;          // k-blocks of weights requested into L2 ahead of the shared-memory ring (0 = none)
  float* ws_partials;    // decode kernel, REDUCE_WORKSPACE
  int* ws_tickets;       // decode kernel, REDUCE_WORKSPACE (zero before first use; self-resetting)
  int token_blocks;      // decode kernel: grid.z, blocks of BN tokens
  const uint8_t* sf_w;   // decode kernel, MX kind: scale image of the weights [K/128][N/128][512]
  const uint8_t* sf_a;   // decode kernel, MX kind: scale image of the activations [K/128][sf_a_tiles][512]
  int sf_a_tiles;        // ceil(M / 128)
  uint32_t fmt_bits;     // decode kernel, MX kind on bytes: operand formats as instruction-descriptor bits (weights << 7 | tokens << 10)
  int bn;                // large-M kernel: output channels per tile (multiple of 32, 32..256)
  int rows_stages;       // large-M kernel: depth of the shared-memory ring
  int tail_parts;        // large-M kernels: column parts of the tiles of the last, partial round (1, 2 or 4; bn / parts a multiple of 64)
  int n_dst;             // scatter kernel: number of output buffers
  int dst_first;         // scatter kernel: buffer stored to first
  int* status;           // device status word (first failure wins)
#ifdef FLYB200_PROFILE
  unsigned long long* prof;  // [16] time stamps (profiling builds only)
#endif
};

template <int KIND>
struct KindTraits;
template <>
struct KindTraits<KIND_F8> {
  static constexpr uint32_t dfmt = 1, abfmt = 0;
  static constexpr bool is_int = false;
};
template <>
struct KindTraits<KIND_I8> {
  static constexpr uint32_t dfmt = 2, abfmt = 1;
  static constexpr bool is_int = true;
};
template <>
struct KindTraits<KIND_MXF8> {  // E4M3 codes with E8M0 block scales: fp32 accumulators, scaled inside the MMA
  static constexpr uint32_t dfmt = 1, abfmt = 0;
  static constexpr bool is_int = false;
};
template <>
struct KindTraits<KIND_MXF4> {  // packed E2M1 codes with E8M0 block scales
  static constexpr uint32_t dfmt = 1, abfmt = 1;
  static constexpr bool is_int = false;
};
template <>
struct KindTraits<KIND_F16> {
  static constexpr uint32_t dfmt = 1, abfmt = 0;
  static constexpr bool is_int = false;
};
template <>
struct KindTraits<KIND_BF16> {
  static constexpr uint32_t dfmt = 1, abfmt = 1;
  static constexpr bool is_int = false;
};

__device__ __forceinline__ void report_failure(int* status, int code, volatile int* abort_flag) {
  *abort_flag = 1;
  atomicCAS(status, 0, code);
}

// acc (raw 32-bit from TMEM) -> scaled/activated fp32, in the reference's
// operation order: float(acc); (v * sa[row]) * sb[col]; + bias; activation.  Scales
// and bias are rounded one by one, here and wherever a kernel does the same on
// several values at once.
template <bool IS_INT>
__device__ __forceinline__ float epilogue_value(uint32_t raw, float sa, float sb, float bias, int epi, bool scaled) {
  float v = IS_INT ? static_cast<float>(static_cast<int32_t>(raw)) : __uint_as_float(raw);
  if (scaled) v = __fmul_rn(__fmul_rn(v, sa), sb);
  if (epi != EPI_NONE) {
    v = __fadd_rn(v, bias);
    if (epi == EPI_BIAS_RELU) {
      v = fmaxf(v, 0.0f);
    } else if (epi == EPI_BIAS_SILU) {
      v = v * (1.0f / (1.0f + __expf(-v)));
    } else if (epi == EPI_BIAS_GELU) {
      float y = 0.7978845608f * (v + 0.044715f * (v * v * v));
      float e = __expf(-2.0f * fabsf(y));
      float num = (y > 0.0f) ? 2.0f : 2.0f * e;
      v = 0.5f * v * (num * (1.0f / (1.0f + e)));
    }
  }
  return v;
}

template <int OUTMODE>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (OUTMODE == OUT_FP16) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  } else {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  }
}
template <int OUTMODE>
__device__ __forceinline__ uint16_t pack1(float v) {
  if constexpr (OUTMODE == OUT_FP16) {
    __half h = __float2half_rn(v);
    return *reinterpret_cast<uint16_t*>(&h);
  } else {
    __nv_bfloat16 h = __float2bfloat16_rn(v);
    return *reinterpret_cast<uint16_t*>(&h);
  }
}
template <int OUTMODE>
__device__ __forceinline__ float load_bias(const void* bias, int col) {
  if constexpr (OUTMODE == OUT_FP16) {
    return __half2float(reinterpret_cast<const __half*>(bias)[col]);
  } else {
    return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(bias)[col]);
  }
}

// 1 / x for 1 <= x < 2^126: the hardware estimate and one Newton-Raphson step whose residual is exact in
// an FMA (Markstein, "Computation of elementary functions on the IBM RISC System/6000", 1990).  Equal to
// the IEEE quotient but for at most 32 of the 2^23 mantissas, where it is one unit off with an error of
// 0.5 + 2^-20 units (tests/test_rows_epilogue_gpu.py), and without its branch.
__device__ __forceinline__ float reciprocal_of(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return fmaf(r, fmaf(-x, r, 1.0f), r);
}

// The activation of epilogue_value on N values at once: the kind is a template argument and nothing
// branches per value, so the chains (exponential, reciprocal) overlap.  The operations and their order
// are those of epilogue_value but for the reciprocal of the silu and gelu denominators, which
// reciprocal_of takes without a division: for at most 32 of its 2^23 mantissas one unit of fp32 apart.
template <int EPI, int N>
__device__ __forceinline__ void activate(float (&v)[N]) {
  if constexpr (EPI == EPI_BIAS_RELU) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = fmaxf(v[i], 0.0f);
  } else if constexpr (EPI == EPI_BIAS_SILU) {
    float d[N];
    bool plain = true;  // false for a value below -87 (its denominator leaves the range above) or NaN
#pragma unroll
    for (int i = 0; i < N; ++i) {
      d[i] = 1.0f + __expf(-v[i]);
      plain &= d[i] < 8.5e37f;
    }
    if (plain) {
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = v[i] * reciprocal_of(d[i]);
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = v[i] * (1.0f / d[i]);
    }
  } else if constexpr (EPI == EPI_BIAS_GELU) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float y = 0.7978845608f * (v[i] + 0.044715f * (v[i] * v[i] * v[i]));
      const float e = __expf(-2.0f * fabsf(y));
      const float num = (y > 0.0f) ? 2.0f : 2.0f * e;
      v[i] = 0.5f * v[i] * (num * reciprocal_of(1.0f + e));
    }
  }
}
template <int N>
__device__ __forceinline__ void activate(int epi, float (&v)[N]) {
  switch (epi) {
    case EPI_BIAS_RELU: return activate<EPI_BIAS_RELU>(v);
    case EPI_BIAS_SILU: return activate<EPI_BIAS_SILU>(v);
    case EPI_BIAS_GELU: return activate<EPI_BIAS_GELU>(v);
  }
}

// Channel scales and bias of 32 neighbouring columns from `col` on (a multiple of 8; N is a multiple of
// 16, so eight columns exist together).  Every lane reads the same addresses: 16-byte loads where the two
// vectors start on 16 bytes (`vec`), single elements otherwise.  Without scales the factor is one.
struct ColumnFactors {
  float sb[32];
  uint32_t bias[16];  // pairs in the output type
};
__device__ __forceinline__ void load_column_factors(ColumnFactors& f, const GemmParams& p, int col, bool scaled, bool vec) {
  const uint16_t* bias = reinterpret_cast<const uint16_t*>(p.bias);
  const bool biased = p.epilogue != EPI_NONE;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const int c = col + 8 * g;
    const bool in = c < p.N;
    if (vec) {
      float4 s0 = make_float4(1.0f, 1.0f, 1.0f, 1.0f), s1 = s0;
      uint4 b = make_uint4(0u, 0u, 0u, 0u);
      if (scaled && in) {
        s0 = __ldg(reinterpret_cast<const float4*>(p.sb + c));
        s1 = __ldg(reinterpret_cast<const float4*>(p.sb + c + 4));
      }
      if (biased && in) b = __ldg(reinterpret_cast<const uint4*>(bias + c));
      f.sb[8 * g] = s0.x, f.sb[8 * g + 1] = s0.y, f.sb[8 * g + 2] = s0.z, f.sb[8 * g + 3] = s0.w;
      f.sb[8 * g + 4] = s1.x, f.sb[8 * g + 5] = s1.y, f.sb[8 * g + 6] = s1.z, f.sb[8 * g + 7] = s1.w;
      f.bias[4 * g] = b.x, f.bias[4 * g + 1] = b.y, f.bias[4 * g + 2] = b.z, f.bias[4 * g + 3] = b.w;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) f.sb[8 * g + i] = scaled && in ? __ldg(p.sb + c + i) : 1.0f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t lo = biased && in ? __ldg(bias + c + 2 * i) : 0u, hi = biased && in ? __ldg(bias + c + 2 * i + 1) : 0u;
        f.bias[4 * g + i] = lo | (hi << 16);
      }
    }
  }
}

// 32 raw accumulators of one row -> scaled, biased, activated, 16-bit; `emit(g, pairs)` takes eight
// columns (8 g ...).  The order of epilogue_value, every operation rounded by itself.  One value at a
// time, with its own switch on the activation, its own division and two scalar loads, the epilogue warps
// took longer than the mainloop they overlap: int8 997 x 10208 x 5120, bias and gelu, 115.7 us for the
// kernel, 52 this way.  Eight epilogue warps instead of four matter where K is short: 2048 x 8192 x 2048 with
// bias and silu 64.4 -> 44.7 us, gelu 54.0 -> 42.5, none 32.2 -> 32.0.
template <bool IS_INT, int OUTMODE, int EPI, typename EmitFn>
__device__ __forceinline__ void epilogue_32(const uint32_t (&r)[32], float sa, const ColumnFactors& f, EmitFn emit) {
  float v[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const float acc = IS_INT ? static_cast<float>(static_cast<int32_t>(r[i])) : __uint_as_float(r[i]);
    v[i] = __fmul_rn(__fmul_rn(acc, sa), f.sb[i]);
    if constexpr (EPI != EPI_NONE) {
      const uint16_t h = static_cast<uint16_t>(f.bias[i / 2] >> (16 * (i & 1)));
      v[i] = __fadd_rn(v[i], load_bias<OUTMODE>(&h, 0));
    }
  }
  activate<EPI>(v);
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    uint32_t pk[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) pk[i] = pack2<OUTMODE>(v[8 * g + 2 * i], v[8 * g + 2 * i + 1]);
    emit(g, pk);
  }
}
template <bool IS_INT, int OUTMODE, typename EmitFn>
__device__ __forceinline__ void epilogue_32(int epi, const uint32_t (&r)[32], float sa, const ColumnFactors& f, EmitFn emit) {
  switch (epi) {
    case EPI_BIAS: return epilogue_32<IS_INT, OUTMODE, EPI_BIAS>(r, sa, f, emit);
    case EPI_BIAS_RELU: return epilogue_32<IS_INT, OUTMODE, EPI_BIAS_RELU>(r, sa, f, emit);
    case EPI_BIAS_SILU: return epilogue_32<IS_INT, OUTMODE, EPI_BIAS_SILU>(r, sa, f, emit);
    case EPI_BIAS_GELU: return epilogue_32<IS_INT, OUTMODE, EPI_BIAS_GELU>(r, sa, f, emit);
    default: return epilogue_32<IS_INT, OUTMODE, EPI_NONE>(r, sa, f, emit);
  }
}

// One warp's share (32 rows x BN columns) of an accumulator tile: TMEM ->
// registers -> scale / bias / activation -> bf16|fp16 -> 128-byte-swizzled
// staging buffer -> TMA store (clipped at M and N), or raw 32-bit stores.
// `release_tmem()` is called once, as soon as the accumulator has been read.
// `tmC` points to `n_dst` tensor maps: the staged chunk is stored through each
// of them (the caller's own output, or the same window of the output buffers of
// several GPUs), starting with map `dst_first` (+ a per-tile, per-warp rotation)
// so that neither the ranks nor the tiles of one rank all hit the same peer at
// the same time.
// cbufs: staging buffers of this warp at `stage_c` (two: the store of one chunk overlaps the
// conversion of the next; one: where shared memory is short).
// share: warps that share these 32 rows; this one, `part`, takes every share-th chunk of 64 columns.
template <int KIND, int OUTMODE, typename ReleaseFn>
__device__ __forceinline__ void epilogue_warp_tile(const GemmParams& p, const CUtensorMap* tmC, int n_dst, int dst_first,
                                                   uint32_t t_row, int m0, int n0, int BN, int lane, uint32_t stage_c,
                                                   int& cbuf, ReleaseFn release_tmem, int cbufs = 2, int share = 1, int part = 0) {
  using KT = KindTraits<KIND>;
  constexpr int C_BUF = 32 * 128;
  const bool scaled = (p.sa != nullptr) && (p.sb != nullptr);
  const int row = m0 + lane;
  const float sa_v = !scaled ? 1.0f : row < p.M ? __ldg(p.sa + row) : 0.0f;
  if constexpr (OUTMODE == OUT_RAW32) {
    uint32_t* out = reinterpret_cast<uint32_t*>(p.c);
#pragma unroll 1
    for (int c0 = 32 * part; c0 < BN; c0 += 32 * share) {
      uint32_t r[32];
      tmem_ld_x32(t_row + c0, r);
      tmem_ld_wait();
      if (row < p.M) {
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const int col = n0 + c0 + j;
          if (col + 3 < p.N) {
            *reinterpret_cast<uint4*>(out + static_cast<size_t>(row) * p.N + col) =
                make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
          } else {
            for (int e = 0; e < 4; ++e)
              if (col + e < p.N) out[static_cast<size_t>(row) * p.N + col + e] = r[j + e];
          }
        }
      }
    }
    release_tmem();
  } else {
    const bool vec = ((reinterpret_cast<uintptr_t>(p.sb) | reinterpret_cast<uintptr_t>(p.bias)) & 15u) == 0;
    ColumnFactors f;
    if (64 * part >= BN) release_tmem();  // nothing to do for this warp
#pragma unroll 1
    for (int c0 = 64 * part; c0 < BN; c0 += 64 * share) {
      if (c0 + 64 > BN) {
        // Last 32 columns of a tile whose width is not a multiple of 64: a
        // 64-column TMA box would reach into the neighbouring tile, so these
        // leave the registers directly (64 contiguous bytes per row).
        uint32_t r[32];
        tmem_ld_x32(t_row + c0, r);
        load_column_factors(f, p, n0 + c0, scaled, vec);
        tmem_ld_wait();
        release_tmem();
        if (row < p.M) {
          uint16_t* out_row = reinterpret_cast<uint16_t*>(p.c) + static_cast<size_t>(row) * p.N;
          epilogue_32<KT::is_int, OUTMODE>(p.epilogue, r, sa_v, f, [&](int g, const uint32_t (&pk)[4]) {
            const int col = n0 + c0 + 8 * g;
            if (col < p.N) *reinterpret_cast<uint4*>(out_row + col) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          });
        }
        break;
      }
      // the store that last used this buffer (two chunks ago with two buffers) has to be done reading it
      if (lane == 0) {
        if (cbufs == 1) bulk_wait_group_read<0>();
        else bulk_wait_group_read<1>();
      }
      __syncwarp();
      const uint32_t cdst = stage_c + cbuf * C_BUF + lane * 128;
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        uint32_t r[32];
        tmem_ld_x32(t_row + c0 + 32 * h, r);
        load_column_factors(f, p, n0 + c0 + 32 * h, scaled, vec);
        tmem_ld_wait();
        // this warp's last read of the accumulator: hand the TMEM buffer back
        if (h == 1 && c0 + 64 * share >= BN) release_tmem();
        epilogue_32<KT::is_int, OUTMODE>(p.epilogue, r, sa_v, f, [&](int g, const uint32_t (&pk)[4]) {
          const int chunk = 4 * h + g;  // 16-byte chunk index inside the 128-byte row
          st_smem_v4(cdst + static_cast<uint32_t>(((chunk ^ (lane & 7)) << 4)), pk[0], pk[1], pk[2], pk[3]);
        });
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (m0 < p.M && (n0 + c0) < p.N) {
          for (int d = 0; d < n_dst; ++d) {
            int which = (dst_first + d) % n_dst;
            tma_store_2d(tmC + which, stage_c + cbuf * C_BUF, n0 + c0, m0);
          }
        }
        bulk_commit_group();
      }
      cbuf = cbufs == 1 ? 0 : cbuf ^ 1;
    }
  }
}

// ===========================================================================
// Large-M kernel
// ===========================================================================
// Shared-memory carve-up of the large-M kernel for a tile width `bn` and a ring
// depth `stages` (computed identically on host and device).
struct RowsLayout {
  int a_stage, b_stage, off_b, off_c, off_bar, off_misc, total;
};
constexpr int ROWS_C_BUF = 32 * 128;  // staging buffer: 32 rows x 64 two-byte columns
constexpr int ROWS_THREADS = 64 + 8 * 32;  // at most: producer, MMA issuer, eight epilogue warps (two per 32 rows); or four
constexpr int ROWS_ACC_COLS = 256;    // TMEM columns between the two accumulator buffers
__host__ __device__ inline RowsLayout rows_layout(int bn, int stages) {
  RowsLayout l;
  l.a_stage = BLOCK_ROWS * KBLOCK_BYTES;
  l.b_stage = bn * KBLOCK_BYTES;
  l.off_b = stages * l.a_stage;
  l.off_c = l.off_b + stages * l.b_stage;       // eight buffers: one per epilogue warp, or two for each of four
  l.off_bar = l.off_c + 8 * ROWS_C_BUF;         // full[S], empty[S], tfull[2], tempty[2]
  l.off_misc = l.off_bar + 8 * (2 * stages + 4);
  l.total = l.off_misc + 16;
  return l;
}

constexpr int MAX_DESTINATIONS = 8;
struct OutputMaps {
  CUtensorMap m[MAX_DESTINATIONS];
};

// Body shared by the two entry kernels below: `tmC` points to `n_dst` output
// tensor maps (kernel parameters of the caller).  The tile width (p.bn, a
// multiple of 32 up to 256) and the ring depth (p.rows_stages) are run-time
// values: the host picks the width that fills the SMs in whole waves.
template <int KIND, int OUTMODE>
__device__ __forceinline__ void gemm_rows_body(const CUtensorMap& tmA, const CUtensorMap* tmC_ptr, int n_dst,
                                               int dst_first, const GemmParams& p) {
  const CUtensorMap& tmC = *tmC_ptr;
#ifdef FLYB200_PROFILE
  long long prof_wait[4] = {0, 0, 0, 0};  // producer:empty, mma:tempty, mma:full, epilogue:tfull
  const long long prof_begin = clock64();
#endif
  using KT = KindTraits<KIND>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t smem_base = smem_u32(smem_raw);
  const int BN = p.bn;
  const int STAGES = p.rows_stages;
  const RowsLayout L = rows_layout(BN, STAGES);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_raw + L.off_misc + 4);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + L.off_misc);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const uint32_t bar_full = smem_base + L.off_bar;
  const uint32_t bar_empty = bar_full + 8 * STAGES;
  const uint32_t bar_tfull = bar_empty + 8 * STAGES;
  const uint32_t bar_tempty = bar_tfull + 16;

  if ((smem_base & 1023u) != 0) {  // uniform over the CTA: the swizzle atoms need 1024-byte alignment
    if (threadIdx.x == 0) atomicCAS(p.status, 0, ST_SMEM_ALIGN);
    return;
  }
  // Programmatic dependent launch (p.pdl != 0): this kernel runs its set-up (barriers, TMEM) while the previous one
  // finishes; no global memory is read or written before griddepcontrol.wait below.  After it the next kernel on
  // the stream may be scheduled onto SMs as this one frees them.

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_tfull + 8 * s, 1);
      mbar_init(bar_tempty + 8 * s, (blockDim.x - 64) >> 5);  // every epilogue warp
    }
    abort_flag[0] = 0;
    abort_flag[1] = 0;  // stays zero: lets the drain below wait on time alone
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&tmA);
    if (OUTMODE != OUT_RAW32) prefetch_tensormap(&tmC);
  }
  constexpr uint32_t TMEM_COLS = 512;  // two accumulator buffers of up to 256 columns
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (p.pdl) {
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the previous kernel has completed
    pdl_trigger();
  }

  const int num_m = (p.M + BLOCK_ROWS - 1) / BLOCK_ROWS;
  const int num_n = (p.N + BN - 1) / BN;
  const int num_tiles = num_m * num_n;
  const int num_kb = p.K_bytes / KBLOCK_BYTES;
  const int gm_full = p.group_m;

  // Tile order: groups of `group_m` row tiles; inside a group the row tile
  // changes fastest and the channel tiles are walked once, so the group's
  // activations stay in L2 while the weights stream through.  Odd groups walk
  // the channels backwards: the weight tiles that the previous group touched
  // last are the first ones the next group asks for.
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

  // Work items: the tiles of the whole rounds, then those of the last, partial round in `parts` column
  // strips each, so that the round costs a strip instead of a tile (host: rows_tail_parts).
  const int parts = p.tail_parts;
  const int whole = parts > 1 ? num_tiles - num_tiles % static_cast<int>(gridDim.x) : num_tiles;
  const int items = whole + (num_tiles - whole) * parts;
  const int strip = BN / parts;
  // item -> row tile, first column and width; false where the strip lies past the last column
  auto item_coords = [&](int i, int& m_blk, int& n0, int& width) {
    int n_blk;
    if (i < whole) {
      tile_coords(i, m_blk, n_blk);
      n0 = n_blk * BN;
      width = BN;
      return true;
    }
    const int j = i - whole;
    tile_coords(whole + j / parts, m_blk, n_blk);
    n0 = n_blk * BN + j % parts * strip;
    width = strip;
    return n0 < p.N;
  };

  if (warp == 0) {
    // ------------------------------ producer ------------------------------
    const bool issuer = elect_one();  // the whole warp runs the loop, here and in the MMA warp, and one lane issues (ptx.cuh)
    const uint64_t pol_a = l2_policy_evict_last();
    const uint64_t pol_w = l2_policy_evict_last();
    int stage = 0;
    uint32_t phase = 0;
    int issued = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
      int m_blk, n0, width;
      if (!item_coords(t, m_blk, n0, width)) continue;
      const uint32_t w_rows = static_cast<uint32_t>(min(width, p.N - n0));
      const uint32_t w_bytes = w_rows * KBLOCK_BYTES;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait_warp(bar_empty + 8 * stage, phase ^ 1u, abort_flag FLYB200_PROF_ARG(&prof_wait[0]))) {
          report_failure(p.status, ST_TIMEOUT, abort_flag);
          ok = false;
          break;
        }
        const uint32_t fb = bar_full + 8 * stage;
        if (issuer) {
          mbar_expect_tx(fb, L.a_stage + w_bytes);
          tma_load_2d(smem_base + stage * L.a_stage, &tmA, fb, kb * KBLOCK_BYTES, m_blk * BLOCK_ROWS, pol_a);
          bulk_load_1d(smem_base + L.off_b + stage * L.b_stage,
                       p.w + (static_cast<size_t>(kb) * p.N + n0) * KBLOCK_BYTES, w_bytes, fb, pol_w);
        }
        ++issued;
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (!ok || *abort_flag) {
      // Drain: wait (bounded) for the copies this warp still has in flight
      // so that none lands in shared memory after the CTA has gone.
      const int pending = min(issued, STAGES);
      for (int i = 0; i < pending; ++i) {
        int s = stage - 1 - i;
        uint32_t ph = phase;
        if (s < 0) {
          s += STAGES;
          ph ^= 1u;
        }
        mbar_wait(bar_full + 8 * s, ph, abort_flag + 1 /* never set: wait on time only */);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issue -----------------------------
    const bool issuer = elect_one();
    const uint64_t adesc0 = umma_desc_sw128_kmajor(smem_base), bdesc0 = umma_desc_sw128_kmajor(smem_base + L.off_b);
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
      int m_blk, n0, width;
      if (!item_coords(t, m_blk, n0, width)) continue;
      const uint32_t idesc = umma_idesc(KT::dfmt, KT::abfmt, BLOCK_ROWS, static_cast<uint32_t>(width));
      if (!mbar_wait_warp(bar_tempty + 8 * acc, acc_phase ^ 1u, abort_flag FLYB200_PROF_ARG(&prof_wait[1]))) {
        report_failure(p.status, ST_TIMEOUT, abort_flag);
        break;
      }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * ROWS_ACC_COLS);
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait_warp(bar_full + 8 * stage, phase, abort_flag FLYB200_PROF_ARG(&prof_wait[2]))) {
          report_failure(p.status, ST_TIMEOUT, abort_flag);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t adesc = adesc0 + static_cast<uint32_t>(stage * (L.a_stage >> 4));
        const uint64_t bdesc = bdesc0 + static_cast<uint32_t>(stage * (L.b_stage >> 4));
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
    const int q = warp & 3;  // TMEM lane quadrant this warp may read
    const int ew = warp - 2; // staging buffer owner
    const int share = (static_cast<int>(blockDim.x) - 64) >> 7;  // epilogue warps per 32 rows (host: rows_epilogue_warps)
    const int cbufs = 2 / share;
    const uint32_t stage_c = smem_base + L.off_c + ew * cbufs * ROWS_C_BUF;
    int acc = 0;
    uint32_t acc_phase = 0;
    int cbuf = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
      int m_blk, n0, width;
      if (!item_coords(t, m_blk, n0, width)) continue;
      const int m0 = m_blk * BLOCK_ROWS + q * 32;
      if (!mbar_wait(bar_tfull + 8 * acc, acc_phase, abort_flag FLYB200_PROF_ARG(&prof_wait[3]))) {
        if (lane == 0) report_failure(p.status, ST_TIMEOUT, abort_flag);
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t t_row =
          tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * ROWS_ACC_COLS);
      // own buffer first for the first tile; every further tile and warp starts one destination later
      const int first = n_dst > 1 ? (dst_first + (t / static_cast<int>(gridDim.x)) + ew) % n_dst : 0;
      epilogue_warp_tile<KIND, OUTMODE>(p, tmC_ptr, n_dst, first, t_row, m0, n0, width, lane, stage_c, cbuf, [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_tempty + 8 * acc);
      }, cbufs, share, ew >> 2);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
    if (lane == 0) bulk_wait_group<0>();
  }

#ifdef FLYB200_PROFILE
  if (lane == 0) {
    const long long total = clock64() - prof_begin;
    if (warp == 0) {
      atomicAdd(p.prof + 0, static_cast<unsigned long long>(prof_wait[0]));
      atomicAdd(p.prof + 4, static_cast<unsigned long long>(total));
    } else if (warp == 1) {
      atomicAdd(p.prof + 1, static_cast<unsigned long long>(prof_wait[1]));
      atomicAdd(p.prof + 2, static_cast<unsigned long long>(prof_wait[2]));
    } else if (warp == 2) {
      atomicAdd(p.prof + 3, static_cast<unsigned long long>(prof_wait[3]));
      atomicAdd(p.prof + 5, static_cast<unsigned long long>(total));
    }
  }
#endif
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// One output buffer (the regular GEMM).
template <int KIND, int OUTMODE>
__global__ void __launch_bounds__(ROWS_THREADS, 1)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmC,
                 const GemmParams p) {
  gemm_rows_body<KIND, OUTMODE>(tmA, &tmC, 1, 0, p);
}

// Every output tile is stored into the same window of up to eight buffers, e.g.
// the full-width output of each GPU of a column-parallel group (peer-mapped
// memory; plain TMA stores, per CTA, no multicast): the all-gather of the
// shards happens tile by tile inside the GEMM.
template <int KIND, int OUTMODE>
__global__ void __launch_bounds__(ROWS_THREADS, 1)
gemm_rows_scatter_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ OutputMaps outs,
                         const GemmParams p) {
  gemm_rows_body<KIND, OUTMODE>(tmA, outs.m, p.n_dst, p.dst_first, p);
}

}  // namespace flyb200
