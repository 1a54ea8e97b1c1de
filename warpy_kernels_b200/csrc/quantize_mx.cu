// MXFP8 quantiser: rows of bf16 / fp32 values -> e4m3 codes plus one ue8m0 scale
// byte per block of 32 consecutive elements.
//
// Arithmetic (bit-exact with the reference's GEMM epilogue quantiser,
// warpy_kernels/gemm/sm89.py:65-93 with warpy_kernels/ptx/common.py:539-565 and
// warpy_kernels/ptx/sm89.py:85-93):
//   A    = max_i (bits(x_i) & 0x7fffffff)                  integer max of |x| bit patterns
//   e    = clamp(((A + 0x1fffff) >> 23) - 8, 0, 254)        scale byte, value 2^(e-127)
//   inv  = float_from_bits(max(254 - e, 1) << 23)           2^(127-e)
//   code = cvt.rn.satfinite.e4m3(x_i * inv)
//
// HBM-bound: 2 (bf16) or 4 (fp32) bytes in, 1 + 1/32 bytes out per element.  Two threads own one block of 32 elements
// (16 each: one 32-byte load for bf16, one 16-byte store of codes), four blocks' scale bytes leave as one word, and a
// CTA covers 1024 consecutive groups and ends: [8192, 14336] bf16 takes 55.4 us (6.43 TB/s, what a plain copy reaches).
// With 8 elements per thread and a grid of resident CTAs that stride through the matrix it was 61.7 us; the same loads
// in such a grid measure 59.5-62 us.
#include "common.cuh"
#include "host_common.h"

namespace wk {
namespace {

constexpr int kThreads = 512;
constexpr int kUnroll = 2;
constexpr int kGroup = 16;  // elements per thread and step

// 16 elements as fp32 bit patterns.  WIDE: 32-byte aligned.
template <bool WIDE>
__device__ __forceinline__ void load32(const void* p, uint32_t (&w)[8]) {
  if (WIDE) {
    asm volatile(
        "ld.global.L1::no_allocate.L2::evict_first.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
        : "l"(p));
  } else {
    const uint4 a = __ldcs(static_cast<const uint4*>(p)), b = __ldcs(static_cast<const uint4*>(p) + 1);
    w[0] = a.x, w[1] = a.y, w[2] = a.z, w[3] = a.w, w[4] = b.x, w[5] = b.y, w[6] = b.z, w[7] = b.w;
  }
}
template <bool WIDE>
__device__ __forceinline__ void load16(const __nv_bfloat16* p, uint32_t (&v)[16]) {
  uint32_t w[8];
  load32<WIDE>(p, w);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[2 * i] = w[i] << 16;
    v[2 * i + 1] = w[i] & 0xffff0000u;
  }
}
template <bool WIDE>
__device__ __forceinline__ void load16(const float* p, uint32_t (&v)[16]) {
  uint32_t w[8];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    load32<WIDE>(p + 8 * h, w);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[8 * h + i] = w[i];
  }
}

// The scale byte and the multiplier for one block's integer amax.
__device__ __forceinline__ void mx_scale(uint32_t amax_bits, uint32_t& e, float& inv) {
  int t = static_cast<int>((amax_bits + 0x1fffffu) >> 23) - 8;
  t = max(t, 0);
  t = min(t, 254);
  e = static_cast<uint32_t>(t);
  inv = __uint_as_float(static_cast<uint32_t>(max(254 - t, 1)) << 23);
}

// CONTIG: rows are back to back (ld_x == cols), so input, code and scale offsets are all linear in the group index and
// no division is needed.  WIDE: rows of x start on 32-byte boundaries, q on a 16-byte and s on a 4-byte one.
template <typename T, bool CONTIG, bool WIDE>
__global__ void __launch_bounds__(kThreads)
quantize_mx_kernel(const T* __restrict__ x, int64_t ld_x, uint8_t* __restrict__ q,
                   uint8_t* __restrict__ s, int64_t total_groups, int groups_per_row) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t base = static_cast<int64_t>(blockIdx.x) * (kThreads * kUnroll) + threadIdx.x;
  uint32_t v[kUnroll][16];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int64_t g = base + u * kThreads;
    if (g < total_groups) {
      int64_t off = g * kGroup;
      if (!CONTIG) {
        const uint32_t row = static_cast<uint32_t>(g / groups_per_row);
        off = row * ld_x + (g - static_cast<int64_t>(row) * groups_per_row) * kGroup;
      }
      load16<WIDE>(x + off, v[u]);
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[u][i] = 0;
    }
  }
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int64_t g = base + u * kThreads;
    uint32_t amax = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = max(amax, v[u][i] & 0x7fffffffu);
    amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    uint32_t e;
    float inv;
    mx_scale(amax, e, inv);
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      w[i] = pack_e4m3x4(__fmul_rn(__uint_as_float(v[u][4 * i]), inv), __fmul_rn(__uint_as_float(v[u][4 * i + 1]), inv),
                         __fmul_rn(__uint_as_float(v[u][4 * i + 2]), inv),
                         __fmul_rn(__uint_as_float(v[u][4 * i + 3]), inv));
    // the scale bytes of the next three blocks
    const uint32_t e1 = __shfl_down_sync(0xffffffffu, e, 2), e2 = __shfl_down_sync(0xffffffffu, e, 4),
                   e3 = __shfl_down_sync(0xffffffffu, e, 6);
    if (g >= total_groups) continue;
    // the outputs are contiguous [rows, cols] and [rows, cols / 32]: linear in g whatever ld_x is
    if (WIDE) {
      *reinterpret_cast<uint4*>(q + g * kGroup) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
      reinterpret_cast<uint2*>(q + g * kGroup)[0] = make_uint2(w[0], w[1]);
      reinterpret_cast<uint2*>(q + g * kGroup)[1] = make_uint2(w[2], w[3]);
    }
    if (WIDE && (g | 7) < total_groups) {
      if ((g & 7) == 0) *reinterpret_cast<uint32_t*>(s + (g >> 1)) = e | e1 << 8 | e2 << 16 | e3 << 24;
    } else if ((g & 1) == 0) {
      s[g >> 1] = static_cast<uint8_t>(e);
    }
  }
}

template <typename T>
int launch(const T* x, int64_t rows, int64_t cols, int64_t ld_x, uint8_t* q, uint8_t* s,
           cudaStream_t stream) {
  int64_t total = rows * (cols / kGroup);
  int per_row = static_cast<int>(cols / kGroup);
  const int64_t grid = (total + kThreads * kUnroll - 1) / (kThreads * kUnroll);
  if (grid > INT32_MAX) return WK_E_ARG;
  const bool contig = ld_x == cols || rows == 1;
  const bool wide = reinterpret_cast<uintptr_t>(x) % 32 == 0 && (contig || ld_x * sizeof(T) % 32 == 0) &&
                    reinterpret_cast<uintptr_t>(q) % 16 == 0 && reinterpret_cast<uintptr_t>(s) % 4 == 0;
  const void* kernel = contig ? (wide ? reinterpret_cast<const void*>(quantize_mx_kernel<T, true, true>)
                                      : reinterpret_cast<const void*>(quantize_mx_kernel<T, true, false>))
                              : (wide ? reinterpret_cast<const void*>(quantize_mx_kernel<T, false, true>)
                                      : reinterpret_cast<const void*>(quantize_mx_kernel<T, false, false>));
  return launch_pdl(kernel, dim3(static_cast<unsigned>(grid)), kThreads, 0, stream, 1,
                    {&x, &ld_x, &q, &s, &total, &per_row});
}

}  // namespace
}  // namespace wk

extern "C" int wk_quantize_mx(const void* x, int dtype, int64_t rows, int64_t cols, int64_t ld_x,
                              void* q, void* s, void* stream) {
  if (rows < 0 || cols < 0 || cols % 32 != 0 || ld_x < cols || ld_x % 8 != 0) return WK_E_ARG;
  if (cols / 8 > 0x7fffffff || rows > 0x7fffffff) return WK_E_ARG;
  if (rows == 0 || cols == 0) return 0;
  if (!x || !q || !s || !wk::aligned16(x) || (reinterpret_cast<uintptr_t>(q) & 7)) return WK_E_ARG;
  if (int unsupported = wk::require_sm100()) return unsupported;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == WK_BF16)
    return wk::launch(static_cast<const __nv_bfloat16*>(x), rows, cols, ld_x,
                      static_cast<uint8_t*>(q), static_cast<uint8_t*>(s), st);
  if (dtype == WK_F32)
    return wk::launch(static_cast<const float*>(x), rows, cols, ld_x, static_cast<uint8_t*>(q),
                      static_cast<uint8_t*>(s), st);
  return WK_E_ARG;
}
