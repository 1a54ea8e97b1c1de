// Rows of the attention forward that its tensor-core kernels cannot represent (FP8 and BF16 inputs).
//
// Those kernels keep one reference exponent per query row, fixed by the row's first 64 keys, and hold scores up to
// 2^100 above it.  A row that meets a later key beyond that range is computed again by the threads that store it, in
// fp32 on the CUDA cores, against the exact row maximum, which they know by then; the reference reaches the same result
// by moving its reference with every 128-key tile and rescaling O (warpy_kernels/attn/fwd_base.py:337-360).  Inputs
// that need it are pathological (one key more than 69 nats above the start of the row), so this path is written for
// clarity, not speed.  The persistent kernel, whose registers are full, only marks such a query block and goes through its
// marked blocks when it has nothing else left to do.  Inside the kernel it costs nothing where no row needs it; as a kernel of its own behind every
// forward, which looked for flagged blocks, it cost a launch: 2 us per call on the GPU and 3 us on the host.
#pragma once
#include "common.cuh"
#include "host_common.h"

namespace wk {

// What the recomputation reads, kept beside a kernel's other parameters.
struct ExactInputs {
  const uint8_t* q;
  const uint8_t* k;
  const uint8_t* v;
  int64_t q_strides[3], k_strides[3], v_strides[3];  // bytes
  int d;
  int* flags;  // the call's workspace, one word per query block (zero between calls), or null: the caller passed
               // none, and the status word reports such a row instead
};

inline ExactInputs exact_inputs(const wk_attn_fwd_args* a, int size) {
  ExactInputs e;
  e.q = static_cast<const uint8_t*>(a->q);
  e.k = static_cast<const uint8_t*>(a->k);
  e.v = static_cast<const uint8_t*>(a->v);
  for (int i = 0; i < 3; ++i) {
    e.q_strides[i] = a->q_strides[i] * size;
    e.k_strides[i] = a->k_strides[i] * size;
    e.v_strides[i] = a->v_strides[i] * size;
  }
  e.d = a->d;
  e.flags = static_cast<int*>(a->workspace);
  return e;
}

// 4 bytes as fp32: 4 e4m3 or 2 bf16 values.
template <bool BF16>
__device__ __forceinline__ void unpack4(uint32_t w, float (&x)[4]) {
  if (BF16) {
    x[0] = __uint_as_float(w << 16);
    x[1] = __uint_as_float(w & 0xffff0000u);
  } else {
    unpack_e4m3x2(static_cast<uint16_t>(w & 0xffffu), x[0], x[1]);
    unpack_e4m3x2(static_cast<uint16_t>(w >> 16), x[2], x[3]);
  }
}

struct ExactRow {
  float m, l;  // largest score in base 2 and the sum of the probabilities relative to it
};

// Computes head-dim columns [col0, col0 + 32) of one output row, whose last visible key is `limit`, stores them at `dst`.
template <bool BF16>
__device__ __noinline__ ExactRow exact_row32(const ExactInputs& e, int b, int hq, int hkv, int row, int limit, float beta,
                                             float sv, int col0, __nv_bfloat16* dst) {
  constexpr int PER = BF16 ? 2 : 4, SIZE = BF16 ? 2 : 1;  // elements per word, bytes per element
  const uint8_t* q = e.q + b * e.q_strides[0] + hq * e.q_strides[1] + row * e.q_strides[2];
  const uint8_t* k = e.k + b * e.k_strides[0] + hkv * e.k_strides[1];
  const uint8_t* v = e.v + b * e.v_strides[0] + hkv * e.v_strides[1] + col0 * SIZE;
  auto score = [&](int key) {
    float s = 0.f;
#pragma unroll 1
    for (int c = 0; c < e.d; c += PER) {
      float x[4], y[4];
      unpack4<BF16>(*reinterpret_cast<const uint32_t*>(q + c * SIZE), x);
      unpack4<BF16>(*reinterpret_cast<const uint32_t*>(k + key * e.k_strides[2] + c * SIZE), y);
#pragma unroll
      for (int i = 0; i < PER; ++i) s = fmaf(x[i], y[i], s);
    }
    return s * beta;
  };
  float m = -INFINITY;
#pragma unroll 1
  for (int key = 0; key <= limit; ++key) m = fmaxf(m, score(key));
  float l = 0.f, o[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) o[i] = 0.f;
#pragma unroll 1
  for (int key = 0; key <= limit; ++key) {
    const float p = exp2f(score(key) - m);
    l += p;
#pragma unroll
    for (int c = 0; c < 32; c += PER) {
      float y[4];
      unpack4<BF16>(*reinterpret_cast<const uint32_t*>(v + key * e.v_strides[2] + c * SIZE), y);
#pragma unroll
      for (int i = 0; i < PER; ++i) o[c + i] = fmaf(p, y[i], o[c + i]);
    }
  }
  const float inv = l > 0.f ? sv / l : 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint4 w;
    w.x = pack_bf16x2(o[8 * i + 0] * inv, o[8 * i + 1] * inv);
    w.y = pack_bf16x2(o[8 * i + 2] * inv, o[8 * i + 3] * inv);
    w.z = pack_bf16x2(o[8 * i + 4] * inv, o[8 * i + 5] * inv);
    w.w = pack_bf16x2(o[8 * i + 6] * inv, o[8 * i + 7] * inv);
    reinterpret_cast<uint4*>(dst)[i] = w;
  }
  return {m, l};
}

}  // namespace wk
