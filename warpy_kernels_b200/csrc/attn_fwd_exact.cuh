// Query blocks of the attention forward that its tensor-core kernels cannot represent (FP8 and BF16 inputs).
//
// Those kernels keep one reference exponent per query row, fixed by the row's first 64 keys, and hold scores up to
// 2^100 above it.  A row that meets a later key beyond that range is computed again in fp32 on the CUDA cores, with a
// row maximum that moves; the reference reaches the same result by moving its reference with every 128-key tile and
// rescaling O (warpy_kernels/attn/fwd_base.py:337-360).  Inputs that need it are pathological (one key more than 69
// nats above the start of the row).  The CTA that found such rows does it at its end, when its shared memory is idle;
// the persistent kernel marks the block and goes through its marked blocks when it has nothing else left to do.  Where
// no row needs it, it costs one barrier with a vote; as a kernel of its own behind every forward, which looked for
// flagged blocks, it cost a launch: 2 us per call on the GPU and 3 us on the host.
//
// Bound by the latency of a step of four keys (3600 cycles; 32 loads from shared memory, 256 multiply-adds): eight threads
// share two rows, each with every eighth quad of the head dimension of Q and O in registers, and read K and V, fp32 in
// shared memory, 64 keys at a time, once for both rows.  128 rows x 16384 keys, d 128: FP8 in the persistent kernel 8.4 ms,
// BF16 (half as many threads) 15.5; four threads to a row took 10.6 and 18.9, steps of two keys 8.6 and 16.9.
#pragma once
#include <type_traits>

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

constexpr int EXACT_KEYS = 64;                          // keys in shared memory at a time
constexpr int EXACT_PITCH = 128 * 4;                    // bytes between their rows
constexpr int EXACT_SMEM = 2 * EXACT_KEYS * EXACT_PITCH;

// Four elements as fp32: 4 bytes of e4m3 (w.x) or 8 of bf16.
template <bool BF16>
__device__ __forceinline__ float4 exact_unpack(uint2 w) {
  float4 x;
  if (BF16) {
    x.x = __uint_as_float(w.x << 16), x.y = __uint_as_float(w.x & 0xffff0000u);
    x.z = __uint_as_float(w.y << 16), x.w = __uint_as_float(w.y & 0xffff0000u);
  } else {
    unpack_e4m3x2(static_cast<uint16_t>(w.x & 0xffffu), x.x, x.y);
    unpack_e4m3x2(static_cast<uint16_t>(w.x >> 16), x.z, x.w);
  }
  return x;
}
__device__ __forceinline__ float4 exact_lds(uint32_t addr) {
  float4 x;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w)
               : "r"(addr));
  return x;
}

// Computes rows of query block `m_blk` again and stores them.  Called by THREADS threads (whole warps, `tid` counts
// them) that use named barrier 2 and EXACT_SMEM bytes of shared memory at `smem`.  `far`: shared address of one word
// per row of the block that says whether the row needs it, or 0: all of them do.
template <bool BF16, int THREADS, class Params>
__device__ __noinline__ void exact_block(const Params& p, int b, int hq, int m_blk, float beta, float sv, uint32_t smem,
                                         uint32_t far, int tid) {
  constexpr int SIZE = BF16 ? 2 : 1;
  constexpr int ROWS = THREADS / 4;  // rows at a time: eight threads share two
  constexpr int PIECE = 16 / SIZE;   // elements per 16-byte load of K or V
  const ExactInputs& e = p.exact;
  const int hkv = hq / (p.Hq / p.Hkv);
  const int nk = p.seqused_k ? max(0, min(p.Nk, p.seqused_k[b])) : p.Nk;
  const int shift = nk - p.Nq;  // key j is visible to query i iff j <= i + shift (causal)
  const int part = tid & 7, lane = tid & 31;
  const int quads = e.d / 32;  // of this thread: quad i holds elements [32 i + 4 part, + 4)
  const uint32_t k_smem = smem, v_smem = smem + EXACT_KEYS * EXACT_PITCH;
  const uint8_t* k_base = e.k + b * e.k_strides[0] + hkv * e.k_strides[1];
  const uint8_t* v_base = e.v + b * e.v_strides[0] + hkv * e.v_strides[1];
  auto barrier = [] { asm volatile("bar.sync 2, %0;" ::"n"(THREADS) : "memory"); };
  auto wanted = [&](int r) {
    uint32_t w;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w) : "r"(far + 4 * r) : "memory");
    return w != 0;
  };

#pragma unroll 1
  for (int r0 = 0; r0 < 128; r0 += ROWS) {
    if (far) {  // the same answer in every warp
      bool any = false;
      for (int r = lane; r < ROWS; r += 32) any |= wanted(r0 + r);
      if (!__any_sync(0xffffffffu, any)) continue;
    }
    int row[2], limit[2];  // limit: last visible key of the row, -1 if it is not wanted
    float q[2][16], o[2][16], m[2], l[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = r0 + (tid >> 3) + h * (ROWS / 2);
      row[h] = m_blk * 128 + r;
      limit[h] = row[h] >= p.Nq || (far && !wanted(r)) ? -1 : p.causal ? min(row[h] + shift, nk - 1) : nk - 1;
      m[h] = -INFINITY, l[h] = 0.f;
      const uint8_t* src = e.q + b * e.q_strides[0] + hq * e.q_strides[1] + min(row[h], p.Nq - 1) * e.q_strides[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint8_t* at = src + (32 * i + 4 * part) * SIZE;
        uint2 w = make_uint2(0, 0);
        if (i < quads) w = BF16 ? *reinterpret_cast<const uint2*>(at) : make_uint2(*reinterpret_cast<const uint32_t*>(at), 0);
        const float4 x = exact_unpack<BF16>(w);
        q[h][4 * i] = x.x, q[h][4 * i + 1] = x.y, q[h][4 * i + 2] = x.z, q[h][4 * i + 3] = x.w;
        o[h][4 * i] = o[h][4 * i + 1] = o[h][4 * i + 2] = o[h][4 * i + 3] = 0.f;
      }
    }
    const int n_keys = p.causal ? max(0, min(nk, min(m_blk * 128 + r0 + ROWS, p.Nq) + shift)) : nk;  // of any row
#pragma unroll 1
    for (int c0 = 0; c0 < n_keys; c0 += EXACT_KEYS) {
      barrier();  // the keys before have been used
      const int pieces = e.d / PIECE;
      for (int i = tid; i < 2 * EXACT_KEYS * pieces; i += THREADS) {
        const bool is_v = i >= EXACT_KEYS * pieces;
        const int j = i % (EXACT_KEYS * pieces), key = j / pieces, col = j % pieces * PIECE;
        uint4 w = make_uint4(0, 0, 0, 0);  // keys past the last one: zeros
        if (c0 + key < nk)
          w = *reinterpret_cast<const uint4*>((is_v ? v_base : k_base) +
                                              (c0 + key) * (is_v ? e.v_strides[2] : e.k_strides[2]) + col * SIZE);
        const uint32_t dst = (is_v ? v_smem : k_smem) + key * EXACT_PITCH + col * 4;
        const uint2 fours[4] = {make_uint2(w.x, w.y), BF16 ? make_uint2(w.z, w.w) : make_uint2(w.y, 0), make_uint2(w.z, 0),
                                make_uint2(w.w, 0)};
#pragma unroll
        for (int c = 0; c < PIECE / 4; ++c) {
          const float4 x = exact_unpack<BF16>(fours[c]);
          asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 16 * c), "f"(x.x), "f"(x.y), "f"(x.z),
                       "f"(x.w)
                       : "memory");
        }
      }
      barrier();
#pragma unroll 1
      for (int j = 0; j < min(EXACT_KEYS, n_keys - c0); j += 4) {  // rows past n_keys are staged or zero, and masked
        float s[2][4] = {};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (i >= quads) break;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float4 x = exact_lds(k_smem + (j + u) * EXACT_PITCH + 128 * i + 16 * part);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              s[h][u] = fmaf(q[h][4 * i], x.x, s[h][u]), s[h][u] = fmaf(q[h][4 * i + 1], x.y, s[h][u]);
              s[h][u] = fmaf(q[h][4 * i + 2], x.z, s[h][u]), s[h][u] = fmaf(q[h][4 * i + 3], x.w, s[h][u]);
            }
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float top = -INFINITY;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
#pragma unroll
            for (int x = 1; x < 8; x *= 2) s[h][u] += __shfl_xor_sync(0xffffffffu, s[h][u], x);
            s[h][u] *= beta;
            if (c0 + j + u <= limit[h]) top = fmaxf(top, s[h][u]);
          }
          if (top > m[h]) {
            const float f = exp2f(m[h] - top);
            m[h] = top;
            l[h] *= f;
#pragma unroll
            for (int i = 0; i < 16; ++i) o[h][i] *= f;
          }
          const float ref = m[h] > -INFINITY ? m[h] : 0.f;  // the scores so far may all have overflowed to -inf
#pragma unroll
          for (int u = 0; u < 4; ++u) {  // a masked key has no part in the row, whatever its V holds
            s[h][u] = c0 + j + u <= limit[h] ? exp2f(s[h][u] - ref) : 0.f;
            l[h] += s[h][u];
          }
        }
        auto add = [&](auto masked) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (i >= quads) break;
              const float4 x = exact_lds(v_smem + (j + u) * EXACT_PITCH + 128 * i + 16 * part);
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const bool drop = decltype(masked)::value && c0 + j + u > limit[h];
                o[h][4 * i] = fmaf(s[h][u], drop ? 0.f : x.x, o[h][4 * i]);
                o[h][4 * i + 1] = fmaf(s[h][u], drop ? 0.f : x.y, o[h][4 * i + 1]);
                o[h][4 * i + 2] = fmaf(s[h][u], drop ? 0.f : x.z, o[h][4 * i + 2]);
                o[h][4 * i + 3] = fmaf(s[h][u], drop ? 0.f : x.w, o[h][4 * i + 3]);
              }
            }
          }
        };
        if (__any_sync(0xffffffffu, c0 + j + 3 > min(limit[0], limit[1])))
          add(std::true_type{});
        else
          add(std::false_type{});
        __syncwarp();
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (row[h] >= p.Nq || (far && !wanted(r0 + (tid >> 3) + h * (ROWS / 2)))) continue;
      const bool empty = !(l[h] > 0.f);
      const float inv = empty ? 0.f : sv / l[h];
      __nv_bfloat16* dst =
          p.out + b * p.out_stride_b + hq * p.out_stride_h + static_cast<int64_t>(row[h]) * p.out_stride_n + 4 * part;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i < quads)
          *reinterpret_cast<uint2*>(dst + 32 * i) = make_uint2(pack_bf16x2(o[h][4 * i] * inv, o[h][4 * i + 1] * inv),
                                                               pack_bf16x2(o[h][4 * i + 2] * inv, o[h][4 * i + 3] * inv));
      if (p.write_lse && part == 0) {
        const int64_t off = b * p.lse_stride_b + hq * p.lse_stride_h + row[h];
        const float lse = empty ? INFINITY : m[h] + log2f(l[h]);
        p.lse[off] = p.lse_natural ? lse * 0.6931471805599453f : lse;
        p.pmax[off] = empty ? 0.f : exp2f(m[h] - lse);
      }
    }
    __syncwarp();
  }
}

}  // namespace wk
