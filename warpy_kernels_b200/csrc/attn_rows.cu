// Attention forward for few query rows (decoding) and for small problems: FP8 (e4m3) and BF16, head dimension 64 and
// 128.
//
// The tensor-core kernels of attn_fwd_fp8.cu and attn_fwd_bf16.cu give every query head tiles of 128 rows.  With one
// new token per sequence 127 of them are padding, each query head of a group reads K and V again, and a block's keys
// are walked by one CTA alone.  Here the rows of all query heads that share a KV head are packed, 16 to a CTA, and the
// keys are split over the four warps of a CTA and over the CTAs of a cluster, which combine their partial results in
// distributed shared memory.  Decoding reads K and V once and is bound by that (16 sequences of 8192 keys, 64 / 8 heads,
// BF16: 115 us, 4.7 TB/s; FP8 from 1024 keys on is attn_decode.cu's); a small problem is bound by latency, which the
// split divides (FP8, 1 x 2 heads, 300 x 777, d 64: 7.2 us).
//
// Structure: every thread fetches its own operand fragments with cp.async into a ring that only it reads (no barrier
// in the loop), 16-byte pieces, so that four lanes cover 64 bytes of a K row and eight lanes a whole V row.  The head
// dimension is permuted to make that possible: in an MMA the index it sums over may be assigned freely as long as
// both operands agree, and so may the columns of V.  The MMAs are mma.sync (16 rows are less than the smallest
// tcgen05 tile, and the arithmetic is far from binding): Q.K^T as e4m3 m16n8k32 straight from the fetched bytes, P.V
// as f16 m16n8k16 with V converted to f16 (exact) on the way; BF16 inputs use bf16 m16n8k16 for both.
//
// Numerics: logits in base 2, online softmax in fp32 per row and warp.  P is rounded to f16 (bf16 for BF16 inputs)
// relative to 2^(m - 14), m a running maximum that moves only when a score exceeds it by more than 1, so that P stays
// below 2^15 and keeps its full precision down to 2^-28 of the row's largest probability.  The row sum adds the
// unrounded values.  The mask, lse, pmax and empty rows are those of the other forward kernels; scores of any range
// are handled (no recomputation).
#include <math.h>

#include "attn_rows.h"
#include "common.cuh"
#include "host_common.h"
#include "pair.cuh"

namespace wk {
namespace {

constexpr int R_WARPS = 4;
constexpr int R_THREADS = 32 * R_WARPS;
constexpr int R_ROWS = 16;
constexpr int R_RING_BYTES = 24 * 1024;  // per warp
constexpr int R_MAX_SPLIT = 8;
constexpr float R_P_SHIFT = 14.f;        // P is stored times 2^14 (FP8 inputs)

struct RowsParams {
  const uint8_t* q;
  const uint8_t* k;
  const uint8_t* v;
  __nv_bfloat16* out;
  float* lse;
  float* pmax;
  const float* q_descale;
  const float* k_descale;
  const float* v_descale;
  int64_t q_strides[3], k_strides[3], v_strides[3];  // bytes
  int64_t out_strides[3], lse_strides[2];            // elements
  int B, Hq, Hkv, Nq, Nk;
  int causal, write_lse, lse_natural;
  const int* seqused_k;
  float softmax_scale;
  int splits;
};

template <bool FP8, int DH>
struct RowsCfg {
  static constexpr int SIZE = FP8 ? 1 : 2;
  static constexpr int KEYS = FP8 ? 32 : 16;              // keys per step of a warp
  static constexpr int K_PIECES = DH * SIZE / 64;         // 16-byte pieces of a K row per lane (four lanes per row)
  static constexpr int V_PIECE = DH * SIZE / 8 >= 16 ? 16 : 8;  // bytes of a V row per lane and piece (eight lanes)
  static constexpr int V_PIECES = DH * SIZE / 8 / V_PIECE;
  static constexpr int V_ELEMS = V_PIECE / SIZE;
  static constexpr int N8 = KEYS / 8;
  static constexpr int K_BYTES = N8 * K_PIECES * 16 * 32;  // per step and warp
  static constexpr int V_BYTES = (KEYS / 4) * V_PIECES * V_PIECE * 32;
  static constexpr int STAGE_BYTES = K_BYTES + V_BYTES;
  static constexpr int MAX_STAGES = R_RING_BYTES / STAGE_BYTES;
  static constexpr int NT = DH / 8;      // column tiles of O
  static constexpr int O_PITCH = DH + 4;  // fp32 values between rows of a partial O in shared memory
  static constexpr int PART_FLOATS = R_ROWS * O_PITCH + 3 * R_ROWS;  // O, then m, l, largest score
};

__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, int bytes) {
  if (bytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}

#define WK_MMA16816(name, ab)                                                                                     \
  __device__ __forceinline__ void name(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {         \
    asm("mma.sync.aligned." ab " {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"                 \
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])                                                          \
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));                                          \
  }
WK_MMA16816(mma_sync_f16, "m16n8k16.row.col.f32.f16.f16.f32")
WK_MMA16816(mma_sync_bf16, "m16n8k16.row.col.f32.bf16.bf16.f32")
WK_MMA16816(mma_sync_e4m3, "m16n8k32.row.col.f32.e4m3.e4m3.f32")
#undef WK_MMA16816

__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// One CTA: 16 packed rows of one (batch, KV head), the keys of its split.
template <bool FP8, int DH>
__global__ void __launch_bounds__(R_THREADS, 2)
attn_rows_kernel(const __grid_constant__ RowsParams p, int stages) {
  using C = RowsCfg<FP8, DH>;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int g = lane / 4, t = lane % 4;  // row group and column pair of an MMA fragment
  const int split = blockIdx.x;          // rank in the cluster
  const int b = blockIdx.y / p.Hkv, hkv = blockIdx.y % p.Hkv;
  const int group = p.Hq / p.Hkv;
  const int rows = group * p.Nq;  // packed: row r is query r % Nq of the group's head r / Nq
  const int row0 = blockIdx.z * R_ROWS;
  pdl_launch_dependents();
  pdl_wait();

  const int nk = p.seqused_k ? max(0, min(p.Nk, p.seqused_k[b])) : p.Nk;
  const int shift = nk - p.Nq;  // key j is visible to query i iff j <= i + shift (causal)
  // the two rows of this thread and their last visible keys
  int limit[2];
  int first_limit = nk - 1, last_limit = -1;  // over the CTA's rows
  {
    int lo = p.Nq - 1, hi = 0;  // smallest and largest query index
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = row0 + g + 8 * h;
      limit[h] = r >= rows ? -1 : p.causal ? min(nk - 1, r % p.Nq + shift) : nk - 1;
    }
    const int last = min(row0 + R_ROWS, rows) - 1;
    if (last / p.Nq != row0 / p.Nq) {
      lo = 0, hi = p.Nq - 1;
    } else {
      lo = row0 % p.Nq, hi = last % p.Nq;
    }
    if (p.causal) {
      first_limit = min(nk - 1, lo + shift);
      last_limit = min(nk - 1, hi + shift);
    } else {
      last_limit = nk - 1;
    }
  }
  // steps of KEYS keys: this split's range, dealt out to the warps in turn
  const int steps = last_limit < 0 ? 0 : last_limit / C::KEYS + 1;
  const int s0 = static_cast<int>(static_cast<int64_t>(steps) * split / p.splits) + warp;
  const int s1 = static_cast<int>(static_cast<int64_t>(steps) * (split + 1) / p.splits);

  const uint8_t* k_base = p.k + b * p.k_strides[0] + hkv * p.k_strides[1] + t * 16;
  const uint8_t* v_base = p.v + b * p.v_strides[0] + hkv * p.v_strides[1] + g * C::V_PIECE;
  const uint32_t ring = smem_u32(smem_raw) + warp * stages * C::STAGE_BYTES;
  auto fetch = [&](int step, int stage) {
    const uint32_t ks = ring + stage * C::STAGE_BYTES + lane * 16;
    const uint32_t vs = ring + stage * C::STAGE_BYTES + C::K_BYTES + lane * C::V_PIECE;
    const int key0 = step * C::KEYS;
#pragma unroll
    for (int j = 0; j < C::N8; ++j) {  // keys beyond the last one are masked: any valid row will do
      const uint8_t* src = k_base + min(key0 + 8 * j + g, nk - 1) * p.k_strides[2];
#pragma unroll
      for (int h = 0; h < C::K_PIECES; ++h) cp_async(ks + (j * C::K_PIECES + h) * 512, src + 64 * h, 16);
    }
#pragma unroll
    for (int j = 0; j < C::KEYS / 4; ++j) {  // key pairs 2 t, 2 t + 1 of each group of eight
      const uint8_t* src = v_base + min(key0 + 8 * (j / 2) + 2 * t + (j & 1), nk - 1) * p.v_strides[2];
#pragma unroll
      for (int h = 0; h < C::V_PIECES; ++h)
        cp_async(vs + (j * C::V_PIECES + h) * (32 * C::V_PIECE), src + 8 * C::V_PIECE * h, C::V_PIECE);
    }
  };
  for (int i = 0; i < stages; ++i) {
    if (s0 + R_WARPS * i < s1) fetch(s0 + R_WARPS * i, i);
    cp_async_commit();
  }

  // Q fragments: the same bytes of each of the two rows as of a K row
  uint4 q[2][C::K_PIECES];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = min(row0 + g + 8 * h, rows - 1);
    const uint8_t* src = p.q + b * p.q_strides[0] + (hkv * group + r / p.Nq) * p.q_strides[1] +
                         (r % p.Nq) * p.q_strides[2] + t * 16;
#pragma unroll
    for (int j = 0; j < C::K_PIECES; ++j) q[h][j] = *reinterpret_cast<const uint4*>(src + 64 * j);
  }
  const int sc = b * p.Hkv + hkv;
  const float beta = p.softmax_scale * 1.4426950408889634f * (FP8 ? p.q_descale[sc] * p.k_descale[sc] : 1.f);
  constexpr float P_SHIFT = FP8 ? R_P_SHIFT : 0.f;

  float o[C::NT][4];
#pragma unroll
  for (int j = 0; j < C::NT; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[j][i] = 0.f;
  float m[2] = {-INFINITY, -INFINITY}, top[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};

  int stage = 0;
  for (int step = s0; step < s1; step += R_WARPS) {
    if (stages == 1)
      cp_async_wait<0>();
    else if (stages == 2)
      cp_async_wait<1>();
    else if (stages == 3)
      cp_async_wait<2>();
    else
      cp_async_wait<5>();
    const uint32_t ks = ring + stage * C::STAGE_BYTES + lane * 16;
    const uint32_t vs = ring + stage * C::STAGE_BYTES + C::K_BYTES + lane * C::V_PIECE;

    // ---- scores: s[j][0..1] row g, keys 8 j + 2 t and + 1; s[j][2..3] row g + 8
    float s[C::N8][4];
#pragma unroll
    for (int j = 0; j < C::N8; ++j) {
      s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#pragma unroll
      for (int h = 0; h < C::K_PIECES; ++h) {
        const uint4 kk = lds128(ks + (j * C::K_PIECES + h) * 512);
        const uint32_t a0[4] = {q[0][h].x, q[1][h].x, q[0][h].y, q[1][h].y};
        const uint32_t a1[4] = {q[0][h].z, q[1][h].z, q[0][h].w, q[1][h].w};
        if (FP8) {
          mma_sync_e4m3(s[j], a0, kk.x, kk.y);
          mma_sync_e4m3(s[j], a1, kk.z, kk.w);
        } else {
          mma_sync_bf16(s[j], a0, kk.x, kk.y);
          mma_sync_bf16(s[j], a1, kk.z, kk.w);
        }
      }
    }
    const int key0 = step * C::KEYS;
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < C::N8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[j][i] *= beta;
    if (key0 + C::KEYS - 1 > first_limit) {
#pragma unroll
      for (int j = 0; j < C::N8; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (key0 + 8 * j + 2 * t + (i & 1) > limit[i >> 1]) s[j][i] = -INFINITY;
    }
#pragma unroll
    for (int j = 0; j < C::N8; ++j) {
      mx[0] = max3(mx[0], s[j][0], s[j][1]);
      mx[1] = max3(mx[1], s[j][2], s[j][3]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
      mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
      top[h] = fmaxf(top[h], mx[h]);
    }
    // the reference moves when the step rises more than 1 above it (and from -inf)
    const bool move0 = mx[0] > m[0] + 1.f, move1 = mx[1] > m[1] + 1.f;
    if (__any_sync(0xffffffffu, move0 || move1)) {
      const float n0 = move0 ? mx[0] : m[0], n1 = move1 ? mx[1] : m[1];
      const float f0 = move0 ? ex2_approx(m[0] - n0) : 1.f, f1 = move1 ? ex2_approx(m[1] - n1) : 1.f;
      m[0] = n0, m[1] = n1;
      l[0] *= f0, l[1] *= f1;
#pragma unroll
      for (int j = 0; j < C::NT; ++j) {
        o[j][0] *= f0, o[j][1] *= f0;
        o[j][2] *= f1, o[j][3] *= f1;
      }
    }
    const float bias0 = m[0] > -INFINITY ? P_SHIFT - m[0] : 0.f, bias1 = m[1] > -INFINITY ? P_SHIFT - m[1] : 0.f;
#pragma unroll
    for (int j = 0; j < C::N8; ++j) {
      s[j][0] = ex2_approx(s[j][0] + bias0), s[j][1] = ex2_approx(s[j][1] + bias0);
      s[j][2] = ex2_approx(s[j][2] + bias1), s[j][3] = ex2_approx(s[j][3] + bias1);
      l[0] += s[j][0] + s[j][1];
      l[1] += s[j][2] + s[j][3];
    }

    // ---- O += P.V, 16 keys at a time
#pragma unroll
    for (int c = 0; c < C::KEYS / 16; ++c) {
      uint32_t a[4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float(&x)[4] = s[2 * c + h];
        a[2 * h] = FP8 ? pack_f16x2(x[0], x[1]) : pack_bf16x2(x[0], x[1]);
        a[2 * h + 1] = FP8 ? pack_f16x2(x[2], x[3]) : pack_bf16x2(x[2], x[3]);
      }
#pragma unroll
      for (int h = 0; h < C::V_PIECES; ++h) {
        uint32_t w[4][4];  // [key 2t, 2t + 1, 2t + 8, 2t + 9][word]
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t addr = vs + ((4 * c + i) * C::V_PIECES + h) * (32 * C::V_PIECE);
          if (C::V_PIECE == 16) {
            const uint4 x = lds128(addr);
            w[i][0] = x.x, w[i][1] = x.y, w[i][2] = x.z, w[i][3] = x.w;
          } else {
            const uint2 x = lds64(addr);
            w[i][0] = x.x, w[i][1] = x.y;
          }
        }
#pragma unroll
        for (int x = 0; x < C::V_PIECE / 4; ++x) {
          if (FP8) {
            // bytes of key pairs side by side, then e4m3 -> f16: two columns per word, four columns per x
            const uint32_t lo0 = __byte_perm(w[0][x], w[1][x], 0x5140), hi0 = __byte_perm(w[0][x], w[1][x], 0x7362);
            const uint32_t lo1 = __byte_perm(w[2][x], w[3][x], 0x5140), hi1 = __byte_perm(w[2][x], w[3][x], 0x7362);
            float(*oo)[4] = o + h * C::V_ELEMS + 4 * x;
            mma_sync_f16(oo[0], a, e4m3x2_to_f16x2(static_cast<uint16_t>(lo0)), e4m3x2_to_f16x2(static_cast<uint16_t>(lo1)));
            mma_sync_f16(oo[1], a, e4m3x2_to_f16x2(static_cast<uint16_t>(lo0 >> 16)), e4m3x2_to_f16x2(static_cast<uint16_t>(lo1 >> 16)));
            mma_sync_f16(oo[2], a, e4m3x2_to_f16x2(static_cast<uint16_t>(hi0)), e4m3x2_to_f16x2(static_cast<uint16_t>(hi1)));
            mma_sync_f16(oo[3], a, e4m3x2_to_f16x2(static_cast<uint16_t>(hi0 >> 16)), e4m3x2_to_f16x2(static_cast<uint16_t>(hi1 >> 16)));
          } else {
            float(*oo)[4] = o + h * C::V_ELEMS + 2 * x;
            mma_sync_bf16(oo[0], a, __byte_perm(w[0][x], w[1][x], 0x5410), __byte_perm(w[2][x], w[3][x], 0x5410));
            mma_sync_bf16(oo[1], a, __byte_perm(w[0][x], w[1][x], 0x7632), __byte_perm(w[2][x], w[3][x], 0x7632));
          }
        }
      }
    }
    // the stage's own reads are done (their values have been used): refill it
    const int next = step + R_WARPS * stages;
    if (next < s1) fetch(next, stage);
    cp_async_commit();
    if (++stage == stages) stage = 0;
  }
  cp_async_wait<0>();
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // the four lanes of a row have summed different keys
    l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
    l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
  }

  // ---- combine: the warps of this CTA, then the CTAs of the cluster ---------------------------------------------
  __syncthreads();  // the rings are free
  float* part = reinterpret_cast<float*>(smem_raw) + warp * C::PART_FLOATS;
#pragma unroll
  for (int j = 0; j < C::NT; ++j) {
    // column tile j holds element j % V_ELEMS of piece j / V_ELEMS of the eight lanes that share a V row
    const int col = (j / C::V_ELEMS) * (8 * C::V_ELEMS) + 2 * t * C::V_ELEMS + j % C::V_ELEMS;
    part[g * C::O_PITCH + col] = o[j][0];
    part[g * C::O_PITCH + col + C::V_ELEMS] = o[j][1];
    part[(g + 8) * C::O_PITCH + col] = o[j][2];
    part[(g + 8) * C::O_PITCH + col + C::V_ELEMS] = o[j][3];
  }
  if (t == 0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      part[R_ROWS * C::O_PITCH + g + 8 * h] = m[h];
      part[R_ROWS * C::O_PITCH + R_ROWS + g + 8 * h] = l[h];
      part[R_ROWS * C::O_PITCH + 2 * R_ROWS + g + 8 * h] = top[h];
    }
  }
  __syncthreads();
  // Each CTA first merges its warps (local shared memory, a result behind theirs), then finishes the rows congruent to
  // its rank from one partial result per CTA: all remote loads of a thread are independent of one another.
  constexpr int QUADS = DH / 4;
  float* merged = reinterpret_cast<float*>(smem_raw) + R_WARPS * C::PART_FLOATS;
  constexpr int M_OFF = R_ROWS * C::O_PITCH, L_OFF = M_OFF + R_ROWS, T_OFF = L_OFF + R_ROWS;
  for (int i = threadIdx.x; i < R_ROWS * QUADS; i += R_THREADS) {
    const int r = i / QUADS, col = (i % QUADS) * 4;
    const float* parts = reinterpret_cast<const float*>(smem_raw);
    float mm = -INFINITY, m_true = -INFINITY, sum = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < R_WARPS; ++w) mm = fmaxf(mm, parts[w * C::PART_FLOATS + M_OFF + r]);
#pragma unroll
    for (int w = 0; w < R_WARPS; ++w) {
      const float* x = parts + w * C::PART_FLOATS;
      const float f = x[M_OFF + r] > -INFINITY ? exp2f(x[M_OFF + r] - mm) : 0.f;
      const float4 c = *reinterpret_cast<const float4*>(x + r * C::O_PITCH + col);
      acc.x = fmaf(c.x, f, acc.x), acc.y = fmaf(c.y, f, acc.y), acc.z = fmaf(c.z, f, acc.z), acc.w = fmaf(c.w, f, acc.w);
      sum = fmaf(x[L_OFF + r], f, sum);
      m_true = fmaxf(m_true, x[T_OFF + r]);
    }
    *reinterpret_cast<float4*>(merged + r * C::O_PITCH + col) = acc;
    if (col == 0) merged[M_OFF + r] = mm, merged[L_OFF + r] = sum, merged[T_OFF + r] = m_true;
  }
  __syncwarp();
  if (p.splits > 1)
    cluster_sync();
  else
    __syncthreads();
  for (int i = threadIdx.x; i < R_ROWS * QUADS; i += R_THREADS) {
    const int r = (i / QUADS) * p.splits + split, col = (i % QUADS) * 4;
    if (r >= R_ROWS || row0 + r >= rows) break;
    float mx[R_MAX_SPLIT], lx[R_MAX_SPLIT], tx[R_MAX_SPLIT], ox[R_MAX_SPLIT][4];
#pragma unroll
    for (int x = 0; x < R_MAX_SPLIT; ++x) {
      mx[x] = tx[x] = -INFINITY;
      lx[x] = ox[x][0] = ox[x][1] = ox[x][2] = ox[x][3] = 0.f;
      if (x < p.splits) {
        const uint32_t base = p.splits > 1 ? mapa(smem_u32(merged), x) : smem_u32(merged);
        auto load = [&](int offset) {
          float y;
          asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(y) : "r"(base + offset * 4));
          return y;
        };
        mx[x] = load(M_OFF + r), lx[x] = load(L_OFF + r), tx[x] = load(T_OFF + r);
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(ox[x][0]), "=f"(ox[x][1]), "=f"(ox[x][2]), "=f"(ox[x][3])
                     : "r"(base + (r * C::O_PITCH + col) * 4));
      }
    }
    float mm = -INFINITY, m_true = -INFINITY, sum = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int x = 0; x < R_MAX_SPLIT; ++x) {
      mm = fmaxf(mm, mx[x]);
      m_true = fmaxf(m_true, tx[x]);
    }
#pragma unroll
    for (int x = 0; x < R_MAX_SPLIT; ++x) {
      const float f = mx[x] > -INFINITY ? exp2f(mx[x] - mm) : 0.f;
      sum = fmaf(lx[x], f, sum);
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[c] = fmaf(ox[x][c], f, acc[c]);
    }
    const bool empty = !(sum > 0.f);
    const float inv = empty ? 0.f : (FP8 ? p.v_descale[sc] : 1.f) / sum;
    const int head = hkv * group + (row0 + r) / p.Nq, query = (row0 + r) % p.Nq;
    uint2 w;
    w.x = pack_bf16x2(acc[0] * inv, acc[1] * inv);
    w.y = pack_bf16x2(acc[2] * inv, acc[3] * inv);
    *reinterpret_cast<uint2*>(p.out + b * p.out_strides[0] + head * p.out_strides[1] + query * p.out_strides[2] + col) = w;
    if (p.write_lse && col == 0) {
      const int64_t off = b * p.lse_strides[0] + head * p.lse_strides[1] + query;
      const float lse = empty ? INFINITY : mm - P_SHIFT + log2f(sum);
      p.lse[off] = p.lse_natural ? lse * 0.6931471805599453f : lse;
      p.pmax[off] = empty ? 0.f : exp2f(m_true - lse);
    }
  }
  __syncwarp();  // lanes leave the loop at different rows; the barrier wants the warp together
  if (p.splits > 1) cluster_sync();  // nobody leaves while its partial results may still be read
}

}  // namespace

namespace {

constexpr int R_DECODE_KEYS = 1024;  // from here on FP8 decoding goes to attn_decode.cu
// Packed rows up to which the split is chosen to fill the GPU and FP8 goes to attn_decode.cu: two CTAs' worth.  Larger
// problems with more rows keep to the 128-row tiles.  That is right for up to two query heads per KV head (33 to 64 rows,
// from 512 keys on: tiles 0.61 of the time here for FP8, 0.44 for BF16, medians of 117 and 128 problems) and gives time
// away where many heads share one: 1.5 and 1.0 times the time here for groups of 4 to 8, 3.8 and 2.3 for groups of 16.
constexpr int R_DECODE_ROWS = 32;

int rows_splits(const wk_attn_fwd_args* a, int sms) {
  const int64_t rows = static_cast<int64_t>(a->Hq / a->Hkv) * a->Nq;
  const int64_t units = static_cast<int64_t>(a->B) * a->Hkv * ((rows + R_ROWS - 1) / R_ROWS);
  if (rows > R_DECODE_ROWS) {
    // A small problem: from the rows alone, so that a batch item attends to its seqused_k keys in the same order as a
    // call on the truncated tensors does.
    const int64_t per_item = static_cast<int64_t>(a->Hkv) * ((rows + R_ROWS - 1) / R_ROWS);
    return per_item <= 40 ? 4 : per_item <= sms ? 2 : 1;
  }
  // two CTAs of four warps per SM; at least 128 keys for a CTA
  int s = 1;
  while (s < R_MAX_SPLIT && units * s * 2 <= 2 * sms && a->Nk >= 256 * s) s *= 2;
  return s;
}

template <bool FP8, int DH>
int launch_rows(RowsParams& p, cudaStream_t stream) {
  using C = RowsCfg<FP8, DH>;
  const void* fn = reinterpret_cast<const void*>(attn_rows_kernel<FP8, DH>);
  // as many stages as a warp has steps, up to what the ring holds (1, 2, 3 or 6: the waits are compile-time)
  const int steps = (p.Nk + C::KEYS - 1) / C::KEYS;
  const int per_warp = (steps + R_WARPS * p.splits - 1) / (R_WARPS * p.splits);
  int stages = per_warp < 3 ? per_warp : per_warp < 6 ? 3 : C::MAX_STAGES;
  if (stages > C::MAX_STAGES) stages = C::MAX_STAGES;
  const int ring = R_WARPS * stages * C::STAGE_BYTES, parts = (R_WARPS + 1) * C::PART_FLOATS * 4;
  const int smem = ring > parts ? ring : parts;
  const int most = R_WARPS * R_RING_BYTES > parts ? R_WARPS * R_RING_BYTES : parts;
  if (allow_smem(fn, most)) return WK_E_CUDA;
  const int rows = p.Hq / p.Hkv * p.Nq;
  return launch_pdl(fn, dim3(p.splits, p.B * p.Hkv, (rows + R_ROWS - 1) / R_ROWS), R_THREADS, smem, stream, p.splits,
                    {&p, &stages});
}

}  // namespace

namespace {

bool few_rows(int64_t B, int64_t Hq, int64_t Hkv, int64_t Nq, int64_t Nk, int d) {
  const int64_t rows = Hq / Hkv * Nq, kv = B * Hkv;
  if (kv > 65535 || rows > 16 * 65535) return false;
  return rows <= R_DECODE_ROWS || kv * rows * Nk <= (d == 64 ? 1 << 22 : 1 << 20);
}

bool decodes(const wk_attn_fwd_args* a, bool bf16) {
  return !bf16 && a->Nk >= R_DECODE_KEYS && static_cast<int64_t>(a->Hq / a->Hkv) * a->Nq <= R_DECODE_ROWS;
}

}  // namespace

bool attn_rows_applies(const wk_attn_fwd_args* a) {
  // an explicit choice between the tensor-core kernels, or a caller who wants their range reported, gets those
  if (a->ctas_per_sm != 0 || !a->workspace) return false;
  return few_rows(a->B, a->Hq, a->Hkv, a->Nq, a->Nk, a->d);
}

// Every kernel is taken to cost a start, and per CTA a fixed part and a part per step over the keys; two CTAs of an SM
// take `both` times as long as one alone, and a grid beyond two CTAs per SM as many times longer as it is larger.  The
// microseconds are fits to 8192 problems inside few_rows()'s limits (1 to 128 sequences, 1 to 32 KV heads, groups of 1 to
// 16, 1 to 2048 queries, 16 to 16384 keys), half of them within 5 to 10 % (decoding 17 %).  Which side is ahead is mostly a
// matter of idle SMs and of padding: FP8, d 128, one query for 16 sequences of 8192 keys, 64 / 8 heads 41 us here and 379
// there, 1 x 2 heads, 300 x 777, d 64 7.2 and 11.6; but 8 x 8 heads, 128 x 128 30.9 and 6.1, 128 x 32 heads, 32 x 1024
// 534 and 229 (BF16 841 and 344).  By these figures 3 % of the problems go where they take more than 3 % longer than on
// the other side, at most 1.5 times; by the row limits alone it was 34 % of the BF16 and 46 % of the FP8 problems up to
// 512 keys, up to 18 times.  Beyond R_DECODE_ROWS the line is drawn as for 256 keys at least, with 0.3 us in favour of this
// side, so that a batch item mostly attends to its seqused_k keys in the kernel that a call on the truncated tensors gets
// (whose results are then the same to the bit); that costs 1 us at most, to one problem in eight.
bool attn_rows_ahead(const wk_attn_fwd_args* a, bool bf16, int sms) {
  struct Cost {
    double start, fixed, step, both;
  };
  static const Cost kTiles[2][2] = {{{2.3, 2.0, 0.66, 1.7}, {2.5, 2.2, 0.67, 1.7}},   // [bf16][d 128], 64 keys a step
                                    {{2.5, 1.9, 0.55, 1.7}, {2.7, 2.1, 0.68, 1.7}}};
  static const Cost kRows[2][2] = {{{2.6, 1.4, 0.81, 1.55}, {2.2, 3.1, 1.41, 1.65}},
                                   {{3.0, 1.0, 0.70, 1.6}, {2.1, 2.7, 1.19, 1.7}}};
  static const Cost kDecode[2] = {{2.4, 3.3, 0.87, 1.65}, {2.15, 4.0, 0.93, 1.7}};
  auto time = [&](const Cost& c, double steps, double ctas) {
    const double full = ctas / (2.0 * sms);
    const double crowd = full <= 0.5 ? 1.0 : full <= 1.0 ? 1.0 + (c.both - 1.0) * (2.0 * full - 1.0) : c.both * full;
    return c.start + (c.fixed + c.step * steps) * crowd;
  };
  const bool wide = a->d == 128;
  const int64_t rows = static_cast<int64_t>(a->Hq / a->Hkv) * a->Nq, kv = static_cast<int64_t>(a->B) * a->Hkv;
  const int64_t nq = a->Nq, nk = rows > R_DECODE_ROWS && a->Nk < 256 ? 256 : a->Nk;
  double tiles = static_cast<double>((nk + 63) / 64);
  if (a->causal) {  // of a block on average: from those of the first block that sees a key to all of them
    const int64_t first = (nq < 128 ? nq : 128) + nk - nq;
    tiles = (tiles + (first > 0 ? (first + 63) / 64 : 1)) / 2 * (nk < nq ? static_cast<double>(nk) / nq : 1.0);
  }
  const double blocks = static_cast<double>(a->B) * a->Hq * ((nq + 127) / 128);
  const double there = time(kTiles[bf16][wide], tiles, blocks) + (rows > R_DECODE_ROWS ? 0.3 : 0.0);
  if (decodes(a, bf16)) {
    const int64_t units = kv * (rows <= 8 ? 1 : (rows + 15) / 16);
    const int s = attn_decode_splits(a, units, sms);
    return time(kDecode[wide], static_cast<double>(((nk + 127) / 128 + s - 1) / s), static_cast<double>(units) * s) <= there;
  }
  const int s = rows_splits(a, sms), keys = bf16 ? 16 : 32, shares = R_WARPS * s;
  const int64_t ctas = kv * ((rows + R_ROWS - 1) / R_ROWS) * s;
  return time(kRows[bf16][wide], static_cast<double>(((nk + keys - 1) / keys + shares - 1) / shares),
              static_cast<double>(ctas)) <= there;
}

int launch_attn_rows(const wk_attn_fwd_args* a, bool bf16, cudaStream_t stream) {
  if (decodes(a, bf16)) return launch_attn_decode(a, stream);
  const int sms = sm_count();
  if (sms <= 0) return WK_E_CUDA;
  RowsParams p = {};
  p.q = static_cast<const uint8_t*>(a->q);
  p.k = static_cast<const uint8_t*>(a->k);
  p.v = static_cast<const uint8_t*>(a->v);
  p.out = static_cast<__nv_bfloat16*>(a->out);
  p.lse = a->lse;
  p.pmax = a->pmax;
  p.q_descale = a->q_descale;
  p.k_descale = a->k_descale;
  p.v_descale = a->v_descale;
  const int64_t size = bf16 ? 2 : 1;
  for (int i = 0; i < 3; ++i) {
    p.q_strides[i] = a->q_strides[i] * size;
    p.k_strides[i] = a->k_strides[i] * size;
    p.v_strides[i] = a->v_strides[i] * size;
    p.out_strides[i] = a->out_strides[i];
  }
  p.lse_strides[0] = a->lse_strides[0];
  p.lse_strides[1] = a->lse_strides[1];
  p.B = a->B, p.Hq = a->Hq, p.Hkv = a->Hkv, p.Nq = a->Nq, p.Nk = a->Nk;
  p.causal = a->causal, p.write_lse = a->write_lse, p.lse_natural = a->lse_natural;
  p.seqused_k = a->seqused_k;
  p.softmax_scale = a->softmax_scale;
  p.splits = rows_splits(a, sms);
  if (bf16) return a->d == 64 ? launch_rows<false, 64>(p, stream) : launch_rows<false, 128>(p, stream);
  return a->d == 64 ? launch_rows<true, 64>(p, stream) : launch_rows<true, 128>(p, stream);
}

}  // namespace wk

extern "C" int wk_attn_fwd_few_rows(int B, int Hq, int Hkv, int Nq, int Nk, int d) {
  if (B <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv || Nq <= 0 || Nk <= 0 || (d != 64 && d != 128)) return WK_E_ARG;
  return wk::few_rows(B, Hq, Hkv, Nq, Nk, d);
}

// One int per block of 128 queries, rounded up to 16 bytes.
extern "C" int64_t wk_attn_fwd_workspace_bytes(int B, int Hq, int Nq) {
  if (B <= 0 || Hq <= 0 || Nq <= 0) return 0;
  const int64_t blocks = static_cast<int64_t>(B) * Hq * ((Nq + 127) / 128);
  return (blocks * 4 + 15) / 16 * 16;
}
