// FP8 attention forward for decoding: few query rows against a long cache of keys, on tcgen05.
//
// The rows of all query heads of a KV head are packed, NR = 8 or 16 to a CTA, and play the N side of the products, so
// that no tensor-core work and no exponential is spent on padding rows:
//   S^T[128 keys, NR]  = K . Q^T      (kind::f8f6f4, A = the K tile, B = the packed rows of Q)
//   O^T[d, 2 NR]      += V^T . P^T    (kind::mxf8f6f4, A = the V tile read MN-major, B = P from shared memory)
// One thread of the four softmax warps owns one key of the tile; a warp's 32 keys are exactly one scale block of P, so
// the block maximum of a row is one warp-wide reduction.  P is carried as two e4m3 terms (value and 2^-4 times the
// residual, rows NR .. 2 NR of the same operand), 7 significant bits for any number of keys.  Keys are split over the
// CTAs of a cluster, which combine their partial results in distributed shared memory.
//
// Bound by reading K and V once.  Per 128 keys (32 KiB, 1440 cycles of an SM's share of the memory bandwidth) a
// softmax warp issues about 250 instructions.  The mma.sync form of the same split (attn_rows.cu), which converts K and
// V to f16 in registers, issues 630 per 32 keys and warp and is bound by their latency.
//
// 224 threads, two CTAs per SM: warp 0 TMA producer (three stages of 128 keys), warps 1 and 6 issue the two products,
// warps 2-5 softmax.
//
// Numerics are those of attn_fwd_fp8.cu: P8 = e4m3(2^(s.beta - e_blk + 8)) with e_blk the exponent of the 32-key block,
// O in units of the row reference m_ref, which is the row maximum of the split's first tile.  A split that meets a score
// more than 2^100 above it goes through its keys a second time with the maximum it then knows.
#include <math.h>

#include "attn_rows.h"
#include "common.cuh"
#include "host_common.h"
#include "pair.cuh"

namespace wk {
namespace {

constexpr int E_KEYS = 128;  // keys per tile
constexpr int E_STAGES = 3;
constexpr int E_TILE_BYTES = E_KEYS * 128;  // rows of 128 bytes (head dimension 64: upper half zero, filled in by TMA)
constexpr int E_THREADS = 224;
constexpr int E_SOFTMAX = 128;
constexpr int E_P_OFFSET = 8;
constexpr float E_MAX_EXP = 100.f;
constexpr int E_TMEM_COLS = 128;
constexpr int E_S_COL = 0;     // two buffers of 32 columns
constexpr int E_O_COL = 64;    // up to 32 columns
constexpr int E_SFA_COL = 96;  // unit scales of V
constexpr int E_SFB_COL = 100; // scales of P, two buffers of 4 columns
constexpr int E_MAX_SPLIT = 8;

struct DecodeParams {
  const uint8_t* q;
  __nv_bfloat16* out;
  float* lse;
  float* pmax;
  const float* q_descale;
  const float* k_descale;
  const float* v_descale;
  int64_t q_strides[3];                    // bytes
  int64_t out_strides[3], lse_strides[2];  // elements
  int B, Hq, Hkv, Nq, Nk, d;
  int causal, write_lse, lse_natural;
  const int* seqused_k;
  float softmax_scale;
  int splits;
  int* status;
};

template <int NR>
struct DecodeCfg {
  static constexpr int N = 2 * NR;                   // rows of P: the values, then the residuals
  static constexpr int QN = NR < 16 ? 16 : NR;       // rows of Q (the smallest N of an M = 128 product is 16)
  static constexpr int Q_BYTES = QN * 128;
  static constexpr int P_BYTES = N * 128;            // one of two buffers
  static constexpr int SF_BYTES = 512;               // likewise
  static constexpr int PITCH = 132;                  // fp32 values between rows of the partial O
  static constexpr int PART_BYTES = NR * PITCH * 4;  // shares the ring's memory
  static constexpr int XCH_BYTES = (4 + 3) * 16 * 4 + 64;  // maxima of the warps; m, l, top of the CTA
  static constexpr int SMEM = E_STAGES * 2 * E_TILE_BYTES + 2 * P_BYTES + Q_BYTES + 2 * SF_BYTES + 4 * 16 * 4 * 2 +
                              XCH_BYTES + 1024 + 256;
};

__device__ __forceinline__ float warp_max(float x) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
  return r;
}
template <int N>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&v)[N]);
template <>
__device__ __forceinline__ void tmem_ld_cols<8>(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld_cols<16>(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void sts_u8(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u8 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ float lds_f32(uint32_t addr) {
  float x;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(addr) : "memory");
  return x;
}
__device__ __forceinline__ void sts_f32(uint32_t addr, float x) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(x) : "memory");
}
__device__ __forceinline__ void softmax_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

template <int NR>
__global__ void __launch_bounds__(E_THREADS, 2)
attn_decode_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                   const __grid_constant__ DecodeParams p) {
  using C = DecodeCfg<NR>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t p_smem = smem_base + E_STAGES * 2 * E_TILE_BYTES;  // 1024-byte aligned like the tiles
  const uint32_t q_smem = p_smem + 2 * C::P_BYTES;
  const uint32_t sf_smem = q_smem + C::Q_BYTES;
  const uint32_t xch = sf_smem + 2 * C::SF_BYTES;  // [4 warps][16] values of two exchanges, then m, l, top of the CTA
  const uint32_t bar_base = xch + 4 * 16 * 4 * 2 + C::XCH_BYTES;
  auto kv_full = [&](int s) { return bar_base + 8u * s; };
  auto kv_empty = [&](int s) { return bar_base + 8u * (E_STAGES + s); };
  const uint32_t misc = bar_base + 8u * (2 * E_STAGES);
  auto s_full = [&](int b) { return misc + 8u * b; };
  auto s_free = [&](int b) { return misc + 8u * (2 + b); };
  auto p_full = [&](int b) { return misc + 8u * (4 + b); };
  auto p_free = [&](int b) { return misc + 8u * (6 + b); };
  const uint32_t o_full = misc + 8u * 8, q_full = misc + 8u * 9;
  const uint32_t tmem_slot = misc + 8u * 10, again_slot = tmem_slot + 4;

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int split = blockIdx.x;  // rank in the cluster
  const int b = blockIdx.y / p.Hkv, hkv = blockIdx.y % p.Hkv;
  const int group = p.Hq / p.Hkv;
  const int rows = group * p.Nq;  // packed: row r is query r % Nq of the group's head r / Nq
  const int row0 = blockIdx.z * NR;

  if (threadIdx.x == 0) {
    for (int s = 0; s < E_STAGES; ++s) {
      mbar_init(kv_full(s), 1);
      mbar_init(kv_empty(s), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(s_full(i), 1);
      mbar_init(s_free(i), E_SOFTMAX);
      mbar_init(p_full(i), E_SOFTMAX);
      mbar_init(p_free(i), 1);
    }
    mbar_init(o_full, 1);
    mbar_init(q_full, E_SOFTMAX);
    mbar_fence_init();
    prefetch_tmap(&tmap_k);
    prefetch_tmap(&tmap_v);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, E_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  pdl_launch_dependents();
  pdl_wait();

  const int nk = p.seqused_k ? max(0, min(p.Nk, p.seqused_k[b])) : p.Nk;
  const int shift = nk - p.Nq;  // key j is visible to query i iff j <= i + shift (causal)
  const int last_row = min(row0 + NR, rows) - 1;
  const int last_query = last_row / p.Nq != row0 / p.Nq ? p.Nq - 1 : last_row % p.Nq;
  const int last_key = p.causal ? min(nk - 1, last_query + shift) : nk - 1;
  const int all_tiles = last_key < 0 ? 0 : last_key / E_KEYS + 1;
  const int t0 = static_cast<int>(static_cast<int64_t>(all_tiles) * split / p.splits);
  const int n_tiles = static_cast<int>(static_cast<int64_t>(all_tiles) * (split + 1) / p.splits) - t0;

  // The loop runs once more if a score outgrew the row reference; every barrier goes on from where it is.
  int base = 0;  // tiles before this pass
  int passes = 0;
  auto another_pass = [&]() {  // asked by every thread after its pass: the softmax warps' answer
    __syncthreads();
    uint32_t again;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(again) : "r"(again_slot) : "memory");
    __syncthreads();
    base += n_tiles;
    ++passes;
    return again != 0 && passes < 2;
  };

  if (warp == 0) {
    do {
      if (lane == 0) {
        for (int j = base; j < base + n_tiles; ++j) {
          const int s = j % E_STAGES;
          if (!mbar_wait(kv_empty(s), ((j / E_STAGES) & 1) ^ 1, p.status, WK_ERR_TIMEOUT_EMPTY)) break;
          mbar_expect_tx(kv_full(s), 2 * E_TILE_BYTES);
          const uint32_t dst = smem_base + s * 2 * E_TILE_BYTES;
          tma_load_4d(dst, &tmap_k, kv_full(s), 0, (t0 + j - base) * E_KEYS, hkv, b);
          tma_load_4d(dst + E_TILE_BYTES, &tmap_v, kv_full(s), 0, (t0 + j - base) * E_KEYS, hkv, b);
        }
      }
      __syncwarp();
    } while (another_pass());
  } else if (warp == 1) {
    // ---- S^T = K.Q^T, as soon as a tile and a buffer are there
    const bool mine = elect_one();
    constexpr uint32_t idesc_qk = make_idesc(0, 0, 0, 0, E_KEYS, C::QN);
    const uint64_t q_desc = smem_desc_sw128(q_smem, 16, 1024);
    bool ok = mbar_wait_warp(q_full, 0, p.status, WK_ERR_TIMEOUT_LOAD);
    do {
      for (int j = base; ok && j < base + n_tiles; ++j) {
        const int s = j % E_STAGES, buf = j & 1;
        if (j >= 2) ok = mbar_wait_warp(s_free(buf), ((j >> 1) - 1) & 1, p.status, WK_ERR_TIMEOUT_P);
        ok = ok && mbar_wait_warp(kv_full(s), (j / E_STAGES) & 1, p.status, WK_ERR_TIMEOUT_LOAD);
        tc_fence_after();
        if (ok && mine) {
          const uint64_t k_desc = smem_desc_sw128(smem_base + s * 2 * E_TILE_BYTES, 16, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (32 * k < p.d) mma_f8_ss(tmem_base + E_S_COL + 32 * buf, k_desc + 2 * k, q_desc + 2 * k, idesc_qk, k != 0);
          tc_commit(s_full(buf));
        }
      }
      __syncwarp();
    } while (another_pass());
  } else if (warp == 6) {
    // ---- O^T += V^T.P^T.  By a warp of its own: one that also waits for the next tile's K before it gets here holds
    // the stage back and with it the next load.
    const bool mine = elect_one();
    bool ok = true;
    do {
      for (int j = base; ok && j < base + n_tiles; ++j) {
        const int s = j % E_STAGES, buf = j & 1;
        ok = mbar_wait_warp(p_full(buf), (j >> 1) & 1, p.status, WK_ERR_TIMEOUT_P);
        tc_fence_after();
        if (ok && mine) {
          tmem_cp_32x128b_warpx4(tmem_base + E_SFB_COL + 4 * buf, smem_desc_plain(sf_smem + buf * C::SF_BYTES, 16, 128));
          // V tile: 128 keys (the MMA's K) x 128 bytes of head dimension (its M): MN-major, 32 keys = 4096 bytes
          const uint64_t v_desc = smem_desc_sw128(smem_base + s * 2 * E_TILE_BYTES + E_TILE_BYTES, 16, 1024);
          const uint64_t p_desc = smem_desc_sw128(p_smem + buf * C::P_BYTES, 16, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mma_mxf8_ss(tmem_base + E_O_COL, v_desc + 256 * k, p_desc + 2 * k, make_idesc_mx_major(128, C::N, 0, k, 1, 0),
                        tmem_base + E_SFA_COL, tmem_base + E_SFB_COL + 4 * buf, (j != base) | (k != 0));
          tc_commit(kv_empty(s));
          tc_commit(p_free(buf));
          if (j == base + n_tiles - 1) tc_commit(o_full);
        }
      }
      __syncwarp();
    } while (another_pass());
  } else {
    const int quad = warp & 3;  // this warp's keys of a tile = its lanes of tensor memory = one scale block
    const int r_key = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    {
      // packed rows of Q to shared memory, swizzled like a TMA tile; unit scales for V
      for (int i = r_key; i < C::QN * 8; i += E_SOFTMAX) {
        const int r = i / 8, c = i % 8;
        uint4 w = make_uint4(0, 0, 0, 0);
        if (row0 + r < rows && r < NR && c * 16 < p.d)
          w = *reinterpret_cast<const uint4*>(p.q + b * p.q_strides[0] + (hkv * group + (row0 + r) / p.Nq) * p.q_strides[1] +
                                              ((row0 + r) % p.Nq) * p.q_strides[2] + c * 16);
        const uint32_t dst = q_smem + r * 128 + ((c ^ (r & 7)) << 4);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w)
                     : "memory");
      }
      tmem_st4(tmem_base + lane_addr + E_SFA_COL, 0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu);
      tc_wait_st();
      tc_fence_before();
      fence_proxy_async_smem();
      mbar_arrive(q_full);
    }
    const int sc = b * p.Hkv + hkv;
    const float beta = p.softmax_scale * p.q_descale[sc] * p.k_descale[sc] * 1.4426950408889634f;
    int limit[NR];  // last visible key of each row; one value unless the mask is causal
#pragma unroll
    for (int r = 0; r < NR; ++r) limit[r] = p.causal ? min(nk - 1, (row0 + r) % p.Nq + shift) : nk - 1;
    const int first_limit = p.causal ? min(nk - 1, (last_row / p.Nq != row0 / p.Nq ? 0 : row0 % p.Nq) + shift) : nk - 1;

    float m_ref[NR], top[NR], l[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) top[r] = -INFINITY;
    bool ok = true;
    bool met = false;  // the one-time meeting of the warps over the row references has taken place
    do {
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        m_ref[r] = top[r];  // second pass: the maximum is known
        l[r] = 0.f;
      }
      for (int j = base; j < base + n_tiles; ++j) {
        const int buf = j & 1;
        if (!mbar_wait_warp(s_full(buf), (j >> 1) & 1, p.status, WK_ERR_TIMEOUT_MMA)) {
          ok = false;
          break;
        }
        tc_fence_after();
        uint32_t raw[NR];
        tmem_ld_cols<NR>(tmem_base + lane_addr + E_S_COL + 32 * buf, raw);
        tc_wait_ld();
        tc_fence_before();
        mbar_arrive(s_free(buf));
        const int key = (t0 + j - base) * E_KEYS + r_key;
        const int tile_end = (t0 + j - base + 1) * E_KEYS - 1;
        if (tile_end > first_limit) {
#pragma unroll
          for (int r = 0; r < NR; ++r)
            if (key > limit[r]) raw[r] = 0xff800000u;
          if (tile_end >= nk && key >= nk) {
            // rows of V beyond the last key: whatever the cache holds there, 0 . V has to be 0
            const uint32_t row = smem_base + (j % E_STAGES) * 2 * E_TILE_BYTES + E_TILE_BYTES + r_key * 128;
#pragma unroll
            for (int c = 0; c < 8; ++c)
              asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(row + 16 * c), "r"(0) : "memory");
          }
        }
        float cm[NR];  // block maxima in base 2 (beta > 0, checked on the host)
#pragma unroll
        for (int r = 0; r < NR; ++r) cm[r] = warp_max(__uint_as_float(raw[r])) * beta;
        if (j == base && passes == 0) {
          // the row reference: maximum over the split's first tile
          const uint32_t mine = xch + quad * 64;
          if (lane == 0)
#pragma unroll
            for (int r = 0; r < NR; ++r) sts_f32(mine + 4 * r, cm[r]);
          softmax_barrier();
          met = true;
#pragma unroll
          for (int r = 0; r < NR; ++r)
            m_ref[r] = fmaxf(fmaxf(lds_f32(xch + 4 * r), lds_f32(xch + 64 + 4 * r)),
                             fmaxf(lds_f32(xch + 128 + 4 * r), lds_f32(xch + 192 + 4 * r)));
        }
        if (j >= 2 && !mbar_wait_warp(p_free(buf), ((j >> 1) - 1) & 1, p.status, WK_ERR_TIMEOUT_MMA)) {
          ok = false;
          break;
        }
        const uint32_t dst = p_smem + buf * C::P_BYTES + (r_key & 15);
        uint32_t my_sf = 0;  // lane r keeps the scale byte of row r
#pragma unroll
        for (int r = 0; r < NR; r += 2) {  // two rows at a time: conversions work on pairs
          float x[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            top[r + i] = fmaxf(top[r + i], cm[r + i]);
            const bool live = cm[r + i] > -INFINITY;
            const float kf = live ? fminf(fmaxf(ceilf(cm[r + i] - m_ref[r + i]), -118.f), E_MAX_EXP) : 0.f;
            const float bias = live ? static_cast<float>(E_P_OFFSET) - kf - m_ref[r + i] : 0.f;
            x[i] = ex2_approx(fmaf(__uint_as_float(raw[r + i]), beta, bias));
            const int sf = live ? 127 + static_cast<int>(kf) - E_P_OFFSET : 0;
            l[r + i] = fmaf(x[i], __uint_as_float(static_cast<uint32_t>(sf) << 23), l[r + i]);
            if (lane == r + i) my_sf = static_cast<uint32_t>(sf);
            if (lane == NR + r + i) my_sf = static_cast<uint32_t>(max(sf - 4, 0));
          }
          const uint16_t hi = cvt_e4m3x2(x[0], x[1]);
          float b0, b1;
          unpack_e4m3x2(hi, b0, b1);
          const uint16_t lo = cvt_e4m3x2((x[0] - b0) * 16.f, (x[1] - b1) * 16.f);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint32_t at = dst + (r + i) * 128 + static_cast<uint32_t>(((r_key >> 4) ^ ((r + i) & 7)) << 4);
            sts_u8(at, i ? hi >> 8 : hi);
            sts_u8(at + NR * 128, i ? lo >> 8 : lo);
          }
        }
        // scale bytes in the layout tcgen05.cp copies: row n at 16 n, key block at byte quad
        if (lane < C::N) sts_u8(sf_smem + buf * C::SF_BYTES + lane * 16 + quad, my_sf);
        fence_proxy_async_smem();
        mbar_arrive(p_full(buf));
      }
      if (!met) {  // no tile, or a wait gave up: this warp still owes the others the meeting
        softmax_barrier();
        met = true;
      }
      // the sums over keys; does any row need the second pass?
      bool far = false;
#pragma unroll
      for (int r = 0; r < NR; ++r) {
#pragma unroll
        for (int i = 16; i > 0; i >>= 1) l[r] += __shfl_xor_sync(0xffffffffu, l[r], i);
      }
      const uint32_t sums = xch + 256 + quad * 64, tops = xch + quad * 64;
      softmax_barrier();
      if (lane == 0)
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          sts_f32(sums + 4 * r, l[r]);
          sts_f32(tops + 4 * r, top[r]);
        }
      softmax_barrier();
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        l[r] = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          l[r] += lds_f32(xch + 256 + w * 64 + 4 * r);
          top[r] = fmaxf(top[r], lds_f32(xch + w * 64 + 4 * r));
        }
        far |= top[r] - m_ref[r] > E_MAX_EXP;
      }
      if (r_key == 0) asm volatile("st.shared.b32 [%0], %1;" ::"r"(again_slot), "r"(far && ok ? 1 : 0) : "memory");
      if (ok && n_tiles > 0) ok = mbar_wait_warp(o_full, passes & 1, p.status, WK_ERR_TIMEOUT_MMA);
      tc_fence_after();
    } while (another_pass());

    // ---- this CTA's partial result: O^T (lane = head-dim element) to shared memory as [row][d]
    const uint32_t part = smem_base;
    uint32_t hi[NR], lo[NR];
    if (n_tiles > 0 && ok) {
      tmem_ld_cols<NR>(tmem_base + lane_addr + E_O_COL, hi);
      tmem_ld_cols<NR>(tmem_base + lane_addr + E_O_COL + NR, lo);
      tc_wait_ld();
    }
#pragma unroll
    for (int r = 0; r < NR; ++r)
      sts_f32(part + (r * C::PITCH + r_key) * 4,
              n_tiles > 0 && ok ? __uint_as_float(hi[r]) + __uint_as_float(lo[r]) : 0.f);
    const uint32_t stats = xch + 512;
    if (r_key == 0)
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const bool seen = top[r] > -INFINITY;
        sts_f32(stats + 4 * r, seen ? m_ref[r] : -INFINITY);
        sts_f32(stats + 64 + 4 * r, l[r]);
        sts_f32(stats + 128 + 4 * r, top[r]);
      }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, E_TMEM_COLS);
  }
  if (p.splits > 1) cluster_sync();
  // ---- combine: each CTA finishes the rows congruent to its rank, in the order of the splits
  const int quads = p.d / 4;
  for (int i = threadIdx.x; i < NR * quads; i += E_THREADS) {
    const int r = (i / quads) * p.splits + split, col = (i % quads) * 4;
    if (r >= NR || row0 + r >= rows) break;
    auto load = [&](int from, uint32_t addr) {
      float x;
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(p.splits > 1 ? mapa(addr, from) : addr));
      return x;
    };
    const uint32_t stats = xch + 512 + 4 * r;
    float m[E_MAX_SPLIT], lsum[E_MAX_SPLIT], tp[E_MAX_SPLIT], o[E_MAX_SPLIT][4];
#pragma unroll
    for (int x = 0; x < E_MAX_SPLIT; ++x) {
      m[x] = tp[x] = -INFINITY;
      lsum[x] = o[x][0] = o[x][1] = o[x][2] = o[x][3] = 0.f;
      if (x < p.splits) {
        m[x] = load(x, stats);
        lsum[x] = load(x, stats + 64);
        tp[x] = load(x, stats + 128);
        const uint32_t addr = smem_base + (r * C::PITCH + col) * 4;
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(o[x][0]), "=f"(o[x][1]), "=f"(o[x][2]), "=f"(o[x][3])
                     : "r"(p.splits > 1 ? mapa(addr, x) : addr));
      }
    }
    float mm = -INFINITY, m_true = -INFINITY, sum = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int x = 0; x < E_MAX_SPLIT; ++x) {
      mm = fmaxf(mm, m[x]);
      m_true = fmaxf(m_true, tp[x]);
    }
#pragma unroll
    for (int x = 0; x < E_MAX_SPLIT; ++x) {
      const float f = m[x] > -INFINITY ? exp2f(m[x] - mm) : 0.f;
      sum = fmaf(lsum[x], f, sum);
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[c] = fmaf(o[x][c], f, acc[c]);
    }
    const bool empty = !(sum > 0.f);
    const float inv = empty ? 0.f : p.v_descale[b * p.Hkv + hkv] / sum;
    const int head = hkv * group + (row0 + r) / p.Nq, query = (row0 + r) % p.Nq;
    uint2 w;
    w.x = pack_bf16x2(acc[0] * inv, acc[1] * inv);
    w.y = pack_bf16x2(acc[2] * inv, acc[3] * inv);
    *reinterpret_cast<uint2*>(p.out + b * p.out_strides[0] + head * p.out_strides[1] + query * p.out_strides[2] + col) = w;
    if (p.write_lse && col == 0) {
      const int64_t off = b * p.lse_strides[0] + head * p.lse_strides[1] + query;
      const float lse = empty ? INFINITY : mm + log2f(sum);
      p.lse[off] = p.lse_natural ? lse * 0.6931471805599453f : lse;
      p.pmax[off] = empty ? 0.f : exp2f(m_true - lse);
    }
  }
  __syncwarp();  // lanes leave the loop at different rows; the barrier wants the warp together
  if (p.splits > 1) cluster_sync();  // nobody leaves while its partial results may still be read
}

template <int NR>
int launch_decode(const CUtensorMap& tk, const CUtensorMap& tv, DecodeParams& p, cudaStream_t stream) {
  using C = DecodeCfg<NR>;
  const void* fn = reinterpret_cast<const void*>(attn_decode_kernel<NR>);
  if (allow_smem(fn, C::SMEM)) return WK_E_CUDA;
  const int rows = p.Hq / p.Hkv * p.Nq;
  return launch_pdl(fn, dim3(p.splits, p.B * p.Hkv, (rows + NR - 1) / NR), E_THREADS, C::SMEM, stream, p.splits,
                    {const_cast<CUtensorMap*>(&tk), const_cast<CUtensorMap*>(&tv), &p});
}

}  // namespace

int attn_decode_splits(const wk_attn_fwd_args* a, int64_t units, int sms) {
  // two CTAs per SM; at least two tiles for a split
  int s = 1;
  while (s < E_MAX_SPLIT && units * s * 2 <= 2 * sms && a->Nk >= 2 * E_KEYS * s * 2) s *= 2;
  return s;
}

int launch_attn_decode(const wk_attn_fwd_args* a, cudaStream_t stream) {
  const int sms = sm_count();
  if (sms <= 0) return WK_E_CUDA;
  DecodeParams p = {};
  p.status = status_word();
  if (!p.status) return WK_E_CUDA;
  CUtensorMap maps[2];
  for (int i = 0; i < 2; ++i) {
    const int64_t* st = i ? a->v_strides : a->k_strides;
    const uint64_t dims[4] = {static_cast<uint64_t>(a->d), static_cast<uint64_t>(a->Nk), static_cast<uint64_t>(a->Hkv),
                              static_cast<uint64_t>(a->B)};
    const uint64_t str[3] = {static_cast<uint64_t>(st[2]), static_cast<uint64_t>(st[1]), static_cast<uint64_t>(st[0])};
    const uint32_t box[4] = {128, E_KEYS, 1, 1};
    if (int r = encode_tmap(&maps[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, i ? a->v : a->k, dims, str, box,
                            CU_TENSOR_MAP_SWIZZLE_128B))
      return r;
  }
  p.q = static_cast<const uint8_t*>(a->q);
  p.out = static_cast<__nv_bfloat16*>(a->out);
  p.lse = a->lse;
  p.pmax = a->pmax;
  p.q_descale = a->q_descale;
  p.k_descale = a->k_descale;
  p.v_descale = a->v_descale;
  for (int i = 0; i < 3; ++i) {
    p.q_strides[i] = a->q_strides[i];
    p.out_strides[i] = a->out_strides[i];
  }
  p.lse_strides[0] = a->lse_strides[0];
  p.lse_strides[1] = a->lse_strides[1];
  p.B = a->B, p.Hq = a->Hq, p.Hkv = a->Hkv, p.Nq = a->Nq, p.Nk = a->Nk, p.d = a->d;
  p.causal = a->causal, p.write_lse = a->write_lse, p.lse_natural = a->lse_natural;
  p.seqused_k = a->seqused_k;
  p.softmax_scale = a->softmax_scale;
  const int rows = a->Hq / a->Hkv * a->Nq;
  const int nr = rows <= 8 ? 8 : 16;
  p.splits = attn_decode_splits(a, static_cast<int64_t>(a->B) * a->Hkv * ((rows + nr - 1) / nr), sms);
  return nr == 8 ? launch_decode<8>(maps[0], maps[1], p, stream) : launch_decode<16>(maps[0], maps[1], p, stream);
}

}  // namespace wk
