// BF16 flash-attention backward for sm_100a, head dimension 128.
//
//   S = alpha . q k^T,  P = softmax(S) = 2^(S . log2e - L)   (L: the forward's base-2 lse)
//   dV = P^T dO,  dP = dO v^T,  D = rowsum(dO * O),  dS = P * (dP - D),
//   dQ = alpha . dS k,  dK = alpha . dS^T q
// as in the reference's bf16 backward (warpy_kernels/attn/bwd_common.py:88-304, bwd_sm120.py:436-464).  Same three
// kernels and the same pipeline as the FP8 backward (attn_bwd_fp8.cu), with tcgen05.mma kind::f16 and P^T, dS^T
// rounded to bf16 instead of MXFP8:
//
//  1. attn_bwd_bf16_prep4_kernel (attn_bwd_bf16_prep_kernel for rows not on 16-byte boundaries): per query row
//     D = sum(dO . O) and the row record (-L, -D).
//  2. attn_bwd_bf16_dkdv_kernel: CTA = 128 keys of one (batch, kv head), K and V resident in shared memory, loop over
//     the group's query heads and query tiles; S^T = K Q^T and dP^T = V dO^T into TMEM, threads turn them into
//     bf16 P^T and dS^T back in TMEM, dV += P^T dO and dK += dS^T Q (A from TMEM, B = the same Q / dO tiles read
//     MN-major).  dV and dK stay in TMEM for the whole CTA.
//  3. attn_bwd_bf16_dq_kernel: CTA = 128 queries, loop over key tiles, recomputes S and dP, dQ += dS K in TMEM: no
//     atomics, deterministic.  It runs beside the dK/dV kernel.
// A row of a tile is 256 bytes, two 128-byte swizzle spans: every tile is two boxes of 64 head-dim elements,
// 16 KiB apart in shared memory.
//
// Tensor-core bound: 10 . B . Hq . Nq . Nk . d flops of algorithmic work (half when causal).  Per 128 x 128 tile the dQ
// kernel takes 2180 cycles (1536 of tensor pipe), the dK/dV kernel 3600 (2560: its N = 64 products are paced by the
// shared-memory reads of their operands); the chain from a score buffer's release to its next scores paces both.  With the
// codes written over the scores and one thread issuing all products the two took 8600 cycles: 4 x 32 heads, 4096 x 4096
// without mask 3966 -> 3491 us, causal 2235 -> 1953, 2 x 32 / 8 heads, 2048 x 2048 causal 278 -> 240.
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "host_common.h"

namespace wk {
namespace {

constexpr int BM = 128;  // queries per tile
constexpr int BN = 128;  // keys per tile
constexpr int D = 128;  // largest head dimension; with 64 (the main kernels are instantiated per head dimension) a row is one swizzle span instead of
                        // two: the second box of every tile is not loaded and the products take half the K steps
constexpr int CHUNK = 64;                        // head-dim elements per 128-byte swizzle span
constexpr int CHUNK_BYTES = 128 * CHUNK * 2;     // 16 KiB: 128 rows x 128 bytes
constexpr int TILE_BYTES = 2 * CHUNK_BYTES;      // 32 KiB: 128 rows x 256 bytes
constexpr int THREADS = 640;        // TMA warp, three MMA warps, 16 element-wise warps (four threads per row of a tile)
constexpr int EW_THREADS = 512;
constexpr int GROUP_THREADS = 256;  // dK/dV: the element-wise threads of one 64-query half of a tile
constexpr int TMEM_COLS = 512;
constexpr float LOG2E = 1.4426950408889634f;

// ---------------------------------------------------------------------------
// 1. prep
// ---------------------------------------------------------------------------
struct PrepParams {
  const __nv_bfloat16* dout;  // [B,Hq,Nq,D] with element strides
  const __nv_bfloat16* out;
  const float* lse;           // [B,Hq,*] base 2
  float* qstat;               // [B,Hq,Nq_pad/128][2][128]: per 128 rows the arrays -L and -D
  int64_t do_sb, do_sh, do_sn;
  int64_t o_sb, o_sh, o_sn;
  int64_t lse_sb, lse_sh;
  int B, Hq, Nq, nq_pad, d;
};

// one warp per query row, 4 consecutive elements per lane
__global__ void __launch_bounds__(256) attn_bwd_bf16_prep_kernel(const PrepParams p) {
  pdl_launch_dependents();  // the dK/dV kernel waits for this one to complete
  pdl_wait();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x % 32;
  const int64_t rows = static_cast<int64_t>(p.B) * p.Hq * p.nq_pad;
  if (warp >= rows) return;
  const int i = warp % p.nq_pad;
  const int h = (warp / p.nq_pad) % p.Hq;
  const int b = warp / (p.nq_pad * p.Hq);
  // the two values of row i sit 128 floats apart inside the row's tile of 128
  float* stat = p.qstat + ((static_cast<int64_t>(b) * p.Hq + h) * p.nq_pad + (i & ~127)) * 2 + (i & 127);
  if (i >= p.Nq) {
    // padding rows: lse = +inf makes every probability zero
    if (lane < 2) stat[lane * 128] = lane == 0 ? -INFINITY : 0.f;
    return;
  }
  const __nv_bfloat16* dsrc = p.dout + b * p.do_sb + h * p.do_sh + static_cast<int64_t>(i) * p.do_sn + lane * 4;
  const __nv_bfloat16* osrc = p.out + b * p.o_sb + h * p.o_sh + static_cast<int64_t>(i) * p.o_sn + lane * 4;
  const bool mine = lane * 4 < p.d;  // head dimension 64: half the lanes only join the reduction
  const uint2 draw = mine ? *reinterpret_cast<const uint2*>(dsrc) : make_uint2(0, 0);
  const uint2 oraw = mine ? *reinterpret_cast<const uint2*>(osrc) : make_uint2(0, 0);
  float dsum = __uint_as_float(draw.x << 16) * __uint_as_float(oraw.x << 16) +
               __uint_as_float(draw.x & 0xffff0000u) * __uint_as_float(oraw.x & 0xffff0000u) +
               __uint_as_float(draw.y << 16) * __uint_as_float(oraw.y << 16) +
               __uint_as_float(draw.y & 0xffff0000u) * __uint_as_float(oraw.y & 0xffff0000u);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) dsum += __shfl_xor_sync(0xffffffffu, dsum, off);
  if (lane == 0) {
    stat[0] = -p.lse[b * p.lse_sb + h * p.lse_sh + i];
    stat[128] = -dsum;
  }
}

// The same for tensors whose strides are multiples of 8 elements: four query rows per warp, 8 lanes per row and 16
// consecutive elements per lane, read with 16-byte loads (the kernel is HBM-bound; one row per warp keeps too few
// bytes in flight).
__global__ void __launch_bounds__(256) attn_bwd_bf16_prep4_kernel(const PrepParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x % 32;
  const int sub = lane & 7;
  const int64_t rows = static_cast<int64_t>(p.B) * p.Hq * p.nq_pad;  // a multiple of 128
  if (warp * 4 >= rows) return;
  const int64_t row_id = warp * 4 + (lane >> 3);
  const int i = static_cast<int>(row_id % p.nq_pad);
  const int h = static_cast<int>((row_id / p.nq_pad) % p.Hq);
  const int b = static_cast<int>(row_id / (static_cast<int64_t>(p.nq_pad) * p.Hq));
  const bool live = i < p.Nq;  // padding rows take part in the shuffles with zeros
  uint4 draw[2] = {}, oraw[2] = {};
  if (live && sub * 16 < p.d) {  // head dimension 64: half the lanes only join the reduction
    const uint4* dsrc = reinterpret_cast<const uint4*>(p.dout + b * p.do_sb + h * p.do_sh +
                                                       static_cast<int64_t>(i) * p.do_sn + sub * 16);
    const uint4* osrc =
        reinterpret_cast<const uint4*>(p.out + b * p.o_sb + h * p.o_sh + static_cast<int64_t>(i) * p.o_sn + sub * 16);
    draw[0] = dsrc[0];
    draw[1] = dsrc[1];
    oraw[0] = osrc[0];
    oraw[1] = osrc[1];
  }
  const uint32_t dw[8] = {draw[0].x, draw[0].y, draw[0].z, draw[0].w, draw[1].x, draw[1].y, draw[1].z, draw[1].w};
  const uint32_t ow[8] = {oraw[0].x, oraw[0].y, oraw[0].z, oraw[0].w, oraw[1].x, oraw[1].y, oraw[1].z, oraw[1].w};
  float dsum = 0.f;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    dsum += __uint_as_float(dw[c] << 16) * __uint_as_float(ow[c] << 16) +
            __uint_as_float(dw[c] & 0xffff0000u) * __uint_as_float(ow[c] & 0xffff0000u);
  }
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) dsum += __shfl_xor_sync(0xffffffffu, dsum, off);
  // the two values of row i sit 128 floats apart inside the row's tile of 128
  float* stat = p.qstat + ((static_cast<int64_t>(b) * p.Hq + h) * p.nq_pad + (i & ~127)) * 2 + (i & 127);
  if (!live) {
    // padding rows: lse = +inf makes every probability zero
    if (sub < 2) stat[sub * 128] = sub == 0 ? -INFINITY : 0.f;
  } else if (sub == 0) {
    stat[0] = -p.lse[b * p.lse_sb + h * p.lse_sh + i];
    stat[128] = -dsum;
  }
}

// ---------------------------------------------------------------------------
// helpers shared by the two main kernels
// ---------------------------------------------------------------------------
// Four consecutive floats from shared memory (the row records: every thread reads the same address, a broadcast).
__device__ __forceinline__ float4 lds_f4(uint32_t saddr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(saddr));
  return v;
}

// The element-wise code keeps a block of 32 values as 16 packed fp32 pairs; they go to TMEM as 16 bf16 pairs.
__device__ __forceinline__ void store_block_bf16(const uint64_t (&x)[16], uint32_t taddr) {
  uint32_t lo[8], hi[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float a, b, c, d;
    unpack_f32x2(x[i], a, b);
    unpack_f32x2(x[8 + i], c, d);
    lo[i] = pack_bf16x2(a, b);
    hi[i] = pack_bf16x2(c, d);
  }
  tmem_st8(taddr, lo);
  tmem_st8(taddr + 8, hi);
}

struct BwdParams {
  const float* qstat;    // [B,Hq,nq_pad/128][2][128]: -L and -D of 128 rows
  __nv_bfloat16* dq;     // [B,Hq,Nq,D] contiguous
  __nv_bfloat16* dk;     // [B,Hkv,Nk,D] contiguous
  __nv_bfloat16* dv;
  int B, Hq, Hkv, Nq, Nk, nq_pad;
  int d;  // head dimension, 128 or 64
  int causal;
  int kv_band, q_band;  // heads whose blocks are handed out together (band_order)
  float softmax_scale;
  int* status;
};

// ---------------------------------------------------------------------------
// 2. dK / dV
// ---------------------------------------------------------------------------
constexpr int A_STAGES = 2;
constexpr int A_STAT_BYTES = BM * 8;
constexpr int A_STAGE_BYTES = 2 * TILE_BYTES + A_STAT_BYTES;
// Requested size is padded past half an SM's shared memory: each CTA allocates all 512 TMEM columns, so a second
// resident CTA could only spin in tcgen05.alloc.
constexpr int A_SMEM_BYTES = 2 * TILE_BYTES + A_STAGES * A_STAGE_BYTES + 1024 + 256;  // 197 KiB: one CTA per SM
// Work goes by units of 64 queries: S^T and dP^T of a unit go into the one score buffer, which the unit's element-wise
// group (h = 0, 1 in turn) frees as soon as it holds the values in registers; P^T and dS^T go to columns of their own, one
// set per group.  So the scores of the next unit are under way while a unit's P and dS are computed and its sums issued.
constexpr int A_ST_COL = 0, A_DPT_COL = 64, A_P_COL = 128, A_DS_COL = 192, A_DV_COL = 256, A_DK_COL = 384;
template <int DH>
__global__ void __launch_bounds__(THREADS, 1)
attn_bwd_bf16_dkdv_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                     const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                     const __grid_constant__ BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t k_smem = smem_base;
  const uint32_t v_smem = k_smem + TILE_BYTES;
  const uint32_t stage_smem = v_smem + TILE_BYTES;  // per stage: Q tile, dO tile, row records
  const uint32_t bar_base = stage_smem + A_STAGES * A_STAGE_BYTES;
  const uint32_t kv_full = bar_base;
  auto q_full = [&](int s) { return bar_base + 8u * (1 + s); };
  auto q_empty = [&](int s) { return bar_base + 8u * (1 + A_STAGES + s); };
  // of the two element-wise groups (h = 0, 1)
  const uint32_t misc = bar_base + 8u * (1 + 2 * A_STAGES);
  auto s_full = [&](int h) { return misc + 8u * h; };
  auto s_free = [&](int h) { return misc + 16 + 8u * h; };
  auto p_full = [&](int h) { return misc + 32 + 8u * h; };  // the group's P^T and dS^T are in tensor memory
  auto p_free = [&](int h) { return misc + 48 + 8u * h; };  // the products that read them are complete
  const uint32_t acc_full = misc + 64;
  const uint32_t tmem_slot = acc_full + 8;

  const int warp = threadIdx.x / 32;
  const int lane = threadIdx.x % 32;
  const BandBlock at = band_order(blockIdx.x, (p.Nk + BN - 1) / BN, p.B * p.Hkv, p.kv_band);
  const int hkv = at.head % p.Hkv;
  const int b = at.head / p.Hkv;
  const int n0 = at.rank * BN;  // the first key blocks see the most queries
  const int group = p.Hq / p.Hkv;
  const int shift = p.Nk - p.Nq;
  const int num_m = (p.Nq + BM - 1) / BM;
  // first query tile that sees a key of this block (bottom-right aligned causal mask)
  const int m_first = p.causal ? min(num_m, max(0, n0 - shift) / BM) : 0;
  const int tiles_per_head = num_m - m_first;
  const int n_iter = group * tiles_per_head;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < A_STAGES; ++s) {
      mbar_init(q_full(s), 1);
      mbar_init(q_empty(s), 1);
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(s_full(h), 2);  // S^T and dP^T come from two threads
      mbar_init(s_free(h), GROUP_THREADS);
      mbar_init(p_full(h), GROUP_THREADS);
      mbar_init(p_free(h), 1);
    }
    mbar_init(acc_full, 1);
    mbar_fence_init();
    prefetch_tmap(&tmap_q);
    prefetch_tmap(&tmap_k);
    prefetch_tmap(&tmap_v);
    prefetch_tmap(&tmap_do);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  // What this kernel reads is there once the prep kernel has completed; the dQ kernel reads the same and may start from
  // here on, beside this one (it ends after it).
  pdl_wait();
  pdl_launch_dependents();

  if (warp == 0) {
    if (lane == 0 && n_iter > 0) {
      const int chunks = DH / CHUNK;
      mbar_expect_tx(kv_full, 2 * chunks * CHUNK_BYTES);
      for (int c = 0; c < chunks; ++c) {
        tma_load_4d(k_smem + c * CHUNK_BYTES, &tmap_k, kv_full, c * CHUNK, n0, hkv, b);
        tma_load_4d(v_smem + c * CHUNK_BYTES, &tmap_v, kv_full, c * CHUNK, n0, hkv, b);
      }
      for (int it = 0; it < n_iter; ++it) {
        const int s = it % A_STAGES;
        const uint32_t ph = (it / A_STAGES) & 1;
        const int hq = hkv * group + it / tiles_per_head;
        const int m0 = (m_first + it % tiles_per_head) * BM;
        if (!mbar_wait(q_empty(s), ph ^ 1, p.status, WK_ERR_TIMEOUT_EMPTY)) break;
        const uint32_t base = stage_smem + s * A_STAGE_BYTES;
        mbar_expect_tx(q_full(s), 2 * chunks * CHUNK_BYTES + A_STAT_BYTES);
        for (int c = 0; c < chunks; ++c) {
          tma_load_4d(base + c * CHUNK_BYTES, &tmap_q, q_full(s), c * CHUNK, m0, hq, b);
          tma_load_4d(base + TILE_BYTES + c * CHUNK_BYTES, &tmap_do, q_full(s), c * CHUNK, m0, hq, b);
        }
        bulk_load(base + 2 * TILE_BYTES, p.qstat + ((static_cast<int64_t>(b) * p.Hq + hq) * p.nq_pad + m0) * 2,
                  A_STAT_BYTES, q_full(s));
      }
    }
    __syncwarp();
  } else if (warp == 1 || warp == 2) {
    if (lane == 0 && n_iter > 0) {
      // S^T = K Q^T by warp 1, dP^T = V dO^T by warp 2, side by side: the time from the buffer's release to its next
      // scores is on every unit's critical path, and a thread needs ~90 cycles per MMA it issues here
      const int which = warp - 1;
      constexpr uint32_t idesc = make_idesc(1, 1, 0, 0, BN, BM / 2);
      const uint32_t d_tmem = tmem_base + (which == 0 ? A_ST_COL : A_DPT_COL);
      const uint64_t a_desc = smem_desc_sw128(which == 0 ? k_smem : v_smem, 16, 1024);
      bool ok = mbar_wait(kv_full, 0, p.status, WK_ERR_TIMEOUT_LOAD);
      for (int n = 0; ok && n < 2 * n_iter; ++n) {
        const int it = n >> 1, h = n & 1, s = it % A_STAGES;
        if (h == 0 && !mbar_wait(q_full(s), (it / A_STAGES) & 1, p.status, WK_ERR_TIMEOUT_LOAD)) break;
        if (n > 0 && !mbar_wait(s_free(1 - h), ((n - 1) >> 1) & 1, p.status, WK_ERR_TIMEOUT_P)) break;
        tc_fence_after();
        // rows 64 h.. of the Q / dO tile are 64 x 128 bytes further on (+512 in descriptor units); 16 head-dim elements
        // per MMA = 32 bytes inside a span, the second span one chunk (16 KiB) further on
        const uint64_t b_desc = smem_desc_sw128(stage_smem + s * A_STAGE_BYTES + which * TILE_BYTES, 16, 1024) + 512 * h;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint64_t off = (k >> 2) * (CHUNK_BYTES >> 4) + 2 * (k & 3);
          if (16 * k < DH) mma_f16_ss(d_tmem, a_desc + off, b_desc + off, idesc, k != 0);
        }
        tc_commit(s_full(h));
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    if (lane == 0 && n_iter > 0) {
      // dV += P^T dO and dK += dS^T Q over the unit's 64 queries.  B operands: the dO / Q tiles again, now read MN-major
      // (K = queries, 16 per step = 2048 bytes; N = head dim, its two spans 16 KiB apart)
      const uint32_t idesc = make_idesc(1, 1, 0, 1, BN, DH);
      for (int n = 0; n < 2 * n_iter; ++n) {
        const int it = n >> 1, h = n & 1, s = it % A_STAGES;
        if (!mbar_wait(q_full(s), (it / A_STAGES) & 1, p.status, WK_ERR_TIMEOUT_LOAD)) break;
        if (!mbar_wait(p_full(h), it & 1, p.status, WK_ERR_TIMEOUT_P)) break;
        tc_fence_after();
        const uint64_t q_desc = smem_desc_sw128(stage_smem + s * A_STAGE_BYTES, CHUNK_BYTES, 1024) + 512 * h;
        const uint64_t do_desc = q_desc + (TILE_BYTES >> 4);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mma_f16_ts(tmem_base + A_DV_COL, tmem_base + A_P_COL + 32 * h + 8 * k, do_desc + 128 * k, idesc, (n | k) != 0);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mma_f16_ts(tmem_base + A_DK_COL, tmem_base + A_DS_COL + 32 * h + 8 * k, q_desc + 128 * k, idesc, (n | k) != 0);
        tc_commit(p_free(h));
        if (h == 1) tc_commit(q_empty(s));
        if (n + 1 == 2 * n_iter) tc_commit(acc_full);
      }
    }
    __syncwarp();
  } else {
    const int quad = warp & 3;
    const int c = (warp - 4) >> 2;   // which block of 32 of the tile's 128 queries this thread handles
    const int h = c >> 1;            // its group
    const int r = quad * 32 + lane;  // key row of the tile == TMEM lane
    const int key = n0 + r;
    const uint32_t lane_tmem = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const float beta = p.softmax_scale * LOG2E;
    bool ok = true;

    int m = m_first;  // this iteration's query tile
    for (int it = 0; it < n_iter; ++it) {
      const int m0 = m * BM;
      if (++m == num_m) m = m_first;
      if (!mbar_wait_warp(s_full(h), it & 1, p.status, WK_ERR_TIMEOUT_MMA)) {
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t sraw[32], draw[32];
      tmem_ld32(lane_tmem + A_ST_COL + 32 * (c & 1), sraw);
      tmem_ld32(lane_tmem + A_DPT_COL + 32 * (c & 1), draw);
      tc_wait_ld();
      tc_fence_before();
      mbar_arrive(s_free(h));
      // the tile's row records: arrays -L and -D of 128 queries each, read four queries at a time
      const uint32_t stat = stage_smem + (it % A_STAGES) * A_STAGE_BYTES + 2 * TILE_BYTES + c * 128;
      uint32_t pw[2][8], dw[2][8];  // P^T and dS^T as bf16 pairs
      auto elements = [&](auto masked) {
        // query column i is visible to this key iff key < Nk and (not causal or key <= m0 + 32 c + i + shift)
        const int first = !decltype(masked)::value ? 0 : key >= p.Nk ? BM : p.causal ? key - shift - m0 - 32 * c : 0;
        const uint64_t beta2 = pack_f32x2(beta, beta);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          // the same addresses for every thread: shared-memory broadcasts
          const float4 nl = lds_f4(stat + 16 * i), nd = lds_f4(stat + 512 + 16 * i);
          const float nlv[4] = {nl.x, nl.y, nl.z, nl.w}, ndv[4] = {nd.x, nd.y, nd.z, nd.w};
#pragma unroll
          for (int x = 0; x < 4; x += 2) {
            const int e = 4 * i + x;
            float x0, x1, d0, d1;
            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sraw[e]), __uint_as_float(sraw[e + 1])), beta2,
                                   pack_f32x2(nlv[x], nlv[x + 1])), x0, x1);
            float p0 = ex2_approx(x0), p1 = ex2_approx(x1);
            if (decltype(masked)::value) {
              if (e < first) p0 = 0.f;
              if (e + 1 < first) p1 = 0.f;
            }
            // dS = P (dP - D)
            unpack_f32x2(mul_f32x2(pack_f32x2(p0, p1),
                                   add_f32x2(pack_f32x2(__uint_as_float(draw[e]), __uint_as_float(draw[e + 1])),
                                             pack_f32x2(ndv[x], ndv[x + 1]))), d0, d1);
            pw[e / 16][e / 2 % 8] = pack_bf16x2(p0, p1);
            dw[e / 16][e / 2 % 8] = pack_bf16x2(d0, d1);
          }
        }
      };
      // uniform over the CTA: does this (key block, query tile) pair contain any masked score?
      if ((n0 + BN > p.Nk) || (p.causal && n0 + BN - 1 > m0 + shift))
        elements(std::true_type{});
      else
        elements(std::false_type{});
      if (it > 0 && !mbar_wait_warp(p_free(h), (it - 1) & 1, p.status, WK_ERR_TIMEOUT_MMA)) {
        ok = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        tmem_st8(lane_tmem + A_P_COL + 16 * c + 8 * i, pw[i]);
        tmem_st8(lane_tmem + A_DS_COL + 16 * c + 8 * i, dw[i]);
      }
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(p_full(h));
    }

    if (n_iter > 0 && ok) ok = mbar_wait_warp(acc_full, 0, p.status, WK_ERR_TIMEOUT_MMA);
    if (ok) {
      tc_fence_after();
      const float dk_scale = p.softmax_scale;
      const int64_t row_off = ((static_cast<int64_t>(b) * p.Hkv + hkv) * p.Nk + key) * DH;
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        const uint32_t src = lane_tmem + (which == 0 ? A_DV_COL : A_DK_COL);
        __nv_bfloat16* dst_row = (which == 0 ? p.dv : p.dk) + row_off;
        const float scale = which == 0 ? 1.f : dk_scale;
        {
          uint32_t v[32];
          if (n_iter > 0) {  // uniform: TMEM loads are warp-wide
            tmem_ld32(src + c * 32, v);
            tc_wait_ld();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0;
          }
          if (key < p.Nk && c * 32 < DH) {
            uint4* dst = reinterpret_cast<uint4*>(dst_row + c * 32);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint4 w;
              w.x = pack_bf16x2(__uint_as_float(v[8 * i + 0]) * scale, __uint_as_float(v[8 * i + 1]) * scale);
              w.y = pack_bf16x2(__uint_as_float(v[8 * i + 2]) * scale, __uint_as_float(v[8 * i + 3]) * scale);
              w.z = pack_bf16x2(__uint_as_float(v[8 * i + 4]) * scale, __uint_as_float(v[8 * i + 5]) * scale);
              w.w = pack_bf16x2(__uint_as_float(v[8 * i + 6]) * scale, __uint_as_float(v[8 * i + 7]) * scale);
              dst[i] = w;
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------
// 3. dQ
// ---------------------------------------------------------------------------
// Per tile of 128 keys S and dP are one N = 128 product each (the operands then cost shared memory as many cycles as
// the tensor pipe; N = 64 half as many again) into one pair of score buffers, which the element-wise warps free as soon as
// they hold the values in registers; dS goes to columns of its own, of which there are two sets.  So the scores of a tile
// are under way while dS of the tile before is computed and its product issued.  K has a ring of three tiles and V one of
// two: V is free once dP is complete, K only after dQ += dS K.
constexpr int B_K_STAGES = 3, B_V_STAGES = 2;
constexpr int B_SMEM_BYTES = (2 + B_K_STAGES + B_V_STAGES) * TILE_BYTES + 1024 + 256;  // 225 KiB: one CTA per SM
constexpr int B_S_COL = 0, B_DP_COL = 128, B_DQ_COL = 256, B_DS_COL = 384;

template <int DH>
__global__ void __launch_bounds__(THREADS, 1)
attn_bwd_bf16_dq_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                   const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                   const __grid_constant__ BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_smem = smem_base;
  const uint32_t do_smem = q_smem + TILE_BYTES;
  const uint32_t k_ring = do_smem + TILE_BYTES;
  const uint32_t v_ring = k_ring + B_K_STAGES * TILE_BYTES;
  const uint32_t bar_base = v_ring + B_V_STAGES * TILE_BYTES;
  auto k_full = [&](int s) { return bar_base + 8u * s; };
  auto k_empty = [&](int s) { return bar_base + 8u * (B_K_STAGES + s); };
  const uint32_t v_bars = bar_base + 8u * (2 * B_K_STAGES);
  auto v_full = [&](int s) { return v_bars + 8u * s; };
  auto v_empty = [&](int s) { return v_bars + 8u * (B_V_STAGES + s); };
  const uint32_t misc = v_bars + 8u * (2 * B_V_STAGES);
  const uint32_t q_full = misc, s_full = misc + 8, s_free = misc + 16, acc_full = misc + 24;
  auto ds_full = [&](int i) { return misc + 32 + 8u * i; };  // the set's dS is in tensor memory
  auto ds_free = [&](int i) { return misc + 48 + 8u * i; };  // the product that reads it is complete
  const uint32_t tmem_slot = misc + 64;

  const int warp = threadIdx.x / 32;
  const int lane = threadIdx.x % 32;
  const int num_m = (p.Nq + BM - 1) / BM;
  const BandBlock at = band_order(blockIdx.x, num_m, p.B * p.Hq, p.q_band);
  const int hq = at.head % p.Hq;
  const int b = at.head / p.Hq;
  const int hkv = hq / (p.Hq / p.Hkv);
  const int m0 = (num_m - 1 - at.rank) * BM;  // the last query blocks see the most keys
  const int shift = p.Nk - p.Nq;
  int n_tiles = (p.Nk + BN - 1) / BN;
  if (p.causal) {
    const int last_key = min(m0 + BM, p.Nq) - 1 + shift;
    n_tiles = last_key < 0 ? 0 : min(n_tiles, last_key / BN + 1);
  }

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < B_K_STAGES; ++s) {
      mbar_init(k_full(s), 1);
      mbar_init(k_empty(s), 1);
    }
    for (int s = 0; s < B_V_STAGES; ++s) {
      mbar_init(v_full(s), 1);
      mbar_init(v_empty(s), 1);
    }
    mbar_init(s_full, 2);  // S and dP come from two threads
    mbar_init(s_free, EW_THREADS);
    for (int i = 0; i < 2; ++i) {
      mbar_init(ds_full(i), EW_THREADS);
      mbar_init(ds_free(i), 1);
    }
    mbar_init(acc_full, 1);
    mbar_fence_init();
    prefetch_tmap(&tmap_q);
    prefetch_tmap(&tmap_k);
    prefetch_tmap(&tmap_v);
    prefetch_tmap(&tmap_do);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  // The dK/dV kernel lets this one start once the prep kernel, whose results both read, has completed: no wait here
  // (pdl_load).  TMA brings in the caller's tensors only.
  pdl_launch_dependents();

  if (warp == 0) {
    if (lane == 0 && n_tiles > 0) {
      const int chunks = DH / CHUNK;
      mbar_expect_tx(q_full, 2 * chunks * CHUNK_BYTES);
      for (int c = 0; c < chunks; ++c) {
        tma_load_4d(q_smem + c * CHUNK_BYTES, &tmap_q, q_full, c * CHUNK, m0, hq, b);
        tma_load_4d(do_smem + c * CHUNK_BYTES, &tmap_do, q_full, c * CHUNK, m0, hq, b);
      }
      for (int j = 0; j < n_tiles; ++j) {
        const int vs = j % B_V_STAGES, ks = j % B_K_STAGES;
        if (!mbar_wait(k_empty(ks), ((j / B_K_STAGES) & 1) ^ 1, p.status, WK_ERR_TIMEOUT_EMPTY)) break;
        mbar_expect_tx(k_full(ks), chunks * CHUNK_BYTES);
        for (int c = 0; c < chunks; ++c)
          tma_load_4d(k_ring + ks * TILE_BYTES + c * CHUNK_BYTES, &tmap_k, k_full(ks), c * CHUNK, j * BN, hkv, b);
        if (!mbar_wait(v_empty(vs), ((j / B_V_STAGES) & 1) ^ 1, p.status, WK_ERR_TIMEOUT_EMPTY)) break;
        mbar_expect_tx(v_full(vs), chunks * CHUNK_BYTES);
        for (int c = 0; c < chunks; ++c)
          tma_load_4d(v_ring + vs * TILE_BYTES + c * CHUNK_BYTES, &tmap_v, v_full(vs), c * CHUNK, j * BN, hkv, b);
      }
    }
    __syncwarp();
  } else if (warp == 1 || warp == 2) {
    if (lane == 0 && n_tiles > 0) {
      // S = Q K^T by warp 1, dP = dO V^T by warp 2, side by side: a thread needs ~90 cycles per MMA it issues here
      const bool is_s = warp == 1;
      constexpr uint32_t idesc = make_idesc(1, 1, 0, 0, BM, BN);
      const uint32_t d_tmem = tmem_base + (is_s ? B_S_COL : B_DP_COL);
      const uint64_t a_desc = smem_desc_sw128(is_s ? q_smem : do_smem, 16, 1024);
      bool ok = mbar_wait(q_full, 0, p.status, WK_ERR_TIMEOUT_LOAD);
      for (int j = 0; ok && j < n_tiles; ++j) {
        const int s = is_s ? j % B_K_STAGES : j % B_V_STAGES;
        const uint32_t full = is_s ? k_full(s) : v_full(s);
        if (!mbar_wait(full, (is_s ? j / B_K_STAGES : j / B_V_STAGES) & 1, p.status, WK_ERR_TIMEOUT_LOAD)) break;
        if (j > 0 && !mbar_wait(s_free, (j - 1) & 1, p.status, WK_ERR_TIMEOUT_P)) break;
        tc_fence_after();
        const uint64_t b_desc = smem_desc_sw128((is_s ? k_ring : v_ring) + s * TILE_BYTES, 16, 1024);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint64_t off = (k >> 2) * (CHUNK_BYTES >> 4) + 2 * (k & 3);
          if (16 * k < DH) mma_f16_ss(d_tmem, a_desc + off, b_desc + off, idesc, k != 0);
        }
        tc_commit(s_full);
        if (!is_s) tc_commit(v_empty(s));
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    if (lane == 0 && n_tiles > 0) {
      // dQ += dS K: A = dS in tensor memory, B = the K tile read MN-major (16 keys = 2048 bytes, the head dimension's
      // two spans one chunk apart)
      const uint32_t idesc = make_idesc(1, 1, 0, 1, BM, DH);
      for (int j = 0; j < n_tiles; ++j) {
        const int s = j % B_K_STAGES, set = j & 1;
        if (!mbar_wait(k_full(s), (j / B_K_STAGES) & 1, p.status, WK_ERR_TIMEOUT_LOAD)) break;
        if (!mbar_wait(ds_full(set), (j >> 1) & 1, p.status, WK_ERR_TIMEOUT_P)) break;
        tc_fence_after();
        const uint64_t k_desc = smem_desc_sw128(k_ring + s * TILE_BYTES, CHUNK_BYTES, 1024);
#pragma unroll
        for (int k = 0; k < BN / 16; ++k)
          mma_f16_ts(tmem_base + B_DQ_COL, tmem_base + B_DS_COL + 64 * set + 8 * k, k_desc + 128 * k, idesc, (j | k) != 0);
        tc_commit(k_empty(s));
        tc_commit(ds_free(set));
        if (j + 1 == n_tiles) tc_commit(acc_full);
      }
    }
    __syncwarp();
  } else {
    const int quad = warp & 3;
    const int c = (warp - 4) >> 2;  // which block of 32 of the tile's 128 columns this thread handles
    const int r = quad * 32 + lane;
    const int row = m0 + r;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t s_tmem = tmem_base + lane_addr + B_S_COL + 32 * c;
    const uint32_t dp_tmem = tmem_base + lane_addr + B_DP_COL + 32 * c;
    const uint32_t ds_tmem = tmem_base + lane_addr + B_DS_COL + 16 * c;
    const float beta = p.softmax_scale * LOG2E;
    const float* rec = p.qstat + ((static_cast<int64_t>(b) * p.Hq + hq) * p.nq_pad + m0) * 2 + r;
    const float neg_l = pdl_load(rec), neg_d = pdl_load(rec + 128);  // -L and -D of this query
    const int row_limit = min(p.causal ? row + shift : p.Nk - 1, p.Nk - 1) - c * 32;
    bool ok = true;

    for (int j = 0; j < n_tiles; ++j) {
      if (!mbar_wait_warp(s_full, j & 1, p.status, WK_ERR_TIMEOUT_MMA)) {
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t sraw[32], draw[32];
      tmem_ld32(s_tmem, sraw);
      tmem_ld32(dp_tmem, draw);
      tc_wait_ld();
      tc_fence_before();
      mbar_arrive(s_free);
      const int limit = row_limit - j * BN;  // columns > limit are masked
      uint64_t ds[16];                       // dS of this query for 32 keys, as packed pairs
      const uint64_t beta2 = pack_f32x2(beta, beta), nl2 = pack_f32x2(neg_l, neg_l), nd2 = pack_f32x2(neg_d, neg_d);
      auto elements = [&](auto masked) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float x0, x1;
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sraw[2 * i]), __uint_as_float(sraw[2 * i + 1])), beta2, nl2),
                       x0, x1);
          float p0 = ex2_approx(x0), p1 = ex2_approx(x1);
          if (decltype(masked)::value) {
            if (2 * i > limit) p0 = 0.f;
            if (2 * i + 1 > limit) p1 = 0.f;
          }
          ds[i] = mul_f32x2(pack_f32x2(p0, p1),
                            add_f32x2(pack_f32x2(__uint_as_float(draw[2 * i]), __uint_as_float(draw[2 * i + 1])), nd2));
        }
      };
      // uniform over the CTA: does this tile contain any masked score?
      if ((j * BN + BN > p.Nk) || (p.causal && j * BN + BN - 1 > m0 + shift))
        elements(std::true_type{});
      else
        elements(std::false_type{});
      const int set = j & 1;
      if (j >= 2 && !mbar_wait_warp(ds_free(set), ((j >> 1) - 1) & 1, p.status, WK_ERR_TIMEOUT_MMA)) {
        ok = false;
        break;
      }
      tc_fence_after();
      store_block_bf16(ds, ds_tmem + 64 * set);
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(ds_full(set));
    }

    if (n_tiles > 0 && ok) ok = mbar_wait_warp(acc_full, 0, p.status, WK_ERR_TIMEOUT_MMA);
    if (ok) {
      tc_fence_after();
      const float scale = p.softmax_scale;
      __nv_bfloat16* dst_row = p.dq + ((static_cast<int64_t>(b) * p.Hq + hq) * p.Nq + row) * DH;
      {
        uint32_t v[32];
        if (n_tiles > 0) {
          tmem_ld32(tmem_base + lane_addr + B_DQ_COL + c * 32, v);
          tc_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0;
        }
        if (row < p.Nq && c * 32 < DH) {
          uint4* dst = reinterpret_cast<uint4*>(dst_row + c * 32);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(v[8 * i + 0]) * scale, __uint_as_float(v[8 * i + 1]) * scale);
            w.y = pack_bf16x2(__uint_as_float(v[8 * i + 2]) * scale, __uint_as_float(v[8 * i + 3]) * scale);
            w.z = pack_bf16x2(__uint_as_float(v[8 * i + 4]) * scale, __uint_as_float(v[8 * i + 5]) * scale);
            w.w = pack_bf16x2(__uint_as_float(v[8 * i + 6]) * scale, __uint_as_float(v[8 * i + 7]) * scale);
            dst[i] = w;
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
  if (blockIdx.x == gridDim.x - 1) pdl_wait();  // this kernel does not end before the dK/dV kernel has
}

int make_map4(CUtensorMap* m, const void* base, int d, int n, int h, int b, const int64_t* strides) {
  const uint64_t dims[4] = {static_cast<uint64_t>(d), static_cast<uint64_t>(n), static_cast<uint64_t>(h), static_cast<uint64_t>(b)};
  const uint64_t str[3] = {static_cast<uint64_t>(strides[2]) * 2, static_cast<uint64_t>(strides[1]) * 2,
                           static_cast<uint64_t>(strides[0]) * 2};
  const uint32_t box[4] = {CHUNK, 128, 1, 1};
  return encode_tmap(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, base, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace
}  // namespace wk

extern "C" int64_t wk_attn_bwd_bf16_workspace_bytes(int B, int Hq, int Nq) {
  if (B < 0 || Hq < 0 || Nq < 0) return WK_E_ARG;
  const int64_t nq_pad = (static_cast<int64_t>(Nq) + 127) / 128 * 128;
  return static_cast<int64_t>(B) * Hq * nq_pad * 16 + 256;
}

extern "C" int wk_attn_bwd_bf16(const wk_attn_bwd_args* a, void* stream) {
  using namespace wk;
  if (!a) return WK_E_ARG;
  if (a->B <= 0 || a->Hq <= 0 || a->Hkv <= 0 || a->Nq <= 0 || a->Nk <= 0 || (a->d != 128 && a->d != 64)) return WK_E_ARG;
  if (a->Hq % a->Hkv || a->B > 65535 || a->Hq > 65535) return WK_E_ARG;
  if (!a->q || !a->k || !a->v || !a->out || !a->dout || !a->lse || !a->dq || !a->dk || !a->dv) return WK_E_ARG;
  if (a->q_descale || a->k_descale || a->v_descale || !a->workspace) return WK_E_ARG;
  if (!(a->softmax_scale > 0.f)) return WK_E_ARG;
  const void* ptrs[] = {a->q, a->k, a->v, a->dout, a->dq, a->dk, a->dv, a->workspace};
  for (const void* ptr : ptrs)
    if (!aligned16(ptr)) return WK_E_ARG;
  if (reinterpret_cast<uintptr_t>(a->out) & 7) return WK_E_ARG;
  for (int i = 0; i < 3; ++i) {
    if (a->q_strides[i] % 8 || a->k_strides[i] % 8 || a->v_strides[i] % 8 || a->dout_strides[i] % 8) return WK_E_ARG;
    if (a->q_strides[i] <= 0 || a->k_strides[i] <= 0 || a->v_strides[i] <= 0 || a->dout_strides[i] <= 0)
      return WK_E_ARG;
    if (a->out_strides[i] % 4 || a->out_strides[i] <= 0) return WK_E_ARG;
  }
  if (a->workspace_bytes < wk_attn_bwd_bf16_workspace_bytes(a->B, a->Hq, a->Nq)) return WK_E_ARG;
  if (int unsupported = require_sm100()) return unsupported;
  int* status = status_word();
  if (!status) return WK_E_CUDA;
  cudaStream_t st = static_cast<cudaStream_t>(stream);

  const int nq_pad = (a->Nq + 127) / 128 * 128;
  float* qstat = static_cast<float*>(a->workspace);

  PrepParams pp;
  pp.dout = static_cast<const __nv_bfloat16*>(a->dout);
  pp.out = static_cast<const __nv_bfloat16*>(a->out);
  pp.lse = a->lse;
  pp.qstat = qstat;
  pp.do_sb = a->dout_strides[0];
  pp.do_sh = a->dout_strides[1];
  pp.do_sn = a->dout_strides[2];
  pp.o_sb = a->out_strides[0];
  pp.o_sh = a->out_strides[1];
  pp.o_sn = a->out_strides[2];
  pp.lse_sb = a->lse_strides[0];
  pp.lse_sh = a->lse_strides[1];
  pp.B = a->B;
  pp.Hq = a->Hq;
  pp.Nq = a->Nq;
  pp.nq_pad = nq_pad;
  pp.d = a->d;
  {
    const int64_t rows = static_cast<int64_t>(a->B) * a->Hq * nq_pad;
    bool wide_loads = aligned16(a->out) && aligned16(a->dout);  // 16-byte loads: rows on 16-byte boundaries
    for (int i = 0; i < 3; ++i) wide_loads = wide_loads && a->out_strides[i] % 8 == 0 && a->dout_strides[i] % 8 == 0;
    const void* kernel = wide_loads ? reinterpret_cast<const void*>(attn_bwd_bf16_prep4_kernel)
                                    : reinterpret_cast<const void*>(attn_bwd_bf16_prep_kernel);
    const int64_t blocks = wide_loads ? (rows + 31) / 32 : (rows + 7) / 8;
    if (int r = launch_pdl(kernel, dim3(static_cast<unsigned>(blocks)), 256, 0, st, 1, {&pp})) return r;
  }

  CUtensorMap tq, tk, tv, tdo;
  int r = make_map4(&tq, a->q, a->d, a->Nq, a->Hq, a->B, a->q_strides);
  if (r) return r;
  r = make_map4(&tk, a->k, a->d, a->Nk, a->Hkv, a->B, a->k_strides);
  if (r) return r;
  r = make_map4(&tv, a->v, a->d, a->Nk, a->Hkv, a->B, a->v_strides);
  if (r) return r;
  r = make_map4(&tdo, a->dout, a->d, a->Nq, a->Hq, a->B, a->dout_strides);
  if (r) return r;

  BwdParams p;
  p.qstat = qstat;
  p.dq = static_cast<__nv_bfloat16*>(a->dq);
  p.dk = static_cast<__nv_bfloat16*>(a->dk);
  p.dv = static_cast<__nv_bfloat16*>(a->dv);
  p.B = a->B;
  p.Hq = a->Hq;
  p.Hkv = a->Hkv;
  p.Nq = a->Nq;
  p.Nk = a->Nk;
  p.nq_pad = nq_pad;
  p.d = a->d;
  p.causal = a->causal;
  p.softmax_scale = a->softmax_scale;
  p.status = status;

  const int num_n = (a->Nk + BN - 1) / BN, num_m = nq_pad / BM;
  const int sms = sm_count();
  if (sms <= 0) return WK_E_CUDA;
  // q, dO, k and v of a KV head
  const int group = a->Hq / a->Hkv;
  const int64_t head_bytes = 4ll * a->d * (static_cast<int64_t>(group) * a->Nq + a->Nk);
  p.kv_band = a->causal ? band_heads(num_n, a->B * a->Hkv, head_bytes, sms) : 1;
  p.q_band = a->causal ? band_heads(num_m, a->B * a->Hq, head_bytes / group, sms) : 1;
  const bool small = a->d == 64;
  const void* dkdv = small ? reinterpret_cast<const void*>(attn_bwd_bf16_dkdv_kernel<64>)
                           : reinterpret_cast<const void*>(attn_bwd_bf16_dkdv_kernel<128>);
  const void* dq = small ? reinterpret_cast<const void*>(attn_bwd_bf16_dq_kernel<64>)
                         : reinterpret_cast<const void*>(attn_bwd_bf16_dq_kernel<128>);
  if (allow_smem(dkdv, A_SMEM_BYTES) || allow_smem(dq, B_SMEM_BYTES)) return WK_E_CUDA;
  const int64_t kv_ctas = static_cast<int64_t>(num_n) * a->Hkv * a->B, q_ctas = static_cast<int64_t>(num_m) * a->Hq * a->B;
  if (kv_ctas > INT32_MAX || q_ctas > INT32_MAX) return WK_E_ARG;
  if ((r = launch_pdl(dkdv, dim3(static_cast<unsigned>(kv_ctas)), THREADS, A_SMEM_BYTES, st, 1, {&tq, &tk, &tv, &tdo, &p})))
    return r;
  return launch_pdl(dq, dim3(static_cast<unsigned>(q_ctas)), THREADS, B_SMEM_BYTES, st, 1, {&tq, &tk, &tv, &tdo, &p});
}
