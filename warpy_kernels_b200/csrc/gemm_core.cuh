// The GEMM kernel of this library, out[M,N] = a[M,K] . b[N,K]^T with the fused epilogue of gemm_epilogue.cuh:
// 16-bit operands (tcgen05 kind::f16) and MXFP8 operands (kind::mxf8f6f4.block_scale), on single CTAs or on CTA pairs,
// with K whole or split over a cluster.  gemm_16bit.cu and gemm_mxfp8.cu instantiate it.
//
//   FORM_SINGLE  one 128 x 256 tile per SM
//   FORM_NARROW  one 128 x 128 tile per SM: twice as many tiles for problems that do not fill the SMs
//   FORM_PAIR    one 256 x 256 tile per two SMs (cta_group::2): each CTA loads its own 128 rows of A and 128 of the
//                tile's 256 rows of B, the even CTA issues the MMAs for both, each CTA's tensor memory holds its half
//                of M.  Per SM a pair moves 32 KiB into shared memory where a single CTA moves 48.
//   split K      a cluster of S CTAs (or S pairs) works on one tile, each on its own range of K; the fp32 partial
//                sums meet in distributed shared memory (each CTA adds up and stores every S-th chunk of 32 columns)
//                in the order of K, so the result does not depend on which form ran.  For problems whose tiles do not
//                fill the SMs: see gemm_plan().
//
// Warps: 0 TMA producer | 1 MMA issue | 2-9 epilogue, two per 32 rows | 10 (MXFP8) copies the scale atoms of a stage
// to tensor memory (tcgen05.cp) so that the MMA warp issues nothing but MMAs: with the three copies, two commits and
// the wait for the operands in its loop it needed more cycles per stage than the tensor pipe does (8192 x 4096 x 14336:
// 2521 -> 2750 TFLOP/s).
//
// "Full" barriers of a pair live in the even CTA and take one arrival: its producer announces the bytes of both CTAs
// and the odd CTA's loads complete against them (a remote mbarrier.arrive.expect_tx per stage held the odd producer
// for about a thousand cycles each).  All waits are bounded; cluster barriers are reached by every thread on every
// path.
#pragma once
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "host_common.h"
#include "pair.cuh"

namespace wk {

constexpr int KIND_16 = 0;  // bf16 / fp16
constexpr int KIND_MX = 1;  // e4m3 with a ue8m0 scale per row and 32 K

constexpr int FORM_SINGLE = 0, FORM_NARROW = 1, FORM_PAIR = 2;
constexpr int SF_ATOM = 512;  // scale bytes of 128 rows x 128 K

struct TileCoord {
  int m_blk, n_blk;
};
// Tiles in groups of `group_m` rows of tiles, M fastest inside a group (the reference's order,
// warpy_kernels/utils/sched.py:8-16): the CTAs that run at the same time share their operand rows in L2.
__device__ __forceinline__ TileCoord tile_coord(int tile, int num_m, int num_n, int group_m) {
  const int per_group = group_m * num_n;
  const int g = tile / per_group;
  const int first_m = g * group_m;
  const int gsz = min(group_m, num_m - first_m);
  const int local = tile - g * per_group;
  TileCoord c;
  c.m_blk = first_m + local % gsz;
  c.n_blk = local / gsz;
  return c;
}

struct GemmParams {
  void* out;
  Epilogue epi;
  int M, N;
  int num_kb;   // K blocks of 128 bytes
  int group_m;
  int splits;   // ranges of K = pairs or CTAs of a cluster (SPLIT kernels)
  int in_f16;   // KIND_16: fp16 instead of bf16
  int a_trans, b_trans;
  int* status;
};

template <int KIND, int FORM>
struct GemmCfg {
  static constexpr bool PAIR = FORM == FORM_PAIR;
  static constexpr int BM = PAIR ? 256 : 128;
  static constexpr int BN = FORM == FORM_NARROW ? 128 : 256;
  static constexpr int B_ROWS = FORM == FORM_SINGLE ? 256 : 128;  // rows of B this CTA loads
  static constexpr int A_BYTES = 128 * 128;                       // a stage is 128 bytes of K: one swizzle span per row
  static constexpr int B_BYTES = B_ROWS * 128;
  static constexpr int AB_BYTES = A_BYTES + B_BYTES;
  // scale atoms of a stage: this CTA's 128 rows of A and all columns of the tile
  static constexpr int SF_ATOMS = KIND == KIND_MX ? 1 + BN / 128 : 0;
  static constexpr int SF_BYTES = SF_ATOMS * SF_ATOM;
  static constexpr int STAGES = FORM == FORM_SINGLE ? 4 : FORM == FORM_NARROW ? (KIND == KIND_MX ? 4 : 5) : 6;
  static constexpr int BK = KIND == KIND_MX ? 128 : 64;  // elements
  static constexpr int T_CHUNK = 64 * 64 * 2;            // 64 K lines x 64 rows of a transposed 16-bit operand
  static constexpr int EPI_WARPS = 8;
  static constexpr int THREADS = 32 * (2 + EPI_WARPS + (KIND == KIND_MX ? 1 : 0));
  // Partial sums of the other splits: chunks of 128 rows x 32 columns.  The narrow form has room for them beside the
  // ring (48 KiB: S = 2 and 4); a pair puts them into the ring, which is idle once every CTA's products are complete.
  static constexpr int CHUNK_BYTES = 128 * 32 * 4;
  static constexpr int RECV_BYTES = FORM == FORM_NARROW ? 3 * CHUNK_BYTES : 0;
  static constexpr int SMEM = STAGES * (AB_BYTES + SF_BYTES) + RECV_BYTES + EPI_WARPS * EPI_STAGE_BYTES +
                              1024 /* alignment slack */ + 256 /* barriers */;
  static_assert(SMEM <= 227 * 1024, "shared memory of a CTA");
  // Tensor memory: two accumulators.  Two of 256 columns with scale factors share 64 columns ([0, 256) and
  // [192, 448)) and the epilogue drains those first.
  static constexpr bool OVERLAP = KIND == KIND_MX && BN == 256;
  static constexpr int ACC_STRIDE = OVERLAP ? 192 : BN;
  static constexpr int SF_COL = 448;
  static constexpr int SF_SLOTS = 4;
  static constexpr int SF_SLOT_COLS = 12;  // 4 (A: 128 rows) + 8 (B: 256 columns)
};

__device__ __forceinline__ void mma_mxf8_ss_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                 uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], %1, %2, %3, [%4], "
      "[%5], p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(sfa_tmem), "r"(sfb_tmem), "r"(accumulate)
      : "memory");
}
// 32 rows x 16 bytes of shared memory to four 32-lane groups of tensor memory, in both CTAs of the pair
__device__ __forceinline__ void tmem_cp_32x128b_warpx4_pair(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}

template <int KIND, int FORM, bool SPLIT>
__global__ void __launch_bounds__(GemmCfg<KIND, FORM>::THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
            const __grid_constant__ CUtensorMap tmap_sfa, const __grid_constant__ CUtensorMap tmap_sfb,
            const __grid_constant__ CUtensorMap tmap_out, const __grid_constant__ CUtensorMap tmap_pre,
            const __grid_constant__ GemmParams p) {
  using C = GemmCfg<KIND, FORM>;
  constexpr bool PAIR = C::PAIR;
  constexpr bool MX = KIND == KIND_MX;
  constexpr int STAGES = C::STAGES, CHUNKS = C::BN / 32;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sf_base = smem_base + STAGES * C::AB_BYTES;
  const uint32_t recv_base = C::RECV_BYTES ? sf_base + STAGES * C::SF_BYTES : smem_base;
  const uint32_t epi_base = sf_base + STAGES * C::SF_BYTES + C::RECV_BYTES;
  const uint32_t bar_base = epi_base + C::EPI_WARPS * EPI_STAGE_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  const uint32_t ovl_bar = bar_base + 8u * (2 * STAGES + 4);  // the columns shared with the next tile are drained
  auto sf_bar = [&](int i) { return bar_base + 8u * (2 * STAGES + 5 + i); };  // scale slot i is in tensor memory
  const uint32_t tmem_slot = bar_base + 8u * (2 * STAGES + 5 + C::SF_SLOTS);

  const int warp = threadIdx.x / 32;
  const int lane = threadIdx.x % 32;
  constexpr bool CLUSTER = PAIR || SPLIT;
  const uint32_t rank = CLUSTER ? cluster_ctarank() : 0;
  const uint32_t half = PAIR ? rank & 1 : 0;        // this CTA's half of the tile's rows; half 0 issues the MMAs
  const uint32_t leader = PAIR ? rank & ~1u : rank;
  const uint32_t split = SPLIT ? (PAIR ? rank >> 1 : rank) : 0;
  const int splits = SPLIT ? p.splits : 1;
  const int per_cluster = (PAIR ? 2 : 1) * splits;
  const int first_tile = blockIdx.x / per_cluster, tile_step = gridDim.x / per_cluster;
  const int num_m = (p.M + C::BM - 1) / C::BM;  // M and N are multiples of 128: the last tile may be half outside,
  const int num_n = (p.N + C::BN - 1) / C::BN;  // where the loads read zeros and the epilogue stores nothing
  const int num_tiles = num_m * num_n;
  // this CTA's range of K blocks
  const int kb0 = static_cast<int>(static_cast<int64_t>(p.num_kb) * split / splits);
  const int num_kb = static_cast<int>(static_cast<int64_t>(p.num_kb) * (split + 1) / splits) - kb0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), (PAIR ? 2 : 1) * C::EPI_WARPS);
    }
    mbar_init(ovl_bar, (PAIR ? 2 : 1) * C::EPI_WARPS / 2);  // the warps that drain the shared columns
    for (int i = 0; i < C::SF_SLOTS; ++i) mbar_init(sf_bar(i), 1);
    mbar_fence_init();
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
    if (MX) {
      prefetch_tmap(&tmap_sfa);
      prefetch_tmap(&tmap_sfb);
    }
  }
  if (warp == 1) {
    if (PAIR) {
      tmem_alloc_pair(tmem_slot, 512);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, 512);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR)
    cluster_sync();  // the other CTA's barriers are initialised before anybody signals them
  else if (SPLIT)
    cluster_arrive();  // waited for before the first partial sums are sent
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  // The next kernel of the stream may be set up beside this one from here on (tensor memory is taken), and nothing of
  // the one before is read or overwritten before it has completed.
  pdl_launch_dependents();
  pdl_wait();

  int stage = 0;       // ring position and parity of this warp's role
  uint32_t phase = 0;
  int slot = 0;        // scale slot, likewise
  uint32_t slot_phase = 0;
  auto next_stage = [&]() {
    if (++stage == STAGES) {
      stage = 0;
      phase ^= 1;
    }
  };
  auto next_slot = [&]() {
    if (++slot == C::SF_SLOTS) {
      slot = 0;
      slot_phase ^= 1;
    }
  };

  // ---- the roles' work on one tile ------------------------------------------------------------------------------
  auto produce = [&](const TileCoord& tc) -> bool {
    const int a_row = tc.m_blk * C::BM + 128 * half, b_row = tc.n_blk * C::BN + (PAIR ? 128 * half : 0);
    for (int i = 0; i < num_kb; ++i) {
      const int kb = kb0 + i;
      if (!mbar_wait(empty_bar(stage), phase ^ 1, p.status, WK_ERR_TIMEOUT_EMPTY)) return false;
      const uint32_t sa = smem_base + stage * C::AB_BYTES;
      const uint32_t sb = sa + C::A_BYTES;
      const uint32_t full = PAIR ? mapa(full_bar(stage), leader) : full_bar(stage);
      // scale atoms of columns beyond N are not announced by a single CTA and read as zeros by a pair
      const int sf_b = PAIR ? 2 : min(C::BN / 128, p.N / 128 - tc.n_blk * (C::BN / 128));
      // a pair's other bytes may land before this announcement: the count just goes negative meanwhile
      if (half == 0)
        mbar_expect_tx(full_bar(stage), (PAIR ? 2 : 1) * (C::AB_BYTES + (MX ? (1 + sf_b) * SF_ATOM : 0)));
      auto load = [&](uint32_t dst, const CUtensorMap* m, int x, int y) {
        if (PAIR)
          tma_load_2d_pair(dst, m, full, x, y);
        else
          tma_load_2d(dst, m, full, x, y);
      };
      // An operand stored [rows, K] arrives as one box of its rows x 128 bytes of K (K-major tile).  A transposed one,
      // stored [K, rows], arrives as boxes of 64 K lines x 64 rows (128 bytes of rows per line), 8 KiB apart.
      if (!MX && p.a_trans) {
#pragma unroll
        for (int c = 0; c < 2; ++c) load(sa + c * C::T_CHUNK, &tmap_a, a_row + 64 * c, kb * C::BK);
      } else {
        load(sa, &tmap_a, kb * C::BK, a_row);
      }
      if (!MX && p.b_trans) {
#pragma unroll
        for (int c = 0; c < C::B_ROWS / 64; ++c) load(sb + c * C::T_CHUNK, &tmap_b, b_row + 64 * c, kb * C::BK);
      } else {
        load(sb, &tmap_b, kb * C::BK, b_row);
      }
      if (MX) {
        const uint32_t ssf = sf_base + stage * C::SF_BYTES;
        auto load_sf = [&](uint32_t dst, const CUtensorMap* m, int row_blk) {
          if (PAIR)
            tma_load_3d_pair(dst, m, full, 0, kb, row_blk);
          else
            tma_load_3d(dst, m, full, 0, kb, row_blk);
        };
        load_sf(ssf, &tmap_sfa, a_row / 128);
        for (int c = 0; c < sf_b; ++c) load_sf(ssf + (1 + c) * SF_ATOM, &tmap_sfb, tc.n_blk * (C::BN / 128) + c);
      }
      next_stage();
    }
    return true;
  };

  // Scale atoms of a stage, shared memory -> tensor memory slot; the slot's last readers were the MMAs of four K
  // blocks back, whose stage is empty by then.
  int cp_back_stage = 0;
  uint32_t cp_back_phase = 0;
  int cp_count = 0;
  auto copy_scales = [&](bool mine) -> bool {
    for (int i = 0; i < num_kb; ++i) {
      if (!mbar_wait_warp(full_bar(stage), phase, p.status, WK_ERR_TIMEOUT_LOAD)) return false;
      if (cp_count >= C::SF_SLOTS) {
        if (!mbar_wait_warp(empty_bar(cp_back_stage), cp_back_phase, p.status, WK_ERR_TIMEOUT_EMPTY)) return false;
        if (++cp_back_stage == STAGES) {
          cp_back_stage = 0;
          cp_back_phase ^= 1;
        }
      } else {
        ++cp_count;
      }
      tc_fence_after();
      if (mine) {
        const uint64_t sf_desc = smem_desc_plain(sf_base + stage * C::SF_BYTES, 16, 128);
        const uint32_t sf_tmem = tmem_base + C::SF_COL + slot * C::SF_SLOT_COLS;
#pragma unroll
        for (int c = 0; c < C::SF_ATOMS; ++c) {
          if (PAIR)
            tmem_cp_32x128b_warpx4_pair(sf_tmem + 4 * c, sf_desc + c * (SF_ATOM / 16));
          else
            tmem_cp_32x128b_warpx4(sf_tmem + 4 * c, sf_desc + c * (SF_ATOM / 16));
        }
        if (PAIR)
          tc_commit_pair(mapa(sf_bar(slot), leader));
        else
          tc_commit(sf_bar(slot));
      }
      next_stage();
      next_slot();
    }
    return true;
  };

  const uint16_t pair_mask = static_cast<uint16_t>(3u << leader);
  auto commit = [&](uint32_t bar) {  // arrives on the barrier of every CTA that works on the tile part
    if (PAIR)
      tc_commit_pair_multicast(bar, pair_mask);
    else
      tc_commit(bar);
  };
  // All lanes wait, one elected lane issues: from a converged warp an MMA costs its issuer 75 cycles instead of 95.
  const uint32_t idesc16 = make_idesc(p.in_f16 ? 0 : 1, p.in_f16 ? 0 : 1, p.a_trans ? 1 : 0, p.b_trans ? 1 : 0, C::BM,
                                      C::BN);
  const uint64_t a_desc0 = smem_desc_sw128(smem_base, !MX && p.a_trans ? C::T_CHUNK : 16, 1024);
  const uint64_t b_desc0 = smem_desc_sw128(smem_base + C::A_BYTES, !MX && p.b_trans ? C::T_CHUNK : 16, 1024);
  // K-major: 32 bytes of K further along the row; MN-major: 16 K lines of 128 bytes further on
  const uint32_t a_kstep = !MX && p.a_trans ? 2048 / 16 : 2, b_kstep = !MX && p.b_trans ? 2048 / 16 : 2;
  auto multiply = [&](uint32_t d_tmem, int acc, bool mine) -> bool {
    for (int i = 0; i < num_kb; ++i) {
      if (!(MX ? mbar_wait_warp(sf_bar(slot), slot_phase, p.status, WK_ERR_TIMEOUT_LOAD)
               : mbar_wait_warp(full_bar(stage), phase, p.status, WK_ERR_TIMEOUT_LOAD)))
        return false;
      tc_fence_after();
      if (mine) {
        const uint64_t step = static_cast<uint64_t>(stage) * (C::AB_BYTES / 16);
        const uint32_t sf_tmem = tmem_base + C::SF_COL + slot * C::SF_SLOT_COLS;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint64_t da = a_desc0 + step + k * a_kstep, db = b_desc0 + step + k * b_kstep;
          const uint32_t add = (i | k) != 0;
          if (MX && PAIR)
            mma_mxf8_ss_pair(d_tmem, da, db, make_idesc_mx(C::BM, C::BN, k, k), sf_tmem, sf_tmem + 4, add);
          else if (MX)
            mma_mxf8_ss(d_tmem, da, db, make_idesc_mx(C::BM, C::BN, k, k), sf_tmem, sf_tmem + 4, add);
          else if (PAIR)
            mma_f16_ss_pair(d_tmem, da, db, idesc16, add);
          else
            mma_f16_ss(d_tmem, da, db, idesc16, add);
        }
        commit(empty_bar(stage));
        if (i == num_kb - 1) commit(tfull_bar(acc));
      }
      next_stage();
      next_slot();
    }
    return true;
  };

  const int quad = warp & 3;       // TMEM lanes [32 quad, 32 quad + 32) are visible to this warp
  const int side = (warp - 2) >> 2;  // which of the two epilogue warps of these rows
  const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
  const bool is_epilogue = warp >= 2 && warp < 2 + C::EPI_WARPS;
  EpilogueTarget target = {&tmap_out, &tmap_pre, epi_base + (warp - 2) * EPI_STAGE_BYTES, lane, 0};

  if (!SPLIT) {
    if (warp == 0) {
      if (lane == 0)
        for (int tile = first_tile; tile < num_tiles; tile += tile_step)
          if (!produce(tile_coord(tile, num_m, num_n, p.group_m))) break;
      __syncwarp();
    } else if (warp == 1) {
      if (half == 0) {
        const bool mine = elect_one();
        int local = 0;
        for (int tile = first_tile; tile < num_tiles; tile += tile_step, ++local) {
          const int acc = local & 1;
          // this accumulator was drained two tiles ago, and the previous tile has given up the columns it shares
          auto wait = [&](uint32_t bar, uint32_t parity) {
            const bool ok = PAIR ? mbar_wait_cluster(bar, parity, p.status, WK_ERR_TIMEOUT_TMEM)
                                 : mbar_wait(bar, parity, p.status, WK_ERR_TIMEOUT_TMEM);
            return static_cast<bool>(__all_sync(0xffffffffu, ok));
          };
          if (!wait(tempty_bar(acc), ((local >> 1) & 1) ^ 1)) break;
          if (C::OVERLAP && local > 0 && !wait(ovl_bar, (local - 1) & 1)) break;
          tc_fence_after();
          if (!multiply(tmem_base + acc * C::ACC_STRIDE, acc, mine)) break;
        }
      }
    } else if (is_epilogue) {
      int local = 0;
      for (int tile = first_tile; tile < num_tiles; tile += tile_step, ++local) {
        const TileCoord tc = tile_coord(tile, num_m, num_n, p.group_m);
        const int acc = local & 1;
        target.row0 = tc.m_blk * C::BM + 128 * half + quad * 32;
        const bool row_ok = target.row0 < p.M;  // the same for the whole CTA
        const float row_scale = row_ok ? epilogue_row_scale(p.epi, target.row0 + lane) : 0.f;
        if (!mbar_wait_warp(tfull_bar(acc), (local >> 1) & 1, p.status, WK_ERR_TIMEOUT_MMA)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + lane_addr + acc * C::ACC_STRIDE;
        auto drained = [&](uint32_t bar) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if (PAIR)
              mbar_arrive_cluster(mapa(bar, leader));
            else
              mbar_arrive(bar);
          }
        };
        // Pairs of chunks in the order they are drained, the 64 columns shared with the other accumulator first; the
        // two warps of a row take turns.
        const int first_chunk = C::OVERLAP && acc == 0 ? 6 : 0;
        const bool another = tile + tile_step < num_tiles;  // a remote arrival that nobody needs costs 1500 cycles
#pragma unroll 1
        for (int i = 2 * side; i < CHUNKS; i += 4) {
          const int c = (i + first_chunk) & (CHUNKS - 1);
          const int col = tc.n_blk * C::BN + c * 32;
          const bool store = row_ok && col < p.N;  // N is a multiple of 128: both chunks or none
          uint32_t v[2][32];
          if (store) {
            tmem_ld32(d_tmem + c * 32, v[0]);
            tmem_ld32(d_tmem + c * 32 + 32, v[1]);
            tc_wait_ld();
          }
          // the shared chunks are in registers (or not wanted): the next tile's main loop may overwrite them
          if (C::OVERLAP && i == 0 && another) drained(ovl_bar);
          if (i + 4 >= CHUNKS && another) drained(tempty_bar(acc));
          if (store) {
            epilogue_chunk(p.epi, target, v[0], row_scale, col, p.N, p.out);
            epilogue_chunk(p.epi, target, v[1], row_scale, col + 32, p.N, p.out);
          }
        }
      }
    } else if (MX) {
      if (half == 0) {
        const bool mine = elect_one();
        for (int tile = first_tile; tile < num_tiles; tile += tile_step)
          if (!copy_scales(mine)) break;
      }
    }
  } else {
    // One tile at a time.
    const bool mine = !is_epilogue && elect_one();
    int local = 0;
    for (int tile = first_tile; tile < num_tiles; tile += tile_step, ++local) {
      const TileCoord tc = tile_coord(tile, num_m, num_n, p.group_m);
      target.row0 = tc.m_blk * C::BM + 128 * half + quad * 32;
      const bool active = is_epilogue && target.row0 < p.M;
      if (warp == 0) {
        if (lane == 0) produce(tc);
      } else if (warp == 1) {
        if (half == 0) multiply(tmem_base, 0, mine);
      } else if (is_epilogue) {
        mbar_wait_warp(tfull_bar(0), local & 1, p.status, WK_ERR_TIMEOUT_MMA);
      } else {
        if (half == 0) copy_scales(mine);
      }
      __syncwarp();
      tc_fence_before();
      if (PAIR)
        cluster_sync();  // every CTA's products are complete: nobody reads or fills a ring
      else
        cluster_wait();  // every CTA has read the partial sums of the tile before (or has started)
      tc_fence_after();
      // Chunk c of 32 columns belongs to split c % S.  A CTA keeps the others' sums of its chunks in slots of 16 KiB,
      // [source][chunk / S], each as eight planes of 128 rows x 16 bytes.
      const int per_owner = (CHUNKS + splits - 1) / splits;
      const int me = static_cast<int>(split);
      auto slot_addr = [&](int source, int owner, int c) {
        const int s = source - (source > owner);
        return recv_base + static_cast<uint32_t>((s * per_owner + c / splits) * C::CHUNK_BYTES) +
               static_cast<uint32_t>(quad * 32 + lane) * 16;
      };
      if (active) {
        // The owner that follows this split first: if all CTAs sent to the same one at the same time, its incoming
        // link would be the bottleneck (15 instead of 30 bytes per cycle and SM).
        int turn = 0;
#pragma unroll 1
        for (int t = 1; t < splits; ++t) {
          const int owner = (me + t) % splits;
#pragma unroll 1
          for (int c = owner; c < CHUNKS; c += splits, turn ^= 1) {
            if (turn != side || tc.n_blk * C::BN + c * 32 >= p.N) continue;
            uint32_t v[32];
            tmem_ld32(tmem_base + lane_addr + c * 32, v);
            tc_wait_ld();
            const uint32_t dst = mapa(slot_addr(me, owner, c), PAIR ? 2 * owner + half : owner);
#pragma unroll
            for (int j = 0; j < 8; ++j)
              st_cluster_v4(dst + j * (128 * 16), v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          }
        }
      }
      __syncwarp();
      cluster_sync();  // all partial sums have arrived
      if (active) {
        const float row_scale = epilogue_row_scale(p.epi, target.row0 + lane);
#pragma unroll 1
        for (int c = me + side * splits; c < CHUNKS; c += 2 * splits) {
          const int col = tc.n_blk * C::BN + c * 32;
          if (col >= p.N) break;
          uint32_t own[32];
          tmem_ld32(tmem_base + lane_addr + c * 32, own);
          tc_wait_ld();
          float sum[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) sum[i] = 0.f;
#pragma unroll 1
          for (int s = 0; s < splits; ++s) {  // in the order of K, whichever CTA adds up
            if (s == me) {
#pragma unroll
              for (int i = 0; i < 32; ++i) sum[i] += __uint_as_float(own[i]);
            } else {
              const uint32_t src = slot_addr(s, me, c);
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                float x, y, z, w;
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(x), "=f"(y), "=f"(z), "=f"(w)
                             : "r"(src + j * (128 * 16)));
                sum[4 * j] += x;
                sum[4 * j + 1] += y;
                sum[4 * j + 2] += z;
                sum[4 * j + 3] += w;
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) own[i] = __float_as_uint(sum[i]);
          epilogue_chunk(p.epi, target, own, row_scale, col, p.N, p.out);
        }
      }
      __syncwarp();
      // a pair's ring: the next tile's TMA writes (async proxy) and MMAs follow these reads
      fence_proxy_async_smem();
      tc_fence_before();
      __syncthreads();
      tc_fence_after();
      if (!PAIR && tile + tile_step < num_tiles) cluster_arrive();
    }
  }

  if (is_epilogue && lane == 0) bulk_wait_all();
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();  // nobody leaves while the other CTA may still signal this one's barriers
  if (warp == 1) {
    tc_fence_after();
    if (PAIR)
      tmem_dealloc_pair(tmem_base, 512);
    else
      tmem_dealloc(tmem_base, 512);
  }
}

// ---- host side --------------------------------------------------------------------------------------------------
struct GemmPlan {
  int form, splits;
};

// How a problem of `num_kb` K blocks is worked on by `sms` SMs.  `force`: 0 free, 1 pairs, 2 single CTAs; the number of
// splits is that of the free choice either way, so the results have the same bits.
//
// The model counts cycles: what a K block takes (the MMAs' time or the loads', whichever is longer), what a round of
// tiles costs besides (first loads, epilogue) and what the exchange of partial sums adds.  Clusters of more than two
// CTAs do not use all SMs: 45, 33, 22 and 15 clusters of 3, 4, 6 and 8 CTAs run at once on 148.  Over 39 shapes from
// 128 x 640 x 2048 to 4096 x 2048 x 8192, bf16 and MXFP8, its choice is within 4 % of the best form but for one; a
// single 128 x 256 CTA was never ahead of a pair or of narrow tiles by more than 1 %, so it runs on request only.
inline GemmPlan gemm_plan(int m, int n, int num_kb, int sms, int force) {
  GemmPlan best = {FORM_PAIR, 1};
  double best_cycles = 1e30;
  auto consider = [&](int form, int s, double per_kb, double per_round, double once) {
    if (s > 1 && num_kb < 4 * s) return;  // a range of less than four K blocks is all start-up
    const int bm = form == FORM_PAIR ? 256 : 128, bn = form == FORM_NARROW ? 128 : 256;
    const int64_t tiles = static_cast<int64_t>((m + bm - 1) / bm) * ((n + bn - 1) / bn);
    const int cluster = (form == FORM_PAIR ? 2 : 1) * s;
    const double used = cluster <= 2 ? 1.0 : cluster <= 6 ? 0.9 : 0.82;
    const int64_t at_once = static_cast<int64_t>(sms * used) / cluster;
    if (at_once < 1) return;
    const int64_t rounds = (tiles + at_once - 1) / at_once;
    const double cycles = once + rounds * ((num_kb + s - 1) / s * per_kb + per_round);
    if (cycles < best_cycles) {
      best_cycles = cycles;
      best = {form, s};
    }
  };
  consider(FORM_NARROW, 1, 400, 1500, 3500);
  consider(FORM_NARROW, 2, 400, 4500, 4500);
  consider(FORM_NARROW, 4, 400, 5000, 4500);
  consider(FORM_PAIR, 1, 535, 1500, 4500);
  consider(FORM_PAIR, 2, 535, 5500, 6500);
  consider(FORM_PAIR, 4, 535, 5500, 6500);
  if (force == 1) best.form = FORM_PAIR;
  if (force == 2 && best.form == FORM_PAIR) best.form = best.splits > 1 ? FORM_NARROW : FORM_SINGLE;
  return best;
}

template <int KIND, int FORM, bool SPLIT>
int launch_gemm_form(CUtensorMap (&maps)[6], GemmParams& p, cudaStream_t stream) {
  using C = GemmCfg<KIND, FORM>;
  const void* fn = reinterpret_cast<const void*>(gemm_kernel<KIND, FORM, SPLIT>);
  const int per_cluster = (C::PAIR ? 2 : 1) * (SPLIT ? p.splits : 1);
  if (allow_smem(fn, C::SMEM)) return WK_E_CUDA;
  const int clusters = clusters_at_once(fn, per_cluster, C::THREADS, C::SMEM);
  if (clusters <= 0) return WK_E_CUDA;
  const int64_t tiles = static_cast<int64_t>((p.M + C::BM - 1) / C::BM) * ((p.N + C::BN - 1) / C::BN);
  if (tiles > INT32_MAX) return WK_E_ARG;
  const int grid = static_cast<int>(tiles < clusters ? tiles : clusters) * per_cluster;
  return launch_pdl(fn, dim3(grid), C::THREADS, C::SMEM, stream, per_cluster,
                    {&maps[0], &maps[1], &maps[2], &maps[3], &maps[4], &maps[5], &p});
}

// Tensor map of an operand: [rows, K] in boxes of `box_rows` x 128 bytes of K, or (16-bit, transposed) [K, rows] in
// boxes of 64 K lines x 64 rows.
template <int KIND>
int encode_operand(CUtensorMap* t, const void* ptr, int rows, int k, int box_rows, bool trans, bool f16) {
  constexpr int SIZE = KIND == KIND_MX ? 1 : 2;
  const CUtensorMapDataType dt = KIND == KIND_MX ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                 : f16           ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                                 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const int inner = trans ? rows : k, outer = trans ? k : rows;
  const uint64_t dims[2] = {static_cast<uint64_t>(inner), static_cast<uint64_t>(outer)};
  const uint64_t strides[1] = {static_cast<uint64_t>(inner) * SIZE};
  const uint32_t box[2] = {128 / SIZE, static_cast<uint32_t>(trans ? 64 : box_rows)};
  return encode_tmap(t, dt, 2, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

// p is complete but for num_kb and splits.  sfa, sfb: re-tiled scale factors (KIND_MX).
template <int KIND>
int launch_gemm(const void* a, const void* b, const uint8_t* sfa, const uint8_t* sfb, int k, int cta_pair, GemmParams& p,
                cudaStream_t stream) {
  constexpr int BK = GemmCfg<KIND, FORM_SINGLE>::BK;
  const int sms = sm_count();
  if (sms < 2) return WK_E_CUDA;
  p.num_kb = k / BK;
  const GemmPlan plan = gemm_plan(p.M, p.N, p.num_kb, sms, cta_pair);
  p.splits = plan.splits;
  CUtensorMap maps[6];  // a, b, scales of a, scales of b, out, pre
  if (int r = encode_operand<KIND>(&maps[0], a, p.M, k, 128, p.a_trans, p.in_f16)) return r;
  if (int r = encode_operand<KIND>(&maps[1], b, p.N, k, plan.form == FORM_SINGLE ? 256 : 128, p.b_trans, p.in_f16))
    return r;
  if (KIND == KIND_MX) {
    // [rows / 128][K / 128] lines of 512 bytes (128 32-bit words)
    auto encode_sf = [&](CUtensorMap* t, const uint8_t* ptr, int rows) {
      const uint64_t kb = static_cast<uint64_t>(p.num_kb);
      const uint64_t dims[3] = {SF_ATOM / 4, kb, static_cast<uint64_t>(rows / 128)};
      const uint64_t strides[2] = {SF_ATOM, SF_ATOM * kb};
      const uint32_t box[3] = {SF_ATOM / 4, 1, 1};
      return encode_tmap(t, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
    };
    if (int r = encode_sf(&maps[2], sfa, p.M)) return r;
    if (int r = encode_sf(&maps[3], sfb, p.N)) return r;
  } else {
    maps[2] = maps[3] = maps[0];  // not read
  }
  auto encode_output = [&](CUtensorMap* t, const void* ptr) {
    const uint64_t dims[2] = {static_cast<uint64_t>(p.N), static_cast<uint64_t>(p.M)};
    const uint64_t strides[1] = {static_cast<uint64_t>(p.N) * 2};
    const uint32_t box[2] = {32, 32};
    return encode_tmap(t, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B);
  };
  if (int r = encode_output(&maps[4], p.out)) return r;
  maps[5] = maps[4];
  if (p.epi.pre_out)
    if (int r = encode_output(&maps[5], p.epi.pre_out)) return r;
  const bool split = plan.splits > 1;
  switch (plan.form) {
    case FORM_PAIR:
      return split ? launch_gemm_form<KIND, FORM_PAIR, true>(maps, p, stream)
                   : launch_gemm_form<KIND, FORM_PAIR, false>(maps, p, stream);
    case FORM_NARROW:
      return split ? launch_gemm_form<KIND, FORM_NARROW, true>(maps, p, stream)
                   : launch_gemm_form<KIND, FORM_NARROW, false>(maps, p, stream);
    default:
      return launch_gemm_form<KIND, FORM_SINGLE, false>(maps, p, stream);
  }
}

}  // namespace wk
