// MXFP8 block-scaled GEMM for sm_100a: re-tiling of the scale factors and the C ABI entry points over the kernel in
// gemm_core.cuh.
//   out[M,N] = alpha . (a8 . 2^(sa-127)) . (b8 . 2^(sb-127))^T      bf16 output, fp32 accumulation
// a8 [M,K], b8 [N,K] e4m3; sa [M,K/32], sb [N,K/32] ue8m0 bytes (one per row and 32 elements along K); either scale
// tensor may be absent (unit scales).  Optionally the fp32 results are also written as MXFP8 (codes + scale byte per
// 32 columns) before they are rounded to bf16.
//
// retile_scales_kernel turns the row-major scale bytes into the 512-byte atoms tcgen05.mma reads them in (128 rows x
// 4 K-blocks: byte offset (row % 32) * 16 + (row / 32 % 4) * 4 + kblock % 4), one atom per 128 rows and 128 K elements,
// atoms ordered [row block][K block].
//
// Arithmetic follows the reference's block-scaled path (warpy_kernels/gemm/sm120.py:121-146: e4m3 products scaled by
// 2^(sfa-127) per row and 32-element K block, fp32 accumulate) and its MX output epilogue
// (warpy_kernels/gemm/sm89.py:65-93).
//
// Tensor-core bound: 2*M*N*K flops per launch.
#include "gemm_core.cuh"

namespace wk {
namespace {

// ---------------------------------------------------------------------------
// scale re-tiling
// ---------------------------------------------------------------------------
struct ScaleTensor {
  const uint8_t* src;  // [rows, 4 num_kb] bytes, or null for unit scales
  uint8_t* dst;        // atoms
  int row_blocks;      // of 128 rows
};

// One warp takes 128 rows x 4 K blocks: lane l reads the 16 scale bytes of rows l, l + 32, l + 64 and l + 96 and writes
// their 16 bytes of each of four atoms, 2 KiB in a row per warp.  Both tensors of a product go in one launch.
constexpr int RETILE_THREADS = 256;
__global__ void __launch_bounds__(RETILE_THREADS)
retile_scales_kernel(const ScaleTensor a, const ScaleTensor b, int num_kb) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x % 32;
  const int groups = (num_kb + 3) / 4;
  int64_t task = static_cast<int64_t>(blockIdx.x) * (RETILE_THREADS / 32) + threadIdx.x / 32;
  const int64_t tasks_a = static_cast<int64_t>(a.row_blocks) * groups;
  const bool second = task >= tasks_a;
  if (second) task -= tasks_a;
  const ScaleTensor& t = second ? b : a;
  if (task >= static_cast<int64_t>(t.row_blocks) * groups) return;
  const int rb = static_cast<int>(task / groups), kb = static_cast<int>(task % groups) * 4;
  const int kbs = min(4, num_kb - kb);
  uint32_t w[4][4];  // [row quarter][K block]
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint8_t* src = t.src + (static_cast<int64_t>(rb) * 128 + 32 * j + lane) * num_kb * 4 + kb * 4;
    if (t.src && (num_kb & 3) == 0 && (reinterpret_cast<uintptr_t>(t.src) & 15) == 0) {
      const uint4 v = *reinterpret_cast<const uint4*>(src);
      w[j][0] = v.x, w[j][1] = v.y, w[j][2] = v.z, w[j][3] = v.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        w[j][i] = t.src && i < kbs ? *reinterpret_cast<const uint32_t*>(src + 4 * i) : 0x7f7f7f7fu;
    }
  }
  uint4* dst = reinterpret_cast<uint4*>(t.dst + (static_cast<int64_t>(rb) * num_kb + kb) * SF_ATOM) + lane;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (i < kbs) dst[i * (SF_ATOM / 16)] = make_uint4(w[0][i], w[1][i], w[2][i], w[3][i]);
}

int retile(const ScaleTensor& a, const ScaleTensor& b, int k, cudaStream_t st) {
  int num_kb = k / 128;
  const int64_t tasks = static_cast<int64_t>(a.row_blocks + b.row_blocks) * ((num_kb + 3) / 4);
  if (tasks == 0) return 0;
  const int64_t blocks = (tasks + RETILE_THREADS / 32 - 1) / (RETILE_THREADS / 32);
  if (blocks > INT32_MAX) return WK_E_ARG;
  return launch_pdl(reinterpret_cast<const void*>(retile_scales_kernel), dim3(static_cast<unsigned>(blocks)),
                    RETILE_THREADS, 0, st, 1,
                    {const_cast<ScaleTensor*>(&a), const_cast<ScaleTensor*>(&b), &num_kb});
}

Epilogue epilogue_of(const wk_gemm_mx_args* a) {
  Epilogue e;
  e.scale_a = a->scale_a;
  e.scale_b = a->scale_b;
  e.scale_a_rows = a->scale_a_rows;
  e.scale_b_cols = a->scale_b_cols;
  e.accum = a->accum;
  e.act = a->act;
  e.out_f16 = a->out_f16;
  e.pre_out = a->pre_out;
  e.pre_in = a->pre_in;
  e.q_mx = static_cast<uint8_t*>(a->q_mx);
  e.s_mx = static_cast<uint8_t*>(a->s_mx);
  return e;
}

bool epilogue_args_ok(const wk_gemm_mx_args* a) {
  if (a->act < 0 || a->act > 2 || (a->act == ACT_DGELU && !a->pre_in)) return false;
  if ((a->pre_out && !aligned16(a->pre_out)) || (a->pre_in && !aligned16(a->pre_in))) return false;
  if (a->scale_b && a->scale_b_cols && !aligned16(a->scale_b)) return false;
  return true;
}

GemmParams params_of(const wk_gemm_mx_args* a, int* status) {
  GemmParams p = {};
  p.out = a->out;
  p.epi = epilogue_of(a);
  p.M = a->m;
  p.N = a->n;
  p.group_m = a->group_m ? a->group_m : 8;
  p.status = status;
  return p;
}

}  // namespace
}  // namespace wk

extern "C" int64_t wk_gemm_mxfp8_workspace_bytes(int m, int n, int k) {
  if (m < 0 || n < 0 || k < 0) return WK_E_ARG;
  return (static_cast<int64_t>(m) + n) * (k / 32) + 32;
}

extern "C" int64_t wk_mx_scales_tiled_bytes(int rows, int k) {
  if (rows < 0 || k < 0 || rows % 128 || k % 128) return WK_E_ARG;
  return static_cast<int64_t>(rows) * (k / 32);
}

extern "C" int wk_tile_mx_scales(const void* s, int rows, int k, void* dst, void* stream) {
  using namespace wk;
  if (rows < 0 || k < 0 || rows % 128 || k % 128 || !dst || !aligned16(dst)) return WK_E_ARG;
  if (s && (reinterpret_cast<uintptr_t>(s) & 3)) return WK_E_ARG;
  if (rows == 0 || k == 0) return 0;
  if (int unsupported = require_sm100()) return unsupported;
  const ScaleTensor t = {static_cast<const uint8_t*>(s), static_cast<uint8_t*>(dst), rows / 128}, none = {};
  return retile(t, none, k, static_cast<cudaStream_t>(stream));
}

extern "C" int wk_gemm_mxfp8(const wk_gemm_mx_args* a, void* stream) {
  using namespace wk;
  if (!a) return WK_E_ARG;
  const int m = a->m, n = a->n, k = a->k;
  if (m < 0 || n < 0 || k < 0 || m % 128 || n % 128 || k % 128) return WK_E_ARG;
  if (m == 0 || n == 0) return 0;
  if (k == 0) return WK_E_ARG;
  if (!a->a || !a->b || !a->out) return WK_E_ARG;
  if (!aligned16(a->a) || !aligned16(a->b) || !aligned16(a->out) || !aligned16(a->workspace)) return WK_E_ARG;
  const bool a_tiled = a->a_scale_tiled != 0, b_tiled = a->b_scale_tiled != 0;
  if (!a->workspace && !(a_tiled && b_tiled)) return WK_E_ARG;  // scratch for whatever is still row-major
  if (a_tiled && (!a->a_scale_mx || !aligned16(a->a_scale_mx))) return WK_E_ARG;
  if (b_tiled && (!a->b_scale_mx || !aligned16(a->b_scale_mx))) return WK_E_ARG;
  if (a->a_scale_mx && (reinterpret_cast<uintptr_t>(a->a_scale_mx) & 3)) return WK_E_ARG;
  if (a->b_scale_mx && (reinterpret_cast<uintptr_t>(a->b_scale_mx) & 3)) return WK_E_ARG;
  if ((a->q_mx == nullptr) != (a->s_mx == nullptr)) return WK_E_ARG;
  if (a->q_mx && !aligned16(a->q_mx)) return WK_E_ARG;
  if (!epilogue_args_ok(a)) return WK_E_ARG;
  if (a->cta_pair < 0 || a->cta_pair > 2 || a->group_m < 0) return WK_E_ARG;
  if (a->workspace && a->workspace_bytes < wk_gemm_mxfp8_workspace_bytes(m, n, k)) return WK_E_ARG;
  if (int unsupported = require_sm100()) return unsupported;
  int* status = status_word();
  if (!status) return WK_E_CUDA;
  cudaStream_t st = static_cast<cudaStream_t>(stream);

  // scale tensors the caller has already tiled (wk_tile_mx_scales) are read where they are; the others are
  // re-tiled into the workspace first
  const uint8_t* sfa = static_cast<const uint8_t*>(a->a_scale_mx);
  const uint8_t* sfb = static_cast<const uint8_t*>(a->b_scale_mx);
  ScaleTensor ta = {}, tb = {};
  if (!a_tiled) {
    ta = {sfa, static_cast<uint8_t*>(a->workspace), m / 128};
    sfa = ta.dst;
  }
  if (!b_tiled) {
    tb = {sfb, static_cast<uint8_t*>(a->workspace) + ((static_cast<int64_t>(m) * (k / 32) + 15) / 16) * 16, n / 128};
    sfb = tb.dst;
  }
  if (int r = retile(ta, tb, k, st)) return r;

  GemmParams p = params_of(a, status);
  return launch_gemm<KIND_MX>(a->a, a->b, sfa, sfb, k, a->cta_pair, p, st);
}

// ---------------------------------------------------------------------------
// Variant for callers that must not allocate device memory.
// ---------------------------------------------------------------------------
// The re-tiled scale factors live in a fixed array that is part of the loaded
// module instead of a caller-provided workspace, and the status word is a module
// variable too, so this entry point never calls cudaMalloc / cudaFree or any
// allocating library routine.  Every GPU that loads the library carries the array
// (WK_NOALLOC_SCRATCH_BYTES) until the process exits.
//
// In host code the names below are only handles for the runtime, not device
// addresses; the real addresses are looked up once per device with
// cudaGetSymbolAddress while that device is current, and those pointers are what
// the kernels receive.
namespace wk {
namespace {

constexpr int64_t kNoAllocScratchBytes = WK_NOALLOC_SCRATCH_BYTES;
static __device__ __align__(256) uint8_t g_noalloc_scratch[kNoAllocScratchBytes];
static __device__ int g_noalloc_status;

constexpr int kNoAllocMaxDevices = 64;
uint8_t* g_noalloc_scratch_ptr[kNoAllocMaxDevices] = {};
int* g_noalloc_status_ptr[kNoAllocMaxDevices] = {};

// Looks the two device addresses up on the first call made on a device.
int noalloc_setup(int dev) {
  if (g_noalloc_scratch_ptr[dev] && g_noalloc_status_ptr[dev]) return 0;
  void* scratch = nullptr;
  void* status = nullptr;
  if (cudaGetSymbolAddress(&scratch, g_noalloc_scratch) != cudaSuccess || !scratch) return WK_E_CUDA;
  if (cudaGetSymbolAddress(&status, g_noalloc_status) != cudaSuccess || !status) return WK_E_CUDA;
  g_noalloc_scratch_ptr[dev] = static_cast<uint8_t*>(scratch);
  g_noalloc_status_ptr[dev] = static_cast<int*>(status);
  return 0;
}

}  // namespace
}  // namespace wk

extern "C" int64_t wk_gemm_mxfp8_noalloc_max_bytes(void) { return wk::kNoAllocScratchBytes; }

extern "C" int wk_gemm_mxfp8_noalloc(const wk_gemm_mx_args* a, void* stream) {
  using namespace wk;
  if (!a) return WK_E_ARG;
  const int m = a->m, n = a->n, k = a->k;
  if (m < 0 || n < 0 || k < 0 || m % 128 || n % 128 || k % 128) return WK_E_ARG;
  if (m == 0 || n == 0) return 0;
  if (k == 0) return WK_E_ARG;
  if (!a->a || !a->b || !a->out) return WK_E_ARG;
  if (!aligned16(a->a) || !aligned16(a->b) || !aligned16(a->out)) return WK_E_ARG;
  if (a->a_scale_mx && (reinterpret_cast<uintptr_t>(a->a_scale_mx) & 3)) return WK_E_ARG;
  if (a->b_scale_mx && (reinterpret_cast<uintptr_t>(a->b_scale_mx) & 3)) return WK_E_ARG;
  if ((a->q_mx == nullptr) != (a->s_mx == nullptr)) return WK_E_ARG;
  if (a->q_mx && !aligned16(a->q_mx)) return WK_E_ARG;
  if (!epilogue_args_ok(a)) return WK_E_ARG;
  // scales that are already tiled need no scratch at all: such a caller uses wk_gemm_mxfp8 with a NULL workspace
  if (a->a_scale_tiled || a->b_scale_tiled) return WK_E_ARG;
  // the fixed array bounds the problem size: (M + N) * K / 32 scale bytes must fit
  if (wk_gemm_mxfp8_workspace_bytes(m, n, k) > kNoAllocScratchBytes) return WK_E_TOO_LARGE;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) return WK_E_CUDA;
  if (int unsupported = require_sm100()) return unsupported;
  int r = noalloc_setup(dev);
  if (r) return r;
  cudaStream_t st = static_cast<cudaStream_t>(stream);

  uint8_t* sfa = g_noalloc_scratch_ptr[dev];
  uint8_t* sfb = sfa + ((static_cast<int64_t>(m) * (k / 32) + 15) / 16) * 16;
  // every atom the GEMM will read is rewritten here, so nothing of the previous call survives into this one
  const ScaleTensor ta = {static_cast<const uint8_t*>(a->a_scale_mx), sfa, m / 128};
  const ScaleTensor tb = {static_cast<const uint8_t*>(a->b_scale_mx), sfb, n / 128};
  if ((r = retile(ta, tb, k, st))) return r;
  GemmParams p = params_of(a, g_noalloc_status_ptr[dev]);
  p.group_m = 8;
  return launch_gemm<KIND_MX>(a->a, a->b, sfa, sfb, k, 2, p, st);
}

extern "C" int wk_gemm_mxfp8_noalloc_status(void) {
  using namespace wk;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) return WK_E_CUDA;
  if (noalloc_setup(dev)) return WK_E_CUDA;
  if (cudaDeviceSynchronize() != cudaSuccess) return WK_E_CUDA;
  int v = 0;
  if (cudaMemcpy(&v, g_noalloc_status_ptr[dev], sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
    return WK_E_CUDA;
  if (v != 0 && cudaMemset(g_noalloc_status_ptr[dev], 0, sizeof(int)) != cudaSuccess) return WK_E_CUDA;
  return v;
}
