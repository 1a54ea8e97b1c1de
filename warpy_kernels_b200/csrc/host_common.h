// Host-side helpers shared by the C-ABI entry points: tensor-map encoding through
// the driver entry point (no link-time dependency on libcuda), the per-device
// status word the kernels report bounded-wait failures to, and argument checks.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <initializer_list>

#include "../../include/warpy_b200.h"

namespace wk {

// Returns 0 and fills *map, or a negative WK_E_* code.
int encode_tmap(CUtensorMap* map, CUtensorMapDataType dtype, uint32_t rank, const void* base,
                const uint64_t* dims, const uint64_t* strides_bytes /* rank-1 entries */,
                const uint32_t* box, CUtensorMapSwizzle swizzle);

// Device pointer of the int status word of the current device (allocated on first use).
int* status_word();

// 100 for a device of compute capability 10.x, WK_E_UNSUPPORTED for any other, WK_E_CUDA if it cannot be asked.
int device_arch_of(int dev);

// 0 if the current device can run this library's kernels, else the negative code an entry point returns
// (WK_E_UNSUPPORTED for a device that is not compute capability 10.x).  Allocates nothing.
int require_sm100();

// Number of SMs of the current device (cached).
int sm_count();

// Raises the dynamic shared memory limit of `func` once per device.
int allow_smem(const void* func, int bytes);

// How many clusters of `size` CTAs of this kernel the current device runs at once (asked once per device).
int clusters_at_once(const void* func, int size, int threads, int smem);

// Launches `func` in clusters of `cluster` CTAs as a programmatic dependent: it may be set up while the kernel before it
// in the stream still runs, so it must execute griddepcontrol.wait before it touches global memory.
int launch_pdl(const void* func, dim3 grid, int threads, int smem, cudaStream_t stream, int cluster,
               std::initializer_list<void*> args);

// Heads whose blocks are handed out longest first together (band_order in common.cuh), of `heads` heads with `blocks`
// blocks each that read `head_bytes` apiece.  Head after head leaves SMs idle behind a long block of the last heads: 2 x 8
// KV heads of 16 key blocks take 102 tile times on 148 SMs where 60 are work, longest first over all of them 65.  That is
// only worth anything where CTAs are few per SM (at eight it is 3 % at most, and neighbours in time no longer share a head's
// tensors), and the heads of a band have to fit L2 together.  BF16 backward: 2 x 32 heads, 2048 x 2048 290 -> 279 us,
// 2 x 16 heads, d 64 130 -> 121, 4 heads, 12000 x 3000 82 -> 65; but 4 x 32 heads, 4096 x 4096 2200 -> 2236.  Forward: BF16, 2 x 32 heads,
// 2048 x 2048 102 -> 88 us, 16 heads, 4096 x 4096 127 -> 97 (FP8 81 -> 70).
inline int band_heads(int blocks, int heads, int64_t head_bytes, int sms) {
  if (static_cast<int64_t>(blocks) * heads > 8ll * sms) return 1;
  const int64_t fit = (96ll << 20) / (head_bytes > 0 ? head_bytes : 1);
  return fit < 1 ? 1 : fit < heads ? static_cast<int>(fit) : heads;
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace wk

#define WK_CUDA_OK(expr)                    \
  do {                                      \
    cudaError_t e__ = (expr);               \
    if (e__ != cudaSuccess) return WK_E_CUDA; \
  } while (0)
