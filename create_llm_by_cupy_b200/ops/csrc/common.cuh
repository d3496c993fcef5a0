// Host-side helpers shared by every translation unit of the native library:
//   * the exported-symbol macro and launch-error convention (every entry point returns a
//     cudaError_t-compatible int, 0 = success);
//   * the device status word kernels use to report a bounded wait that ran out;
//   * a cache of TMA tensor maps (cuTensorMapEncodeTiled is looked up through the runtime so the
//     library does not link against libcuda).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#define B200_API extern "C" __attribute__((visibility("default")))

#define B200_CHECK(expr)                                                                      \
  do {                                                                                        \
    cudaError_t _e = (expr);                                                                  \
    if (_e != cudaSuccess) {                                                                  \
      fprintf(stderr, "[b200] %s failed at %s:%d: %s\n", #expr, __FILE__, __LINE__,           \
              cudaGetErrorString(_e));                                                        \
      return static_cast<int>(_e);                                                            \
    }                                                                                         \
  } while (0)

// Kernels that are meant to run BESIDE the persistent GEMM / attention CTAs (collectives, AdamW pipelined with
// the next forward) ask for the same shared-memory carve-out as those CTAs, the maximum. An SM holds one
// carve-out configuration at a time: a small kernel left on the driver's default (a small shared-memory
// partition) and a 225 KiB GEMM CTA cannot be resident on one SM together, so each waits for the other to
// drain - and a persistent GEMM cannot finish before every one of its CTAs has had its turn.
#define B200_PREFER_MAX_SMEM(kernel)                                                                            \
  do {                                                                                                          \
    static bool _done = false;                                                                                  \
    if (!_done) {                                                                                               \
      cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared); \
      _done = true;                                                                                             \
    }                                                                                                           \
  } while (0)

namespace b200 {

typedef __nv_bfloat16 bf16;
typedef __nv_bfloat162 bf162;

// Device pointer to a 4-int status block owned by the Python side:
// [0] first error code, [1] kernel id that raised it, [2..3] free for detail.
int* status_ptr();

enum SwizzleMode { SWIZZLE_NONE_ = 0, SWIZZLE_128B_ = 3 };

// A tensor map by value (the cache it came from may drop its entry at any time); converts to a pointer to itself, null
// when it could not be made.
struct TensorMap {
  CUtensorMap map;
  bool valid = false;
  operator const CUtensorMap*() const { return valid ? &map : nullptr; }
};

// 2D tensor map for a row-major matrix of `rows` x `cols` elements of `elem_bytes` bytes with a row pitch of `ld`
// elements. The box is box_cols x box_rows. Not valid (and prints why) when the matrix breaks a TMA rule (16-byte base /
// pitch).
TensorMap get_tensor_map_2d(const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows,
                            uint32_t box_cols, int elem_bytes, int swizzle);

TensorMap get_tensor_map_bthd(const void* base, uint64_t B, uint64_t T, uint64_t heads, uint64_t D, uint64_t bs,
                              uint64_t ts, uint64_t hs, uint32_t box_t, uint32_t box_d);

int num_sms();

#ifdef __CUDACC__
// Programmatic dependent launch. A kernel launched with `launch_pdl` may become resident while the kernel before it on
// its stream still runs: its launch latency, barrier set-up and tensor-memory allocation then lie under that kernel's
// tail (about 2 us of every pair of dependent kernels). The two halves of the rule:
//   * pdl_wait() returns when every kernel before this one has completed and its stores are visible. Nothing that another
//     kernel may have written - weights included: the one before may be the optimizer - is read, and nothing is written,
//     before it; only an L2 prefetch, which cannot go stale, may come earlier. Inputs are read through plain
//     pointers: no `const __restrict__`, no __ldg or __ldcs. A load that the compiler takes for invariant, or an intrinsic that
//     is not volatile, could be moved above the wait, and the read-only path is only for data that nobody writes while the
//     kernel is resident.
//   * pdl_trigger() lets the next kernel start once all CTAs of this one have got there (or have ended; a kernel need not
//     call it); the first thread of a CTA that gets there counts for the CTA. It never stands before pdl_wait(), so that one kernel at most is waiting while another runs: with the
//     trigger first, two or three kernels' CTAs piled up on the SMs that happened to be free (777 tokens through the 125M
//     model: 1152 us without all this, 1049 with the trigger first, 979 like this; one token 520 / 386 / 372).
// A kernel that waits for another GPU neither triggers nor is launched this way.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// `bytes` (a multiple of 16) from the 16-byte aligned `p` on their way into L2; nothing waits and nothing is delivered.
__device__ __forceinline__ void l2_prefetch(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "r"(bytes) : "memory");
}

// cluster_x > 0: thread-block clusters of that many CTAs along x (0: none, or fixed by the kernel). An error is the caller's
// alone: it does not stay behind for the next one that asks cudaGetLastError.
template <typename... Params, typename... Args>
inline cudaError_t launch_pdl(void (*kern)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster_x,
                              Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cluster_x > 0) {
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster_x;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

// A length or index that a kernel reads from device memory (valid key lengths, target ids) and then uses to bound
// its loops or to pick a column. Every build clamps it into [0, hi]; the debug build (-DB200_BOUNDS_CHECK=1, made by
// ``B200_BOUNDS_CHECK=1 python -m create_llm_by_cupy_b200.ops.build``) also reports a value outside that range through
// the status word (error 4, the kernel id, the offending value) - the stand-in for a memory checker on arguments
// that only exist on the device.
__device__ __forceinline__ int checked_index(int v, int hi, int* status, int kernel_id) {
#ifdef B200_BOUNDS_CHECK
  if ((v < 0 || v > hi) && status != nullptr && atomicCAS(status, 0, 4) == 0) {
    status[1] = kernel_id;
    status[2] = v;
  }
#else
  (void)status;
  (void)kernel_id;
#endif
  return v < 0 ? 0 : (v > hi ? hi : v);
}
#endif

}  // namespace b200
