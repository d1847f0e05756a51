// hx_host.h — host-side helpers shared by the libhx translation units.
#pragma once
#include <atomic>
#include <cstdint>
#include <cuda_runtime.h>
#include "../../include/hx.h"

// NVTX ranges name each C-ABI call in Nsight Systems timelines and for
// `ncu --nvtx` filters. NVTX v3 is header-only; with no tool attached a range
// costs one call that returns at once. Build with -DHX_NVTX=0 to compile
// them out.
#ifndef HX_NVTX
#define HX_NVTX 1
#endif
#if HX_NVTX
#include <nvtx3/nvToolsExt.h>
#endif

namespace hx {

#if HX_NVTX
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange&) = delete;
  NvtxRange& operator=(const NvtxRange&) = delete;
};
#define HX_RANGE(name) ::hx::NvtxRange hx_nvtx_range_(name)
#else
#define HX_RANGE(name) ((void)0)
#endif

// Records the CUDA error for hx_last_cuda_error() and maps it to a status.
hx_status cuda_status(cudaError_t e);
#define HX_CUDA(call)                                   \
  do {                                                  \
    cudaError_t hx_e_ = (call);                         \
    if (hx_e_ != cudaSuccess) return ::hx::cuda_status(hx_e_); \
  } while (0)
// Checks the launch that was just issued and counts it.
hx_status after_launch();

// The current context's driver-assigned id, unique for the life of the process
// (0 when the driver does not provide it).
unsigned long long current_context_id();

int sm_count();  // SMs of the current device (cached per device)

// A device array of elements of `align` bytes must start at a multiple of
// `align`: the kernels load and store whole elements (and pairs as one 8- or
// 16-byte access), so a misaligned pointer is rejected before any launch.
inline bool misaligned(const void* p, unsigned align) {
  return (reinterpret_cast<uintptr_t>(p) % align) != 0;
}

// Blocks per SM for a kernel at a block size (cached by the caller).
template <class F>
int blocks_per_sm(F kernel, int block, size_t smem = 0) {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, block, smem) != cudaSuccess || nb < 1) nb = 1;
  return nb;
}

// Stream-ordered device memory from libhx's own pool of the current device: scratch of
// calls and tables that were grown into. The device's default pool hands freed memory to the driver
// at every synchronisation, so a caller that waits for each result has its scratch
// mapped anew on every call (the first copy_if of 2^28 words on new arrays: 0.66 ms, with
// this pool 0.45 ms), and a growing map every new table (2*10^7 u32 keys into a map of the
// default size, in six chunks: 5.32 ms, with this pool 3.60 ms). At a synchronisation this
// pool holds at most kPoolKeepBytes beyond what is in use while a map or batch of the
// device exists, and kPoolIdleBytes otherwise. Scratch of one call: 4.6 GB at most for
// look-ups; for inserts 6.4 GB (2^27 u64 pairs into 2^29 buckets), 4.8 GB into 2^27. Safe with several threads and streams, as any stream-ordered
// pool is. A server's tables are in a pool of its own.
constexpr uint64_t kPoolKeepBytes = 5ull << 30;
constexpr uint64_t kPoolIdleBytes = 1ull << 30;
// counted: in the count of what is in use, and given back with pool_free; not counted: a
// small buffer of one call, given back with cudaFreeAsync.
cudaError_t pool_alloc(void** p, uint64_t bytes, cudaStream_t s, bool counted = true);
cudaError_t pool_free(void* p, cudaStream_t s);
void pool_free_now(void* p);  // after a synchronisation; p may be of cudaMalloc or null
void pool_trim(uint64_t keep_free);         // of the current device, to what is in use and keep_free
void pool_object(int change, int dev);      // +1: created, -1: destroyed (after a device synchronisation)
// cudaMalloc; where the device has no room, once more when the pool has given back what is free.
cudaError_t device_alloc(void** p, uint64_t bytes);

// Stream-ordered scratch: a caller buffer when given, else pool_alloc
// on the stream, released stream-ordered by the destructor.
struct Scratch {
  void* ptr = nullptr;
  bool owned = false;
  cudaStream_t s = nullptr;
  hx_status get(void* caller, uint64_t caller_bytes, uint64_t need, cudaStream_t stream);
  ~Scratch();
};

}  // namespace hx
