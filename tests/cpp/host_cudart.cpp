// A stand-in for the CUDA runtime that keeps "device" memory on the host and launches
// nothing, so that libhx's host code (buffer sizes, bookkeeping, error paths) runs
// without a GPU. Linked with libhx's own objects in place of libcudart.
//
// Every allocation ends at a page that may not be touched: a write past a buffer ends
// the process. fake_* functions let a test look at memory and make calls fail.
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstdint>
#include <cstring>
#include <map>

namespace {
struct Block {
  void* base;
  size_t mapped, bytes;
  bool host, captured;
};
std::map<void*, Block> g_live;
struct Pool {
  uint64_t used = 0, held = 0, threshold = 0;
};
std::map<void*, Pool*> g_of_pool;
size_t g_fail_from = 0;    // pool allocations of at least this many bytes fail (0: none)
int g_fail_host = 0;       // the next so many page-locked allocations fail
bool g_capturing = false;
cudaError_t g_last = cudaSuccess;

uint64_t g_capacity = ~0ull;  // bytes of the device

cudaError_t fail(cudaError_t e) { return g_last = e; }
uint64_t taken();  // by the pools, and by allocations outside them
cudaError_t make(void** p, size_t bytes, bool host = false) {
  const size_t page = 4096, body = (bytes + page - 1) / page * page + (bytes ? 0 : page);
  char* m = static_cast<char*>(mmap(nullptr, body + page, PROT_READ | PROT_WRITE,
                                    MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0));
  if (m == MAP_FAILED) return fail(cudaErrorMemoryAllocation);
  mprotect(m + body, page, PROT_NONE);
  *p = m + (body - (bytes + 15) / 16 * 16);
  g_live[*p] = Block{m, body + page, bytes, host, g_capturing};
  return cudaSuccess;
}
cudaError_t drop(void* p) {
  if (!p) return cudaSuccess;
  auto it = g_live.find(p);
  if (it == g_live.end()) return fail(cudaErrorInvalidValue);
  auto of = g_of_pool.find(p);
  if (of != g_of_pool.end()) {
    of->second->used -= it->second.bytes;
    g_of_pool.erase(of);
  }
  munmap(it->second.base, it->second.mapped);
  g_live.erase(it);
  return cudaSuccess;
}
// What a pool does at a synchronisation: hands back what it holds above its threshold.
struct Pools {
  std::map<Pool*, int> all;
  void settle() {
    for (auto& p : all)
      if (p.first->held > p.first->threshold)
        p.first->held = p.first->used > p.first->threshold ? p.first->used : p.first->threshold;
  }
} g_pools;
uint64_t taken() {
  uint64_t n = 0;
  for (auto& p : g_pools.all) n += p.first->held;
  for (auto& b : g_live) n += b.second.host || g_of_pool.count(b.first) ? 0 : b.second.bytes;
  return n;
}
dim3 g_grid, g_block;
size_t g_smem;
cudaStream_t g_stream;
}  // namespace

extern "C" {
void* fake_find(size_t bytes) {  // a live device allocation of exactly so many bytes
  for (auto& b : g_live)
    if (b.second.bytes == bytes && !b.second.host) return b.first;
  return nullptr;
}
int fake_live(int captured) {  // live device allocations: made under capture, or outside
  int n = 0;
  for (auto& b : g_live) n += !b.second.host && b.second.captured == (captured != 0);
  return n;
}
void fake_fail_pool_from(size_t bytes) { g_fail_from = bytes; }
void fake_capacity(uint64_t bytes) { g_capacity = bytes; }
void fake_fail_host(int count) { g_fail_host = count; }
void fake_capture(int on) { g_capturing = on != 0; }
uint64_t fake_pool_held() {  // bytes that every pool holds once all work is done
  g_pools.settle();
  uint64_t n = 0;
  for (auto& p : g_pools.all) n += p.first->held;
  return n;
}

void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(f));
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
  g_grid = g, g_block = b, g_smem = smem, g_stream = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = g_grid, *b = g_block, *smem = g_smem, *static_cast<cudaStream_t*>(s) = g_stream;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return cudaSuccess; }

cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_capacity != ~0ull && taken() + n > g_capacity) return fail(cudaErrorMemoryAllocation);
  return make(p, n);
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return make(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) {
  if (g_fail_host > 0) {
    --g_fail_host;
    return fail(cudaErrorMemoryAllocation);
  }
  return make(p, n, true);
}
cudaError_t cudaFree(void* p) { return drop(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return drop(p); }
cudaError_t cudaFreeHost(void* p) { return drop(p); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
  Pool* q = new Pool();
  g_pools.all[q] = 1;
  *p = reinterpret_cast<cudaMemPool_t>(q);
  return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) {
  g_pools.all.erase(reinterpret_cast<Pool*>(p));
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t) {
  if (g_fail_from && n >= g_fail_from) return fail(cudaErrorMemoryAllocation);
  Pool* q = reinterpret_cast<Pool*>(pool);
  if (g_capacity != ~0ull && q->used + n > q->held && taken() + (q->used + n - q->held) > g_capacity)
    return fail(cudaErrorMemoryAllocation);
  const cudaError_t e = make(p, n);
  if (e != cudaSuccess) return e;
  g_of_pool[*p] = q;
  q->used += n;
  if (q->held < q->used) q->held = q->used;
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void* v) {
  if (a == cudaMemPoolAttrReleaseThreshold) reinterpret_cast<Pool*>(p)->threshold = *static_cast<uint64_t*>(v);
  return cudaSuccess;
}
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void* v) {
  const Pool* q = reinterpret_cast<Pool*>(p);
  *static_cast<uint64_t*>(v) = a == cudaMemPoolAttrUsedMemCurrent ? q->used : q->held;
  return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t keep) {
  Pool* q = reinterpret_cast<Pool*>(p);
  if (q->held > keep) q->held = q->used > keep ? q->used : keep;
  return cudaSuccess;
}

cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() {
  g_pools.settle();
  return cudaSuccess;
}
cudaError_t cudaDeviceSetLimit(cudaLimit, size_t) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 152;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 4;
  return cudaSuccess;
}
static CUresult fake_ctx(CUcontext* c) {
  *c = reinterpret_cast<CUcontext>(&g_last);
  return static_cast<CUresult>(0);
}
static CUresult fake_ctx_id(CUcontext, unsigned long long* id) {
  *id = 1;
  return static_cast<CUresult>(0);
}
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
  *f = std::strcmp(name, "cuCtxGetId") ? reinterpret_cast<void*>(fake_ctx) : reinterpret_cast<void*>(fake_ctx_id);
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
  *p = const_cast<void*>(s);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(&g_stream);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  g_pools.settle();
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
  *c = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
static cudaError_t event(cudaEvent_t* e) {
  *e = reinterpret_cast<cudaEvent_t>(&g_stream);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return event(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return event(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0.f;
  return cudaSuccess;
}
}  // extern "C"
