// hx_internal.h — host-side internals shared by the libhx translation units:
// the map handle and its probe tuning.
#pragma once
#include <cstdint>
#include <mutex>
#include <vector>
#include <cuda_runtime.h>
#include "../../include/hx.h"
#include "hx_host.h"
#include "hx_probe.cuh"

namespace hx {

struct Tuning {
  int group = 0;   // lanes per key; 0 = automatic policy (auto_policy)
  int unroll = 1;  // keys in flight per thread when group == 1
  int block = 256;
  bool blind = true;  // thread-per-key insert: CAS the home bucket without reading it first
  bool wide = false;  // thread-per-key windows of 64 B instead of 32 B
};

// A device buffer kept from call to call. One that a graph was captured with lives on
// when a larger one takes its place: replays use it.
struct ScratchBuf {
  void* ptr = nullptr;
  uint64_t bytes = 0;
  bool in_graph = false;
  std::vector<void*> kept;
  void release() {  // after a device synchronisation
    pool_free_now(ptr);
    for (void* p : kept) pool_free_now(p);
    ptr = nullptr;
    bytes = 0;
    kept.clear();
  }
};

}  // namespace hx

struct hx_map {
  int key_bytes = 0, val_bytes = 0;
  int sp = 0;
  int device = 0;
  void* buckets = nullptr;
  hx::DInfo* info = nullptr;
  uint64_t fill_ub = 0;  // host upper bound on fill (exact after a sync)
  hx::ScratchBuf own_scratch;
  hx::ScratchBuf* scratch = &own_scratch;  // views of a batch's maps share the batch's
  hx::Tuning tune;
  bool err_success = false;  // info->err is known to be success (see set_err_success)
  bool viewed = false;       // a device view was handed out: kernels of the caller may write info->err
  bool replayed = false;     // an insert, clean or resize was captured: replays may change fill and info->err unseen
  std::mutex mu;  // guards scratch growth; a map is not thread-safe otherwise
};


namespace hx {
// The plain per-map paths on a map handle (also used on views into a batch).
hx_status map_insert_view(hx_map* m, const void* keys, const void* vals, const void* pairs, uint64_t n,
                          cudaStream_t s);
hx_status map_find_view(hx_map* m, const void* keys, void* vals, void* pairs, uint64_t n, bool erase,
                        cudaStream_t s);
// device_rehash of the viewed table into a new cudaMallocAsync allocation of
// 2^new_sp buckets; the old bucket array is released stream-ordered.
hx_status map_rehash_view(hx_map* m, int new_sp, cudaStream_t s);

// A batch on one table, for the slice-by-slice kernels (hx_bulk.cu).
enum class BulkOp : int { INSERT, FIND, ERASE };
struct BulkCall {
  BulkOp op;
  int key_bytes;
  void* table;
  int sp;
  DInfo* info;
  const void* keys;   // keys (with vals: inserts; without: inserts of the index, look-ups, erases) ...
  const void* vals;
  const void* pairs;  // ... or pairs; look-ups write pairs' values
  void* out;          // look-ups: the values, or the pairs
  uint64_t n;
  uint64_t expected;  // about how many of the n records hold a key (sentinels are skipped)
  uint64_t fill_bound;  // the host's bound of the keys in the table after this call's inserts
};
// Whether the stream is being captured (also if the runtime cannot say).
bool capturing(cudaStream_t s);
// Runs the batch if the rule for such sizes says so and its scratch can be had;
// *done says whether it did (if not, nothing was launched).
hx_status bulk_try(const BulkCall& c, cudaStream_t s, bool* done);
}  // namespace hx
