// hx_bulk.cuh — large batches of inserts, look-ups and erases, slice by slice.
//
// A random access to a table larger than L2 costs a DRAM sector of its own:
// 25 G CAS/s and 44 G reads/s on GB300, whatever the kernel does (1.4 TB/s of
// the 6.8 TB/s that a copy reaches). A batch with more than about one key per
// few buckets touches nearly every line of the table anyway, so these kernels
// sort the batch by table slice first and then stream the table once:
//   1. split (one pass, or two for more than kMaxDigits slices): the keys
//      (with their values, or with their number in the batch) are binned by
//      the top bits of their home bucket. A tile is binned in shared memory
//      and leaves as one contiguous run per bin.
//   2. slice: one CTA per slice of 32 KiB of buckets reads it, looks the bin's
//      keys up in shared memory, and writes the buckets that change, and only
//      those: the CTA of the slice before may at the same time write values and
//      TOMBSTONEs into this slice's first buckets (its own keys that sit past its
//      end), which a write of the whole slice would undo.
//   3. left: a key that may belong past the end of its slice is handled in the
//      whole table, after every slice.
//   4. scatter (look-ups): the values found leave step 2 binned by their place
//      in the output, and are written to it region by region, so that the
//      writes meet in L2.
// Every step reads and writes memory in order, and the table once.
//
// Bins have a fixed room, a little over what equally likely home buckets give
// (bulk_bin_room); a key that finds its bin full is handled at once in the
// whole table, which no CTA holds a copy of yet. So any key distribution is
// handled, and one that does not spread costs what a random access costs.
//
// The decisions per bucket are those of hx_probe.cuh: a key goes to the first
// EMPTY bucket after its home unless it is found before it; TOMBSTONE buckets
// are never reused.
#pragma once
#include "hx_internal.h"
#include "hx_probe.cuh"
#include "../../include/hx_stream.cuh"

namespace hx {

// Where a split reads its records: keys with values, pairs, keys whose value
// is their index, or the bins of the split before.
enum class BulkSrc : int { KEYS, PAIRS, INDEX, BINS };

constexpr int kBulkThreads = 512;
constexpr int kMaxDigitLog = 9;  // bins of one split: 512
constexpr int kMaxDigits = 1 << kMaxDigitLog;
constexpr int kRegionLog = 7;  // output regions of the look-ups: at most 2^7 (+ a ragged one)
constexpr int kMaxRegions = (1 << kRegionLog) + 1;
// Slices of 32 KiB (4096 u32 or 2048 u64 buckets), 512 threads, three CTAs per SM (40
// registers). On 2^27 u32 buckets / 2^26 keys, insert + look-up: 2.94 ms, slices of half
// the size with 256 threads and six CTAs 3.0 ms, 256 threads on the full size 4.2 ms.
#ifndef HX_SLICE_THREADS
#define HX_SLICE_THREADS 512
#endif
#ifndef HX_SLICE_LOG
#define HX_SLICE_LOG 12
#endif
#ifndef HX_SLICE_MINB
#define HX_SLICE_MINB 3
#endif
constexpr int kSliceThreads = HX_SLICE_THREADS;

template <class P>
__host__ __device__ constexpr int slice_log() {
  return sizeof(P) == 8 ? HX_SLICE_LOG : HX_SLICE_LOG - 1;
}

// What travels with a key: its value, its number in the batch, or nothing.
struct NoPay {};
template <class P, BulkOp OP>
struct BulkPay {
  using T = typename PairTraits<P>::V;
};
template <class P>
struct BulkPay<P, BulkOp::FIND> {
  using T = uint32_t;
};
template <class P>
struct BulkPay<P, BulkOp::ERASE> {
  using T = NoPay;
};
template <class P, BulkOp OP>
__host__ __device__ constexpr unsigned bulk_record_bytes() {
  return sizeof(typename PairTraits<P>::K) + (OP == BulkOp::ERASE ? 0 : sizeof(typename BulkPay<P, OP>::T));
}
template <class P, BulkOp OP>
__host__ __device__ constexpr int bulk_items() {  // records per thread and tile: 64 KiB of shared memory a tile at most
  return bulk_record_bytes<P, OP>() <= 8 ? 16 : 8;
}
template <class P, BulkOp OP>
__host__ __device__ constexpr unsigned bulk_tile() {
  return kBulkThreads * bulk_items<P, OP>();
}

// A value found by a look-up, on its way to output element idx.
template <class V>
struct alignas(2 * sizeof(V)) FoundRec {
  V idx;
  V val;
};

template <class P>
struct BulkArgs {
  using K = typename PairTraits<P>::K;
  using V = typename PairTraits<P>::V;
  P* table;
  int sp;
  DInfo* info;
  V* out;               // look-ups: output element i is out[i * out_stride]
  unsigned out_stride;
  // the batch
  const K* keys;
  const V* vals;
  const P* pairs;
  uint64_t n;
  uint64_t first;  // number of its first key in the caller's batch (insertIndex)
};

struct BulkBins {
  void* keys;
  void* pay;
  unsigned* count;  // records asked for; min(count, room) are in the bin
  unsigned room;
  int log_bins;
};

// One key straight into the whole table; the counters go to the caller.
struct BulkCounts {
  unsigned ins = 0, maxd = 0, erased = 0;
  bool fail = false;
};
template <class P, BulkOp OP, class Y>
__device__ __noinline__ void bulk_direct(const BulkArgs<P>& a, typename PairTraits<P>::K key, Y pay, unsigned limit,
                                         BulkCounts& c) {
  using V = typename PairTraits<P>::V;
  constexpr int B = sizeof(P) == 8 ? 4 : 2;
  if constexpr (OP == BulkOp::INSERT) {
    insert_one_t1_win<P, B>(a.table, a.sp, key, pay, c.ins, c.maxd, c.fail);
  } else {
    const uint32_t h = home_slot(key, a.sp);
    Window<P, B> w;
    load_buckets<B>(a.table + (h & ~(uint32_t)(B - 1)), w.k, w.v);
    uint32_t slot;
    V v;
    if (find_t1<P, B>(a.table, a.sp, key, limit, h, w, slot, v)) {
      if constexpr (OP == BulkOp::ERASE) {
        if (cas_key(a.table + slot, key, PairTraits<P>::TOMB)) ++c.erased;
      } else {
        a.out[(uint64_t)pay * a.out_stride] = v;
      }
    }
  }
}

__device__ __forceinline__ void bulk_publish(DInfo* info, const BulkCounts& c, int lane) {
  const unsigned ins = __reduce_add_sync(0xffffffffu, c.ins);
  const unsigned maxd = __reduce_max_sync(0xffffffffu, c.maxd);
  const unsigned erased = __reduce_add_sync(0xffffffffu, c.erased);
  const bool fail = __any_sync(0xffffffffu, c.fail);
  if (lane == 0) {
    if (ins) atomicAdd(&info->fill, (unsigned long long)ins);
    if (maxd) atomicMax(&info->max_probe, maxd);
    if (erased) {
      atomicAdd(&info->tombstones, (unsigned long long)erased);
      atomicAdd(&info->fill, 0ull - (unsigned long long)erased);
    }
    if (fail) atomicExch(&info->err, HX_STATUS_FAIL);
  }
}

// ---------------------------------------------------------------------------
// split: bins one tile of records by `log_digits` bits of the home bucket from
// bit `shift` on. From the caller's arrays the whole batch is one input bin; from
// bins (BINS), CTA c works on tile c % tiles_per_bin of input bin
// c / tiles_per_bin, and input bin b's digits are output bins b * digits + d.
// ---------------------------------------------------------------------------
template <class P, BulkOp OP, BulkSrc SRC>
__global__ void __launch_bounds__(kBulkThreads, 2) k_bulk_split(BulkArgs<P> a, BulkBins in, BulkBins out,
                                                            unsigned tiles_per_bin, int shift, int log_digits) {
  using K = typename PairTraits<P>::K;
  using V = typename PairTraits<P>::V;
  using Y = typename BulkPay<P, OP>::T;
  constexpr bool HAS_PAY = OP != BulkOp::ERASE;
  constexpr int IT = bulk_items<P, OP>();
  constexpr unsigned T = kBulkThreads, TILE = bulk_tile<P, OP>();
  static_assert(kMaxDigits <= (int)T, "one thread per digit");
  extern __shared__ __align__(16) unsigned char s_tile[];
  K* s_key = reinterpret_cast<K*>(s_tile);
  Y* s_pay = reinterpret_cast<Y*>(s_key + TILE);
  __shared__ unsigned s_hist[kMaxDigits], s_off[kMaxDigits], s_dst[kMaxDigits];
  __shared__ unsigned s_warp[T / 32];
  __shared__ unsigned s_total;
  const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned digits = 1u << log_digits;

  uint64_t first, end;  // records of this tile
  unsigned bin = 0;
  const K* in_keys;
  const Y* in_pay = nullptr;
  if constexpr (SRC == BulkSrc::BINS) {
    bin = blockIdx.x / tiles_per_bin;
    const unsigned held = min(in.count[bin], in.room);
    first = (uint64_t)(blockIdx.x % tiles_per_bin) * TILE;
    if (first >= held) return;
    end = held;
    in_keys = static_cast<const K*>(in.keys) + (uint64_t)bin * in.room;
    if constexpr (HAS_PAY) in_pay = static_cast<const Y*>(in.pay) + (uint64_t)bin * in.room;
  } else {
    first = (uint64_t)blockIdx.x * TILE;
    end = a.n;
    in_keys = a.keys;
  }
  if (tid < digits) s_hist[tid] = 0;

  K key[IT];
  Y pay[IT];
  bool act[IT];
#pragma unroll
  for (int j = 0; j < IT; ++j) {
    const uint64_t i = first + j * T + tid;
    act[j] = i < end;
    if (act[j]) {
      if constexpr (SRC == BulkSrc::PAIRS) {
        const P pr = a.pairs[i];
        key[j] = pr.first;
        if constexpr (OP == BulkOp::INSERT) pay[j] = pr.second;
      } else {
        key[j] = in_keys[i];
        if constexpr (SRC == BulkSrc::BINS && HAS_PAY) pay[j] = in_pay[i];
        if constexpr (SRC == BulkSrc::KEYS && OP == BulkOp::INSERT) pay[j] = a.vals[i];
        if constexpr (SRC == BulkSrc::INDEX && OP == BulkOp::INSERT) pay[j] = (V)(a.first + i);
      }
      if constexpr (SRC != BulkSrc::BINS && OP == BulkOp::FIND) pay[j] = (uint32_t)i;
    }
  }
  __syncthreads();
  auto digit_of = [&](K k) -> unsigned { return (home_slot(k, a.sp) >> shift) & (digits - 1); };
  unsigned code[IT];  // digit and rank within the tile's run of it
#pragma unroll
  for (int j = 0; j < IT; ++j) {
    if constexpr (SRC != BulkSrc::BINS)
      if (act[j]) act[j] = key[j] != PairTraits<P>::EMPTY && key[j] != PairTraits<P>::TOMB;
    if (act[j]) {
      const unsigned d = digit_of(key[j]);
      code[j] = d << 16 | atomicAdd(&s_hist[d], 1u);
    }
  }
  __syncthreads();
  {
    const unsigned c = tid < digits ? s_hist[tid] : 0u;
    const unsigned incl = hxs::warp_incl_scan(c, lane);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    unsigned before = 0;
    for (unsigned w = 0; w < warp; ++w) before += s_warp[w];
    const unsigned off = before + incl - c;
    if (tid < digits) {
      s_off[tid] = off;
      s_dst[tid] = (c ? atomicAdd(out.count + ((uint64_t)bin << log_digits) + tid, c) : 0u) - off;
    }
    if (tid == T - 1) s_total = before + incl;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < IT; ++j) {
    if (act[j]) {
      const unsigned pos = s_off[code[j] >> 16] + (code[j] & 0xffffu);
      s_key[pos] = key[j];
      if constexpr (HAS_PAY) s_pay[pos] = pay[j];
    }
  }
  __syncthreads();
  const unsigned total = s_total;
  K* out_keys = static_cast<K*>(out.keys);
  Y* out_pay = static_cast<Y*>(out.pay);
  BulkCounts c;
  bool any_over = false;
#pragma unroll 4
  for (unsigned i = tid; i < total; i += T) {
    const K k = s_key[i];
    const unsigned d = digit_of(k);
    const unsigned pos = s_dst[d] + i;
    if (pos < out.room) {
      const uint64_t at = (((uint64_t)bin << log_digits) + d) * out.room + pos;
      out_keys[at] = k;
      if constexpr (HAS_PAY) out_pay[at] = s_pay[i];
    } else {
      any_over = true;
    }
  }
  if (__syncthreads_or(any_over)) {  // a full bin: these keys go to the whole table
    const unsigned limit = OP == BulkOp::INSERT ? 0u : a.info->max_probe;
    for (unsigned base = 0; base < total; base += T) {
      const unsigned i = base + tid;
      K k{};
      bool over = false;
      if (i < total) {
        k = s_key[i];
        over = s_dst[digit_of(k)] + i >= out.room;
      }
      const unsigned m = __ballot_sync(0xffffffffu, over);
      if (over) {
        // a key repeated within the warp is inserted or erased once (k_insert_t1 has why)
        if (OP == BulkOp::FIND || __ffs(__match_any_sync(m, k)) - 1 == (int)lane) {
          Y y{};
          if constexpr (HAS_PAY) y = s_pay[i];
          bulk_direct<P, OP, Y>(a, k, y, limit, c);
        }
      }
    }
    bulk_publish(a.info, c, lane);
  }
}

// ---------------------------------------------------------------------------
// slice
// ---------------------------------------------------------------------------
// One bin against its slice, without probing key by key. A key sits in its home
// bucket, or, if that is not EMPTY, somewhere after it: the CTA chains the slice's
// keys that are not at home by their home (heads in shared memory), so a key of the
// bin is compared with its home bucket and, if need be, with a short chain, whatever
// the load factor. The slice's keys that sit past its end are found by walking on to
// the first EMPTY bucket there. An insert takes its home bucket with one CAS if that
// is EMPTY; the others (a quarter of a fresh table's keys at load factor 0.5) are
// queued and finished together: each joins the chain of its home (so a key repeated
// in the bin is inserted once) and takes the first EMPTY bucket after its home, found
// in a bitmap, 32 buckets at a look. Measured on 2^27 u32 buckets, 2^26 inserts into
// an empty table / 121 M look-ups at load factor 0.9: probing the slice in shared
// memory took 0.75 / 7.0 ms, bound by the instructions of long and uneven probes;
// grouping the keys by home with a counting sort 1.96 / 0.97 ms.
//
// An insert that finds its slice full from its home on goes to `left` and takes a
// bucket of the next slice after all slices are done. A slice whose end lies in a run
// of more than kTailBuckets full buckets, or with more than kTailNodes keys in it,
// leaves the keys that it cannot decide to `left` too, for a probe of the table.
constexpr uint32_t kNil = 0xffffu;
constexpr unsigned kTailNodes = 256, kTailBuckets = 4096;
constexpr unsigned kLeftProbe = 0x80000000u;  // in left.count: these keys probe from home

template <class P>
__host__ __device__ constexpr unsigned bin_room_max() {  // records of a bin at most (inserts)
  return (1u << slice_log<P>()) / 8 * 9;
}
template <class P, BulkOp OP>
__host__ __device__ constexpr unsigned slice_nodes() {  // the buckets, the tail's keys and, for inserts, the bin's
  return (1u << slice_log<P>()) + kTailNodes + (OP == BulkOp::INSERT ? bin_room_max<P>() : 0);
}
template <class P, BulkOp OP>
__host__ __device__ constexpr unsigned slice_smem() {
  using K = typename PairTraits<P>::K;
  return slice_nodes<P, OP>() * (sizeof(K) + 2) + (1u << slice_log<P>()) / 2 * 4 +
         (OP == BulkOp::FIND ? ((1u << slice_log<P>()) + kTailNodes) * sizeof(K) : 0) +
         (OP == BulkOp::INSERT ? bin_room_max<P>() * 2 : 0);
}
// Starts bringing `bytes` (a multiple of 16, from a 16-byte boundary) into L2.
__device__ __forceinline__ void prefetch_l2(const void* p, unsigned bytes) {
  if (bytes) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
// How many slices ahead a CTA fetches into L2: its first loads then wait for L2 and not
// for DRAM. 2^27 u32 buckets, 2^26 keys, insert / look-up: 1.34 / 1.60 ms without, 1.24 /
// 1.51 ms with 228 or 456 slices (half of or all that run at once), 1.28 / 1.53 with 912.
#ifndef HX_SLICE_AHEAD
#define HX_SLICE_AHEAD 228
#endif
__device__ __forceinline__ uint32_t smem_cas(uint32_t* p, uint32_t e, uint32_t d) { return atomicCAS(p, e, d); }
__device__ __forceinline__ uint64_t smem_cas(uint64_t* p, uint64_t e, uint64_t d) {
  return atomicCAS(reinterpret_cast<unsigned long long*>(p), (unsigned long long)e, (unsigned long long)d);
}

template <class P, BulkOp OP>
__global__ void __launch_bounds__(kSliceThreads, HX_SLICE_MINB) k_bulk_slice(BulkArgs<P> a, BulkBins bins,
                                                                            BulkBins left, void* recs,
                                                                            unsigned* rec_count, int region_log) {
  using K = typename PairTraits<P>::K;
  using V = typename PairTraits<P>::V;
  using Y = typename BulkPay<P, OP>::T;
  constexpr bool INS = OP == BulkOp::INSERT, FIND = OP == BulkOp::FIND, HAS_PAY = OP != BulkOp::ERASE;
  constexpr K EMPTY = PairTraits<P>::EMPTY, TOMB = PairTraits<P>::TOMB;
  constexpr unsigned SB = 1u << slice_log<P>(), T = kSliceThreads, NODES = slice_nodes<P, OP>();
  constexpr unsigned TAIL = SB, NEW = SB + kTailNodes;  // first nodes of the tail's keys and of the bin's
  constexpr unsigned HEADS = SB / 2;        // two homes share a chain
  constexpr unsigned PER = 32 / sizeof(P);  // buckets per 32-byte load
  constexpr unsigned N = SB / PER / T;      // such loads per thread
  extern __shared__ __align__(128) unsigned char s_slice[];
  K* s_key = reinterpret_cast<K*>(s_slice);        // per node
  V* s_val = reinterpret_cast<V*>(s_key + NODES);  // look-ups: per node
  unsigned* s_head = reinterpret_cast<unsigned*>(s_val + (FIND ? NODES : 0));
  uint16_t* s_next = reinterpret_cast<uint16_t*>(s_head + HEADS);  // per node
  uint16_t* s_queue = s_next + NODES;                              // inserts: records that wait
  __shared__ uint16_t s_tail_at[FIND ? 1 : kTailNodes];            // the tail's keys: buckets after the slice's end
  __shared__ unsigned s_empty[INS ? SB / 32 : 1];                  // bit set: the bucket may be EMPTY
  __shared__ unsigned s_last, s_left, s_done, s_max, s_tail, s_queued;
  __shared__ bool s_tail_known;
  __shared__ unsigned s_region[FIND ? kMaxRegions : 1];
  const unsigned s = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  const unsigned cnt = min(bins.count[s], bins.room);
  if (cnt == 0) return;
  const K* keys = static_cast<const K*>(bins.keys) + (uint64_t)s * bins.room;
  const Y* pays = static_cast<const Y*>(bins.pay) + (HAS_PAY ? (uint64_t)s * bins.room : 0);
  const uint32_t base = s << slice_log<P>(), tmask = (1u << a.sp) - 1u;
  auto home_of = [&](K k) -> unsigned { return home_slot(k, a.sp) - base; };  // SB or more: another slice's
  auto leave = [&](K k, Y y) {
    const uint64_t i = (uint64_t)s * left.room + atomicAdd(&s_left, 1u);
    static_cast<K*>(left.keys)[i] = k;
    if constexpr (HAS_PAY) static_cast<Y*>(left.pay)[i] = y;
  };
  // The bin's records, U per thread at a time; the first ones are under way with the table.
  constexpr unsigned U = sizeof(P) == 8 ? 5 : 4;
  K key[U];
  Y pay[U];
  auto fetch = [&](unsigned c0) {
#pragma unroll
    for (unsigned u = 0; u < U; ++u) {
      const unsigned i = c0 + u * T + tid;
      if (i < cnt) {
        key[u] = keys[i];
        if constexpr (HAS_PAY) pay[u] = pays[i];
      }
    }
  };

  if (tid == 64 && s + HX_SLICE_AHEAD < gridDim.x) {
    const unsigned f = s + HX_SLICE_AHEAD;
    prefetch_l2(a.table + ((uint64_t)f << slice_log<P>()), SB * sizeof(P));
    const unsigned n = min(bins.count[f], bins.room);
    prefetch_l2(static_cast<const K*>(bins.keys) + (uint64_t)f * bins.room, (n * (unsigned)sizeof(K) + 15) & ~15u);
    if constexpr (HAS_PAY)
      prefetch_l2(static_cast<const Y*>(bins.pay) + (uint64_t)f * bins.room, (n * (unsigned)sizeof(Y) + 15) & ~15u);
  }
  // ---- the slice's keys, those away from home chained ------------------------
  K tk[N][PER];
  V tv[N][PER];
#pragma unroll
  for (unsigned j = 0; j < N; ++j) load_buckets<(int)PER>(a.table + base + (j * T + tid) * PER, tk[j], tv[j]);
  K ek[PER];  // the last warp: the buckets after the slice
  V ev[PER];
  const bool tail_warp = tid >= T - 32;
  if (tail_warp) load_buckets<(int)PER>(a.table + ((base + SB + lane * PER) & tmask), ek, ev);
  fetch(0);
  for (unsigned i = tid; i < HEADS; i += T) s_head[i] = kNil;
  if (tid == 0) {
    s_last = s_left = s_done = s_max = s_tail = s_queued = 0;
    s_tail_known = true;
  }
  if constexpr (FIND)
    if (tid < kMaxRegions) s_region[tid] = 0;
  __syncthreads();
  unsigned past_empty = 0;  // one after the thread's last EMPTY bucket
#pragma unroll
  for (unsigned j = 0; j < N; ++j) {
    const unsigned b0 = (j * T + tid) * PER;
    unsigned m = 0;
#pragma unroll
    for (unsigned q = 0; q < PER; ++q) {
      const K k = tk[j][q];
      const unsigned h = home_of(k);
      if (k == EMPTY) m |= 1u << q;
      else if (k != TOMB && h < SB && h != b0 + q) s_next[b0 + q] = (uint16_t)atomicExch(&s_head[h % HEADS], b0 + q);
    }
    if constexpr (sizeof(P) == 8) {
      *reinterpret_cast<uint4*>(s_key + b0) = make_uint4(tk[j][0], tk[j][1], tk[j][2], tk[j][3]);
      if constexpr (FIND) *reinterpret_cast<uint4*>(s_val + b0) = make_uint4(tv[j][0], tv[j][1], tv[j][2], tv[j][3]);
    } else {
      *reinterpret_cast<ulonglong2*>(s_key + b0) = make_ulonglong2(tk[j][0], tk[j][1]);
      if constexpr (FIND) *reinterpret_cast<ulonglong2*>(s_val + b0) = make_ulonglong2(tv[j][0], tv[j][1]);
    }
    if (m) past_empty = b0 + 32 - __clz(m);
    if constexpr (INS) {  // 32 / PER neighbouring lanes hold the bits of one word
      m <<= b0 % 32;
#pragma unroll
      for (unsigned o = 1; o < 32 / PER; o <<= 1) m |= __shfl_xor_sync(0xffffffffu, m, o);
      if (b0 % 32 == 0) s_empty[b0 / 32] = m;
    }
  }
  past_empty = __reduce_max_sync(0xffffffffu, past_empty);
  if (lane == 0 && past_empty) atomicMax(&s_last, past_empty);
  if (tail_warp) {  // the slice's keys between its end and the first EMPTY bucket there
    for (unsigned d = 0;; d += 32 * PER) {
      if (d) load_buckets<(int)PER>(a.table + ((base + SB + d + lane * PER) & tmask), ek, ev);
      unsigned m = 0;
#pragma unroll
      for (unsigned q = 0; q < PER; ++q) m |= (unsigned)(ek[q] == EMPTY) << q;
      const unsigned ends = __ballot_sync(0xffffffffu, m != 0);
      const unsigned stop = ends ? __ffs(ends) - 1 : 32;
      const unsigned mine = lane < stop ? PER : (lane == stop ? __ffs(m) - 1 : 0u);  // of this lane's buckets
#pragma unroll
      for (unsigned q = 0; q < PER; ++q) {
        const unsigned h = home_of(ek[q]);
        if (q < mine && ek[q] != TOMB && h < SB) {
          const unsigned t = atomicAdd(&s_tail, 1u);
          if (t < kTailNodes) {
            s_key[TAIL + t] = ek[q];
            if constexpr (FIND) s_val[TAIL + t] = ev[q];
            else s_tail_at[t] = (uint16_t)(d + lane * PER + q);
            s_next[TAIL + t] = (uint16_t)atomicExch(&s_head[h % HEADS], TAIL + t);
          } else {
            s_tail_known = false;
          }
        }
      }
      if (ends) break;
      if (d + 32 * PER >= kTailBuckets) {
        if (lane == 0) s_tail_known = false;
        break;
      }
    }
  }
  __syncthreads();
  const unsigned last = s_last;  // homes from `last` on have no EMPTY bucket after them
  const bool known = s_tail_known;
  volatile K* v_key = s_key;  // inserts add nodes while others walk the chains
  volatile uint16_t* v_next = s_next;
  // The node of chain [from, to) that holds key k, or kNil.
  auto walk = [&](unsigned from, unsigned to, K k) -> unsigned {
    for (unsigned c = from; c != to; c = v_next[c])
      if (v_key[c] == k) return c;
    return kNil;
  };
  // The bucket of a node of the slice or its tail.
  auto bucket = [&](unsigned m) -> P* {
    return m < SB ? a.table + base + m : a.table + ((base + SB + s_tail_at[m - TAIL]) & tmask);
  };
  unsigned done = 0, maxd = 0;

  if constexpr (FIND) {
    FoundRec<V>* rec = static_cast<FoundRec<V>*>(recs);
    for (unsigned c0 = 0; c0 < cnt; c0 += U * T) {
      if (c0) fetch(c0);
      unsigned rank[U];
      V val[U];
      __syncthreads();  // `left` is this bin's own storage: these records are read, earlier ones written over
#pragma unroll
      for (unsigned u = 0; u < U; ++u) {
        rank[u] = ~0u;
        if (c0 + u * T + tid < cnt) {
          const unsigned h = home_of(key[u]);
          const K at_home = s_key[h];
          unsigned m = h;
          if (at_home != key[u]) {
            m = kNil;
            if (at_home != EMPTY) {
              m = walk(s_head[h % HEADS], kNil, key[u]);
              if (m == kNil && !known && h >= last) leave(key[u], pay[u]);
            }
          }
          if (m != kNil) {
            val[u] = s_val[m];
            rank[u] = atomicAdd(&s_region[pay[u] >> region_log], 1u);
          }
        }
      }
      __syncthreads();
      if (tid < kMaxRegions) {
        const unsigned c = s_region[tid];
        if (c) s_region[tid] = atomicAdd(rec_count + tid, c);
      }
      __syncthreads();
#pragma unroll
      for (unsigned u = 0; u < U; ++u) {
        if (rank[u] == ~0u) continue;
        const unsigned r = pay[u] >> region_log;
        FoundRec<V> f;
        f.idx = pay[u];
        f.val = val[u];
        rec[((uint64_t)r << region_log) + s_region[r] + rank[u]] = f;
      }
      if (c0 + U * T < cnt) {
        __syncthreads();
        if (tid < kMaxRegions) s_region[tid] = 0;
      }
    }
  } else if constexpr (OP == BulkOp::ERASE) {
    for (unsigned c0 = 0; c0 < cnt; c0 += U * T) {
      if (c0) fetch(c0);
      __syncthreads();  // as above
#pragma unroll
      for (unsigned u = 0; u < U; ++u) {
        if (c0 + u * T + tid < cnt) {
          const unsigned h = home_of(key[u]);
          const unsigned m = v_key[h] == key[u] ? h : walk(s_head[h % HEADS], kNil, key[u]);
          if (m != kNil) {  // a key repeated in the batch is erased once
            if (smem_cas(s_key + m, key[u], TOMB) == key[u]) {
              bucket(m)->first = TOMB;
              ++done;
            }
          } else if (!known && h >= last) {
            leave(key[u], Y{});
          }
        }
      }
    }
  } else {
    for (unsigned c0 = 0; c0 < cnt; c0 += U * T) {
      if (c0) fetch(c0);
#pragma unroll
      for (unsigned u = 0; u < U; ++u) {
        const unsigned i = c0 + u * T + tid;
        bool wait = false;
        if (i < cnt) {
          const K k = key[u];
          const unsigned h = home_of(k);
          const K was = smem_cas(s_key + h, EMPTY, k);
          if (was == EMPTY) {
            P pr;
            pr.first = k;
            pr.second = pay[u];
            a.table[base + h] = pr;
            atomicAnd(&s_empty[h / 32], ~(1u << (h % 32)));
            ++done;
            maxd = max(maxd, 1u);
          } else if (was == k) {
            a.table[base + h].second = pay[u];
          } else {
            wait = true;
            s_key[NEW + i] = k;
          }
        }
        const unsigned waits = __ballot_sync(0xffffffffu, wait);
        unsigned q = 0;
        if (lane == 0 && waits) q = atomicAdd(&s_queued, __popc(waits));
        q = __shfl_sync(0xffffffffu, q, 0);
        if (wait) s_queue[q + __popc(waits & ((1u << lane) - 1u))] = (uint16_t)i;
      }
    }
    __syncthreads();
    const unsigned queued = s_queued;
    for (unsigned q = tid; q < queued; q += T) {
      const unsigned i = s_queue[q];
      const K k = s_key[NEW + i];
      const Y y = pays[i];
      const unsigned h = home_of(k);
      unsigned* head = &s_head[h % HEADS];
      unsigned seen = *const_cast<volatile unsigned*>(head);
      unsigned m = walk(seen, kNil, k);
      while (m == kNil) {  // join the chain, unless the key has joined it meanwhile
        s_next[NEW + i] = (uint16_t)seen;
        __threadfence_block();
        const unsigned now = atomicCAS(head, seen, NEW + i);
        if (now == seen) break;
        m = walk(now, seen, k);
        seen = now;
      }
      if (m < NEW) {
        bucket(m)->second = y;
      } else if (m == kNil) {  // the first EMPTY bucket from its home on
        unsigned w = h / 32, mask = ~0u << (h % 32);
        for (;;) {
          const unsigned free = *const_cast<volatile unsigned*>(&s_empty[w]) & mask;
          if (free) {
            const unsigned at = w * 32 + __ffs(free) - 1, bit = free & (0u - free);
            const bool won = smem_cas(s_key + at, EMPTY, k) == EMPTY;
            atomicAnd(&s_empty[w], ~bit);
            if (won) {
              P pr;
              pr.first = k;
              pr.second = y;
              a.table[base + at] = pr;
              ++done;
              maxd = max(maxd, at - h + 1);
              break;
            }
          } else {
            if (++w == SB / 32) {
              leave(k, y);
              break;
            }
            mask = ~0u;
          }
        }
      }
    }
  }
  done = __reduce_add_sync(0xffffffffu, done);
  maxd = __reduce_max_sync(0xffffffffu, maxd);
  if (lane == 0) {
    if (done) atomicAdd(&s_done, done);
    if (maxd) atomicMax(&s_max, maxd);
  }
  __syncthreads();
  if (tid == 0) {
    if constexpr (INS) {
      if (s_done) atomicAdd(&a.info->fill, (unsigned long long)s_done);
      if (s_max) atomicMax(&a.info->max_probe, s_max);
    } else if (s_done) {
      atomicAdd(&a.info->tombstones, (unsigned long long)s_done);
      atomicAdd(&a.info->fill, 0ull - (unsigned long long)s_done);
    }
    left.count[s] = s_left | (known ? 0u : kLeftProbe);
  }
}

// The keys that their slice could not take or decide: one warp per slice. Keys to
// insert whose slice has no EMPTY bucket from their home on, and that are nowhere in
// the table, share one walk from the slice's end: as many of them as there are EMPTY
// buckets in the window take those at once. The others probe from home, 8 lanes per
// key (128 bytes of buckets a step: such probes start near the end of a long run).
template <class P, BulkOp OP>
__global__ void __launch_bounds__(256) k_bulk_left(BulkArgs<P> a, BulkBins left, unsigned slices) {
  using K = typename PairTraits<P>::K;
  using V = typename PairTraits<P>::V;
  using Y = typename BulkPay<P, OP>::T;
  constexpr int G = 8, B = 16 / sizeof(P);
  const int lane = threadIdx.x & 31;
  const unsigned s = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  if (s >= slices) return;
  const unsigned word = left.count[s], cnt = word & ~kLeftProbe;
  if (cnt == 0) return;
  const K* keys = static_cast<const K*>(left.keys) + (uint64_t)s * left.room;
  const Y* pays = static_cast<const Y*>(left.pay) + (OP == BulkOp::ERASE ? 0 : (uint64_t)s * left.room);
  BulkCounts c;
  if (OP == BulkOp::INSERT && !(word & kLeftProbe)) {
    const uint32_t tmask = (1u << a.sp) - 1u, end = (s + 1) << slice_log<P>();
    unsigned next = 0;  // keys [0, next) are placed
    for (uint64_t d = 0; next < cnt; d += 32) {
      if (d > tmask) {  // the table is full
        c.fail = true;
        break;
      }
      P* b = a.table + ((end + (uint32_t)d + lane) & tmask);
      K ek[1];
      V ev[1];
      load_buckets<1>(b, ek, ev);
      bool free = ek[0] == PairTraits<P>::EMPTY;
      for (;;) {
        const unsigned m = __ballot_sync(0xffffffffu, free);
        if (m == 0 || next >= cnt) break;
        // EMPTY bucket number r of the window tries key next + r
        const unsigned i = next + __popc(m & ((1u << lane) - 1u));
        bool won = false;
        K key{};
        V val{};
        if (free && i < cnt) {
          key = keys[i];
          if constexpr (OP == BulkOp::INSERT) val = pays[i];
          won = cas_pair(b, ek[0], ev[0], key, val);
          if (won || ek[0] != PairTraits<P>::EMPTY) free = false;
          if (won) {
            ++c.ins;
            const uint32_t at = (uint32_t)(b - a.table);
            c.maxd = max(c.maxd, ((at - home_slot(key, a.sp)) & tmask) + 1);
          }
        }
        // keys that lost their bucket to another slice's are tried again: move them behind the ones placed
        const unsigned tried = __ballot_sync(0xffffffffu, won || (m >> lane & 1u && i < cnt));
        const unsigned placed = __ballot_sync(0xffffffffu, won);
        if (placed != tried) {
          const unsigned lost = tried & ~placed;
          const unsigned to = next + __popc(placed) + __popc(lost & ((1u << lane) - 1u));
          __syncwarp();
          if (lost >> lane & 1u) {
            const_cast<K*>(keys)[to] = key;
            if constexpr (OP == BulkOp::INSERT) const_cast<Y*>(pays)[to] = val;
          }
          __syncwarp();
        }
        next += __popc(placed);
      }
    }
  } else {
    const unsigned limit = OP == BulkOp::INSERT ? 0u : a.info->max_probe;
    const unsigned gmask = group_mask<G>(lane);
    for (unsigned i = lane / G; i < cnt; i += 32 / G) {
      const K key = keys[i];
      if constexpr (OP == BulkOp::INSERT) {
        unsigned d1 = 0;
        const int r = probe_insert_live<P, G, B>(a.table, a.sp, key, pays[i], lane, gmask, d1);
        if (d1) {
          ++c.ins;
          c.maxd = max(c.maxd, d1);
        }
        if (r == PR_FAIL) c.fail = true;
      } else {
        uint32_t slot;
        V v;
        const int w = probe_find<P, G, B>(a.table, a.sp, key, limit, lane, gmask, slot, v);
        if (w >= 0 && (lane & (G - 1)) == w) {
          if constexpr (OP == BulkOp::ERASE) {
            if (cas_key(a.table + slot, key, PairTraits<P>::TOMB)) ++c.erased;
          } else {
            a.out[(uint64_t)pays[i] * a.out_stride] = v;
          }
        }
      }
    }
    __syncwarp();
  }
  bulk_publish(a.info, c, lane);
}

// The values found to their output elements, region by region.
constexpr unsigned kScatterRecs = 4096;  // per CTA of 256 threads
template <class P>
__global__ void __launch_bounds__(256) k_bulk_scatter(BulkArgs<P> a, const void* recs, const unsigned* rec_count,
                                                      int region_log, unsigned parts) {
  using V = typename PairTraits<P>::V;
  const unsigned r = blockIdx.x / parts;
  const unsigned first = blockIdx.x % parts * kScatterRecs;
  const unsigned cnt = rec_count[r];
  if (first >= cnt) return;
  const unsigned end = min(cnt, first + kScatterRecs);
  const FoundRec<V>* rec = static_cast<const FoundRec<V>*>(recs) + ((uint64_t)r << region_log);
#pragma unroll 4
  for (unsigned i = first + threadIdx.x; i < end; i += 256) {
    const FoundRec<V> f = rec[i];
    a.out[(uint64_t)f.idx * a.out_stride] = f.val;
  }
}

}  // namespace hx
