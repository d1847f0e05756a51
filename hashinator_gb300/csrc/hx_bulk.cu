// hx_bulk.cu — host side of the slice-by-slice batches (hx_bulk.cuh).
#include <cmath>

#include "hx_bulk.cuh"
#include "hx_host.h"
#include "hx_internal.h"

namespace hx {

// Room of a bin that gets `mean` of the batch's keys on average: eight standard
// deviations of a random spread above it, so that with keys that hash evenly no
// bin ever fills.
static unsigned bulk_bin_room(uint64_t mean) {
  const double r = (double)mean + 8.0 * std::sqrt((double)mean) + 64.0;
  return ((unsigned)r + 31u) & ~31u;
}

static int log2_ceil(uint64_t x) {
  int l = 0;
  while ((1ull << l) < x) ++l;
  return l;
}

constexpr uint64_t kBulkChunk = 1ull << 27;  // keys of one batch at a time: bounds the scratch

// Scratch of one batch of n records of which `expected` hold keys, in the order
// [counts][bins of the second split][bins of the first split / left records / found records].
template <class P, BulkOp OP>
struct BulkPlan {
  using K = typename PairTraits<P>::K;
  using V = typename PairTraits<P>::V;
  int log1 = 0, log2 = 0;  // digits of the two splits; log1 = 0: one split
  unsigned room1 = 0, room2 = 0;
  int region_log = 0;
  unsigned regions = 0;
  uint64_t count_words = 0, bin_records = 0, total = 0;
  uint64_t at_keys2 = 0, at_pay2 = 0, at_keys1 = 0, at_pay1 = 0;
  static constexpr unsigned kPay = OP == BulkOp::ERASE ? 0 : sizeof(typename BulkPay<P, OP>::T);

  BulkPlan(int sp, uint64_t n, uint64_t expected) {
    const int bits = sp - slice_log<P>();
    log2 = bits <= kMaxDigitLog ? bits : bits / 2;
    log1 = bits - log2;
    const uint64_t slices = 1ull << bits;
    room2 = bulk_bin_room(expected >> bits);
    room1 = log1 ? bulk_bin_room(expected >> log1) : 0;
    if (OP == BulkOp::FIND) {
      region_log = log2_ceil(n) - kRegionLog;
      if (region_log < 10) region_log = 10;
      regions = (unsigned)((n + (1ull << region_log) - 1) >> region_log);
    }
    count_words = slices * 2 + (1ull << log1) + kMaxRegions;  // bins, left, first split, found
    auto up = [](uint64_t b) { return (b + 255) / 256 * 256; };
    const uint64_t rec2 = slices * room2, rec1 = (uint64_t)room1 << log1;
    // the second buffer holds the first split's bins, then the left records of inserts
    // (as many as the bins may hold) or the values found
    const uint64_t recb = OP == BulkOp::INSERT && rec2 > rec1 ? rec2 : rec1;
    uint64_t at = up(count_words * 4);
    at_keys2 = at;
    at += up(rec2 * sizeof(K));
    at_pay2 = at;
    at += up(rec2 * kPay);
    at_keys1 = at;
    uint64_t second;
    if (OP == BulkOp::FIND) {
      second = up(rec1 * sizeof(K)) + up(rec1 * kPay);
      const uint64_t found = up(((uint64_t)regions << region_log) * sizeof(FoundRec<V>));
      at_pay1 = at + up(rec1 * sizeof(K));
      if (found > second) second = found;
    } else {
      second = up(recb * sizeof(K)) + up(recb * kPay);
      at_pay1 = at + up(recb * sizeof(K));
    }
    total = at + second;
  }
};

template <class Kern>
static cudaError_t allow_smem(Kern kern, size_t smem) {
  return smem > 32 * 1024 ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
                          : cudaSuccess;
}

template <class P, BulkOp OP, BulkSrc SRC>
static hx_status launch_split(const BulkArgs<P>& a, const BulkBins& in, const BulkBins& out, unsigned bins_in,
                              uint64_t records, int shift, int log_digits, cudaStream_t s) {
  auto kern = k_bulk_split<P, OP, SRC>;
  const size_t smem = (size_t)bulk_tile<P, OP>() * bulk_record_bytes<P, OP>();
  HX_CUDA(allow_smem(kern, smem));
  const unsigned tiles = (unsigned)((records + bulk_tile<P, OP>() - 1) / bulk_tile<P, OP>());
  kern<<<tiles * bins_in, kBulkThreads, smem, s>>>(a, in, out, tiles, shift, log_digits);
  return after_launch();
}

template <class P, BulkOp OP>
static hx_status bulk_chunk(const BulkArgs<P>& a, BulkSrc src, uint64_t expected, char* scratch, cudaStream_t s) {
  const BulkPlan<P, OP> pl(a.sp, a.n, expected);
  const int bits = pl.log1 + pl.log2;
  const unsigned slices = 1u << bits;
  unsigned* counts = reinterpret_cast<unsigned*>(scratch);
  HX_CUDA(cudaMemsetAsync(counts, 0, pl.count_words * 4, s));
  BulkBins fine{scratch + pl.at_keys2, scratch + pl.at_pay2, counts, pl.room2, bits};
  // inserts read a bin more than once, so what is left of it goes to the first split's room;
  // the others write it over the part of the bin that they have read
  BulkBins left{scratch + (OP == BulkOp::INSERT ? pl.at_keys1 : pl.at_keys2),
                scratch + (OP == BulkOp::INSERT ? pl.at_pay1 : pl.at_pay2), counts + slices, pl.room2, bits};
  BulkBins coarse{scratch + pl.at_keys1, scratch + pl.at_pay1, counts + 2ull * slices, pl.room1, pl.log1};
  unsigned* found = counts + 2ull * slices + (1u << pl.log1);
  const BulkBins none{};
  const BulkBins& to = pl.log1 ? coarse : fine;
  const int shift1 = slice_log<P>() + (pl.log1 ? pl.log2 : 0), digits1 = pl.log1 ? pl.log1 : pl.log2;
  hx_status st;
  if (src == BulkSrc::PAIRS) st = launch_split<P, OP, BulkSrc::PAIRS>(a, none, to, 1, a.n, shift1, digits1, s);
  else if (src == BulkSrc::INDEX && OP == BulkOp::INSERT)
    st = launch_split<P, OP, OP == BulkOp::INSERT ? BulkSrc::INDEX : BulkSrc::KEYS>(a, none, to, 1, a.n, shift1,
                                                                                   digits1, s);
  else st = launch_split<P, OP, BulkSrc::KEYS>(a, none, to, 1, a.n, shift1, digits1, s);
  if (st != HX_OK) return st;
  if (pl.log1) {
    st = launch_split<P, OP, BulkSrc::BINS>(a, coarse, fine, 1u << pl.log1, pl.room1, slice_log<P>(), pl.log2, s);
    if (st != HX_OK) return st;
  }
  auto kern = k_bulk_slice<P, OP>;
  void* recs = scratch + pl.at_keys1;
  HX_CUDA(allow_smem(kern, slice_smem<P, OP>()));
  kern<<<slices, kSliceThreads, slice_smem<P, OP>(), s>>>(a, fine, left, recs, found, pl.region_log);
  if ((st = after_launch()) != HX_OK) return st;
  if constexpr (OP == BulkOp::FIND) {
    const unsigned parts = (unsigned)(((1ull << pl.region_log) + kScatterRecs - 1) / kScatterRecs);
    k_bulk_scatter<P><<<pl.regions * parts, 256, 0, s>>>(a, recs, found, pl.region_log, parts);
    if ((st = after_launch()) != HX_OK) return st;
  }
  k_bulk_left<P, OP><<<(slices + 7) / 8, 256, 0, s>>>(a, left, slices);
  return after_launch();
}

template <class P, BulkOp OP>
static hx_status bulk_run(BulkArgs<P> a, BulkSrc src, uint64_t expected, cudaStream_t s, bool* done) {
  *done = false;
  const uint64_t n = a.n;
  uint64_t chunk = n < kBulkChunk ? n : kBulkChunk;
  if (OP == BulkOp::INSERT) {  // a bin's new keys are sorted in shared memory
    uint64_t mean = bin_room_max<P>();
    while (bulk_bin_room(mean) > bin_room_max<P>()) mean -= 32;
    const double share = (double)(mean << (a.sp - slice_log<P>())) / (double)expected;  // of the batch, at once
    if (share < 1.0) {
      const uint64_t pieces = (uint64_t)std::ceil(1.0 / share);
      const uint64_t most = (n + pieces - 1) / pieces;
      if (chunk > most) chunk = most;
    }
  }
  const uint64_t exp1 = expected < n ? (uint64_t)((double)expected * ((double)chunk / (double)n)) : chunk;
  const BulkPlan<P, OP> pl(a.sp, chunk, exp1);
  void* scratch = nullptr;
  if (pool_alloc(&scratch, pl.total, s) != cudaSuccess) {
    cudaGetLastError();  // no room for the scratch: the caller probes directly
    return HX_OK;
  }
  hx_status st = HX_OK;
  const BulkArgs<P> all = a;
  for (uint64_t at = 0; at < n && st == HX_OK; at += chunk) {
    a.n = n - at < chunk ? n - at : chunk;
    a.first = all.first + at;
    if (all.keys) a.keys = all.keys + at;
    if (all.vals) a.vals = all.vals + at;
    if (all.pairs) a.pairs = all.pairs + at;
    if (all.out) a.out = all.out + at * all.out_stride;
    st = bulk_chunk<P, OP>(a, src, exp1, static_cast<char*>(scratch), s);
  }
  *done = true;
  HX_CUDA(pool_free(scratch, s));
  return st;
}

// The rule: a batch goes slice by slice if it has at least one key per `spread`
// buckets. A slice costs the same however few of its buckets the batch asks for, and
// probing directly costs more the fuller the table is and the less of it stays in L2
// (128 MiB of it do); a look-up costs more here than an insert or an erase, as its
// value has to go back to its place. Measured on GB300, direct time over slice time
// for u32 / u64 tables (of the size in brackets, for one key per so many buckets):
//   load factor 0.5:  insert [128 MiB] 1/2 1.28 / 1.22, [256] 1/4 1.49 / 1.13; erase
//                     [256] 1/4 1.5 / 1.2; look-up [256] 1/2 0.92 / 0.86, [1 GiB] 1/2
//                     1.40 / 1.00, [2 GiB] 1.16 (u64)
//   load factor 0.72: insert [128] 1/5 0.86 / 0.73, [256] 1/5 1.34 / 1.18; erase [256]
//                     1/18 1.20 / 1.04; look-up [256] 1/3 0.92 / 0.94, [512] 1.31 (u64)
//   load factor 0.8:  look-up [256] 1/3 1.20 / 1.3
//   load factor 0.86: insert [128] 1/5 1.20 / 1.46, [32] 1/5 1.08 / 1.85; erase [128]
//                     1/15 1.34 / 1.62; look-up [128] 1/5 1.0 / 1.34, [256] 1/5 1.45 / 2.4
//   load factor 0.92: insert [32] 1/4 2.0 / 4.1; erase [32] 1/14 2.8 / 5.4; look-up
//                     [32] 1/4 2.1 / 2.2, [128] 2.2 / 3.3
// What the host cannot tell, direct time over slice time. Look-ups of keys all absent /
// half / all present, load factor 0.5: u32 [512 MiB] 1.48 / 1.08 / 0.99, [1 GiB] 1.81 /
// 1.29 / 1.12; u64 [2 GiB] 1.78 / 1.09 / 0.86, [4 GiB] 1.81 / 1.11 / 0.88. Batches that do
// not spread over the table (2^26 u32 keys, 2^27 buckets): every second key the same,
// insert 4.5, look-up 0.73, erase 1.7; zipf(1) 5.8 / 0.79 / 1.7; 1024 distinct keys 2.5 /
// 0.71 / 2.1; keys in bucket order 0.54 / 0.99 / 0.44. A rehash of 2^27 u64 buckets 1.14
// with keys spread over 64 bits, 0.86 with keys below 2^(64 - sp), whose old and new
// buckets are in one order.
// The load factor is the host's bound of it (after the inserts of this call); a bound
// above the table's size says nothing, and counts as a low one.
static unsigned bulk_spread(BulkOp op, bool p32, uint64_t bytes, double lf) {
  const uint64_t mib = bytes >> 20;
  if (mib < 16) return 0;
  if (op == BulkOp::FIND) {
    if (lf >= 0.9) return mib >= 128 ? 16 : 4;
    if (lf >= 0.85) return mib >= 256 ? 6 : (mib >= 128 ? 4 : (p32 ? 0 : 2));
    if (lf >= 0.75) return mib >= 256 ? 3 : 0;
    return mib >= (p32 ? 512 : 2048) ? 2 : 0;
  }
  if (op == BulkOp::ERASE) {
    if (lf >= 0.85) return 16;
    if (lf >= 0.7) return mib >= 256 ? 16 : (mib >= 128 ? 8 : 0);
    return mib >= 256 ? 8 : (mib >= 128 ? 4 : 0);
  }
  if (lf >= 0.85) return mib >= 512 ? 16 : (mib >= 128 ? 6 : (lf >= 0.88 ? 4 : 0));
  if (lf >= 0.7) return mib >= 512 ? 8 : (mib >= 128 ? 4 : 0);
  return mib >= 128 ? 4 : 0;
}
static bool bulk_pays(const BulkCall& c) {
  const uint64_t slots = 1ull << c.sp, bytes = (uint64_t)(c.key_bytes * 2) << c.sp;
  const int bits = c.sp - (c.key_bytes == 4 ? slice_log<P32>() : slice_log<P64>());
  if (bits < 1 || bits > 2 * kMaxDigitLog) return false;
  const double lf = c.fill_bound <= slots ? (double)c.fill_bound / (double)slots : 0.0;
  const unsigned spread = bulk_spread(c.op, c.key_bytes == 4, bytes, lf);
  return spread && c.expected >= slots / spread;
}

bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return cs != cudaStreamCaptureStatusNone;
}

template <class P>
static hx_status bulk_typed(const BulkCall& c, cudaStream_t s, bool* done) {
  using K = typename PairTraits<P>::K;
  using V = typename PairTraits<P>::V;
  BulkArgs<P> a{};
  a.table = static_cast<P*>(c.table);
  a.sp = c.sp;
  a.info = c.info;
  a.keys = static_cast<const K*>(c.keys);
  a.vals = static_cast<const V*>(c.vals);
  a.pairs = static_cast<const P*>(c.pairs);
  a.n = c.n;
  a.out_stride = c.pairs ? 2 : 1;
  a.out = c.pairs ? reinterpret_cast<V*>(static_cast<P*>(c.out)) + 1 : static_cast<V*>(c.out);
  const BulkSrc src = c.pairs ? BulkSrc::PAIRS : (c.op == BulkOp::INSERT && !c.vals ? BulkSrc::INDEX : BulkSrc::KEYS);
  if (c.op != BulkOp::FIND) a.out = nullptr;
  switch (c.op) {
    case BulkOp::INSERT: return bulk_run<P, BulkOp::INSERT>(a, src, c.expected, s, done);
    case BulkOp::FIND: return bulk_run<P, BulkOp::FIND>(a, src, c.expected, s, done);
    default: return bulk_run<P, BulkOp::ERASE>(a, src, c.expected, s, done);
  }
}

hx_status bulk_try(const BulkCall& c, cudaStream_t s, bool* done) {
  *done = false;
  if (!bulk_pays(c) || capturing(s)) return HX_OK;
  return c.key_bytes == 4 ? bulk_typed<P32>(c, s, done) : bulk_typed<P64>(c, s, done);
}

}  // namespace hx
