// hx_stream.cuh — phase-partitioned streaming kernels: stable stream
// compaction (copy_if, extractPattern) and the
// exclusive u32 scan, for 16-byte-aligned inputs.
//
// Header-only so that the drop-in C++ header can instantiate the same
// compaction for a caller's own `Rule` functor in the caller's translation
// unit; libhx instantiates it for its predicate descriptors.
//
// Shape. One cooperative launch of G co-resident CTAs (G = resident CTAs per
// SM x SMs). The input is cut into slices (one stage of shared memory); phase p
// gives slice p*G + b to CTA b, so a phase is G consecutive slices. Each CTA
// keeps STAGES slices in flight, each filled by one bulk copy (cp.async.bulk,
// completion on an mbarrier).
//   pass 1, phase p: read the slice from shared memory, evaluate the rule (or
//     sum, for the scan), write the CTA-local result back into the same stage
//     (the selected elements packed at the front, or the local exclusive
//     sums), and publish the CTA's count for phase p in a slot of scratch.
//   pass 2, of an earlier phase: read every CTA's count of that phase, which
//     by then are almost always published, add up those of the CTAs before
//     this one and of all earlier phases, write the stage's result to global
//     memory at that offset, and refill the stage with a later slice.
// So the input is read once, the output written once, and the only exchange
// between CTAs is one count per CTA per phase, whose latency is hidden behind
// other phases instead of sitting on every tile's critical path as in a
// decoupled look-back.
//
// Compaction: two groups of 256 threads select, each from every second slice,
// and 384 threads write out what they packed. Pass 1 is a chain of dependent
// steps (load, rule, ranks, barrier, pack) that leaves most issue slots empty:
// with 16 warps in step the SM issued 1.75 instructions a cycle and DRAM stood
// at 42%. Two groups fill each other's waits, and the write-out of one phase no
// longer waits for pass 1 of the next. 2^28 u32, 1 / 25 / 50 / 75 / 99 of 100
// selected: 304 / 340 / 373 / 419 / 473 us with every thread in both passes,
// 280 / 305 / 332 / 366 / 420 so. Pairs out of 2^27 buckets: 371 -> 331 us. A caller's
// rule that computes much gains nothing and can lose: 2^27 u32 by 32 hash rounds 1.15 ->
// 1.22 ms, by sinf, expf, logf and cosf 0.90 -> 1.13 ms; fewer writers, for more registers
// a thread, do not help it (1.10 - 1.17 ms with 128 - 256).
//
// Co-residency: every CTA waits for the counts of every other, so the launch
// is cooperative (the runtime guarantees all CTAs resident). Every wait is
// still bounded: an mbarrier wait or a count wait that runs out (about one
// second) sets the scratch error word; every CTA that sees the error word
// stops, waits (bounded) for the bulk copies it issued, and returns.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <map>
#include <mutex>
#include <type_traits>
#include <utility>

namespace hxs {

// ---- PTX helpers --------------------------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
constexpr unsigned long long kWaitNs = 1000000000ull;  // about one second per wait
// Waits for the phase of `bar` with `parity`; false after about a second.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long t0 = globaltimer();
  for (unsigned i = 0; i < (1u << 26); ++i) {
    if (mbar_try(bar, parity)) return true;
    if ((i & 255) == 255 && globaltimer() - t0 > kWaitNs) return false;
  }
  return false;
}
// One bulk copy of `bytes` (a multiple of 16, both addresses 16-byte aligned)
// from global into shared memory, completing `bytes` transactions on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// A barrier of `threads` threads of the CTA, and the same with an OR over them.
__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ bool bar_or(int id, int threads, bool p) {
  unsigned r;
  asm volatile(
      "{\n .reg .pred a, b;\n setp.ne.u32 a, %3, 0;\n barrier.cta.red.or.pred b, %1, %2, a;\n selp.u32 %0, 1, 0, b;\n}\n"
      : "=r"(r)
      : "r"(id), "r"(threads), "r"((unsigned)p)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_relaxed_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned warp_incl_scan(unsigned x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// ---- geometry and scratch -------------------------------------------------
// The compaction's. Threads of a CTA: kPack that select, in kGroups groups, and kWrite
// that write out. 2^28 u32, 1 / 50 / 99 of 100 selected, in us, and pairs of 2^27 buckets:
//   1 group, 64 KiB slices, 3 stages, D 1, 256 writers   294 / 341 / 407, 351
//   2 groups, 32 KiB, 6 stages, D 3, 256 writers         268 / 341 / 443, 311
//   2 groups, 32 KiB, 6 stages, D 3, 384 writers         280 / 332 / 420, 331  (this)
//   2 groups, 32 KiB, 6 stages, D 1, 256 writers         well behind: a count is published too late
//   512 writers (64 registers a thread)                  305 / 399 / 447, 360
//   3 groups of 256, 6 stages                            276 / 353 / 468, 323
#ifndef HX_STREAM_BLOCK
#define HX_STREAM_BLOCK 896
#endif
#ifndef HX_STREAM_WRITERS
#define HX_STREAM_WRITERS 384
#endif
#ifndef HX_STREAM_GROUPS
#define HX_STREAM_GROUPS 2
#endif
#ifndef HX_STREAM_R
#define HX_STREAM_R 8  // uint4 per selecting thread per slice: 256 threads x 8 x 16 B = 32 KiB slices
#endif
#ifndef HX_STREAM_STAGES
#define HX_STREAM_STAGES 6
#endif
#ifndef HX_STREAM_DEFER
#define HX_STREAM_DEFER 3
#endif
#ifndef HX_STREAM_LANE_CHUNKS
#define HX_STREAM_LANE_CHUNKS 0  // compaction: each lane owns kR consecutive uint4s (see the kernel)
#endif
constexpr int kBlock = HX_STREAM_BLOCK;
constexpr int kWrite = HX_STREAM_WRITERS;
constexpr int kPack = kBlock - kWrite;
constexpr int kGroups = HX_STREAM_GROUPS;
constexpr int kGroup = kPack / kGroups;  // threads that select from one slice
constexpr int kWriteBar = 1 + kGroups;   // the writers' barrier; group g has barrier 1 + g, the CTA barrier 0
static_assert(kWrite % 32 == 0 && kWrite > 0 && kPack % (32 * kGroups) == 0 && kPack > 0 && kBlock <= 1024, "whole warps");
static_assert(kGroup <= 1024 && kWriteBar < 16, "one barrier per group, one warp scan over a group's warps");
constexpr int kR = HX_STREAM_R;
constexpr int kStages = HX_STREAM_STAGES;
constexpr int kDefer = HX_STREAM_DEFER;
constexpr bool kLaneChunks = HX_STREAM_LANE_CHUNKS != 0;
static_assert(kStages % kGroups == 0, "a stage belongs to one group");
static_assert(kDefer >= 1 && kDefer < kStages, "a stage must be free to load while D phases wait");
// Count slots per CTA. A CTA publishes its count of phase p once its own writers are
// done with p - 1 - D, for which they read every CTA's count of that phase; so every
// CTA has published p - 1 - D, and every CTA's writers are done with p - 2 - 2D. The
// row of phase p is the row of phase p - kSlots, so kSlots = 2D + 2.
constexpr int kSlots = 2 * kDefer + 2;
constexpr int kMaxGrid = 512;  // CTAs at most (GB300: 152); a larger device runs 512
constexpr int kSlotLoads = (kMaxGrid + kWrite - 1) / kWrite;  // count slots each writer reads per phase
constexpr unsigned kSliceBytes = kGroup * kR * 16;

// Scratch: [error word u32][pad .. 256 B][count slots u64, rows of one per CTA].
// The launcher zeroes the part it uses: one row per phase, at most kSlots.
// 32 B per 64 KiB of input, for at most 1024 of those, hold the scan's 4 rows of one
// slot per 64 KiB slice. They hold the compaction's rows too: one row of 8 B per 32 KiB
// slice when there is one phase, and when there are P > 1 on G CTAs, min(P, 8) rows of
// G slots, against more than (P - 1) G slices.
constexpr uint64_t kScratchBytes = 256 + 32ull * 1024;
static_assert(8ull * kSlots * kMaxGrid <= 32ull * 1024, "the compaction's slots fit");
// Scratch a pass over n elements of elem_bytes each needs.
inline uint64_t scratch_need(uint64_t n, unsigned elem_bytes) {
  uint64_t units = (n * elem_bytes + 65535) / 65536;
  if (units < 1) units = 1;
  if (units > 1024) units = 1024;
  return 256 + 32 * units;
}

struct Scratch {
  unsigned* error;
  unsigned long long* slots;
};
inline Scratch carve(void* p) {
  Scratch s;
  s.error = reinterpret_cast<unsigned*>(p);
  s.slots = reinterpret_cast<unsigned long long*>(static_cast<char*>(p) + 256);
  return s;
}

// What a selected element writes: the element, or only the key of a pair.
template <class T, class O>
__device__ __forceinline__ O project(const T& x) {
  if constexpr (std::is_same<T, O>::value) return x;
  else return x.first;
}

// Selector concept (compaction): a copyable struct with
//   __device__ bool operator()(const T& x) const;
//   static constexpr bool kIndexed;    // true: the rule is called as at(x, i), i the element's index
// kIndexed lets a rule depend on where the element sits (a bucket's home).
template <class F>
struct FunctorSel {
  F f;
  static constexpr bool kIndexed = false;
  template <class T>
  __device__ __forceinline__ bool operator()(const T& x) const {
    return f(x);
  }
};
struct ScanSel {  // placeholder selector of the scan
  static constexpr bool kIndexed = false;
  template <class T>
  __device__ __forceinline__ bool operator()(const T&) const {
    return true;
  }
};

struct Done {                              // what the pass reports, and where it starts
  unsigned long long* d_count;              // if set, *d_count = min(total, count_max) (compaction)
  unsigned long long count_max = ~0ull;     // the largest count written to *d_count
  const unsigned long long* base_from = nullptr;  // if set, output starts at out[*base_from] (and
                                                  // the total counts it), after elements placed earlier
  const unsigned long long* n_from = nullptr;     // if set, the input has min(n, *n_from) elements,
                                                  // read on the device (n is then an upper bound)
};

// ---------------------------------------------------------------------------
// The compaction: out[0..c) = the selected elements (projected to O) in input
// order, writes beyond `capacity` dropped, c to *done.d_count.
// ---------------------------------------------------------------------------
template <class T, class O, class Sel>
__global__ void __launch_bounds__(kBlock, 1) k_compact(const T* __restrict__ in, O* __restrict__ out, uint64_t n, Sel sel,
                                                     uint64_t capacity, Done done, Scratch sc) {
  constexpr int E = 16 / sizeof(T);
  constexpr int WARPS = kGroup / 32, WWARPS = kWrite / 32;
  constexpr unsigned SU4 = kGroup * kR;  // uint4 per slice
  constexpr unsigned SE = SU4 * E;      // elements per slice
  static_assert(sizeof(O) <= sizeof(T), "the packed result fits in its stage");
  extern __shared__ __align__(128) uint4 s_stage[];  // kStages x SU4
  __shared__ __align__(8) uint64_t s_full[kStages];     // the stage holds its slice
  __shared__ __align__(8) uint64_t s_packed[kStages];   // the stage holds its packed result
  __shared__ __align__(8) uint64_t s_written[kStages];  // the stage's result is written out
  __shared__ unsigned s_warp[kGroups][2][WARPS];  // by the parity of the group's phases
  __shared__ unsigned s_cnt[kStages];
  __shared__ uint2 s_red[WWARPS];  // per warp: (count before this CTA, phase total), both < 2^32

  // Device-side inputs: the same values for every CTA, so every CTA runs the
  // same phases and none waits on a CTA that skipped.
  if (done.n_from && *done.n_from < n) n = *done.n_from;
  const int lane = threadIdx.x & 31;
  const unsigned G = gridDim.x, b = blockIdx.x;
  const uint64_t full_slices = n / SE;  // slices wholly inside [0, n)
  const unsigned phases = (unsigned)(((n + SE - 1) / SE + G - 1) / G);  // below 2^32 - kDefer (launch)
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&s_packed[s], WARPS);
      mbar_init(&s_written[s], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto next = [](unsigned& i, unsigned m) { i = i + 1 == m ? 0u : i + 1; };

  if (threadIdx.x < kPack) {
    // ---- a selecting group: pass 1 of every kGroups-th phase --------------------
    const unsigned grp = threadIdx.x / kGroup;
    const int warp = (threadIdx.x % kGroup) >> 5;
    unsigned st = grp;    // stage of phase p
    unsigned par = 0;     // parity of the next wait for a full stage, bit per stage
    unsigned buf = 0;
    for (unsigned p = grp; p < phases; p += kGroups) {
      const bool ok = mbar_wait(&s_full[st], (par >> st) & 1u);
      par ^= 1u << st;
      const uint64_t t = (uint64_t)p * G + b;
      const bool whole = t < full_slices;
      const uint64_t e0 = t * SE;
      T x[kR][E];
      uint4* stage = s_stage + (size_t)st * SU4;
      const unsigned wbase = warp * 32 * kR;  // this warp's first uint4 of the slice
      // Where register row r comes from. By default row r of the warp is 32
      // consecutive uint4s, one per lane. With lane chunks (compaction only),
      // lane l owns the kR consecutive uint4s l*kR .. l*kR+kR-1 of the warp's
      // part and row r holds its uint4 (r + l) mod kR: rotated, so that with
      // kR = 8 the 8 lanes of a shared-memory wavefront read 8 different bank
      // groups.
      constexpr bool LANE = kLaneChunks && (kR & (kR - 1)) == 0 && kR * E <= 32;
      auto u_of = [&](int r) -> unsigned {
        if constexpr (LANE) return wbase + lane * kR + ((r + lane) & (kR - 1));
        else return wbase + r * 32 + lane;
      };
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        const unsigned u = u_of(r);
        if (whole) {
          const uint4 q = stage[u];
          memcpy(&x[r][0], &q, 16);
        } else {
#pragma unroll
          for (int q = 0; q < E; ++q) {
            const uint64_t e = e0 + (uint64_t)u * E + q;
            if (e < n) x[r][q] = in[e];
            else memset(&x[r][q], 0, sizeof(T));
          }
        }
      }
      unsigned pre[kR];
      unsigned acc = 0;
      unsigned bits[kR];
      unsigned cnt[kR];
      unsigned lm = 0;  // lane chunks: the lane's selections, bit j*E + q for element q of its uint4 j
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        {
          const uint64_t e = e0 + (uint64_t)u_of(r) * E;
          unsigned m = 0;
          if (whole) {  // block-uniform: no per-element bounds checks in a whole slice
#pragma unroll
            for (int q = 0; q < E; ++q) {
              bool s;
              if constexpr (Sel::kIndexed) s = sel.at(x[r][q], e + q);
              else s = sel(x[r][q]);
              m |= (unsigned)s << q;
            }
          } else {
#pragma unroll
            for (int q = 0; q < E; ++q) {
              const bool in_range = e + q < n;
              bool s = false;
              if (in_range) {
                if constexpr (Sel::kIndexed) s = sel.at(x[r][q], e + q);
                else s = sel(x[r][q]);
              }
              if (s) m |= 1u << q;
            }
          }
          bits[r] = m;
          if constexpr (LANE) lm |= m << (((r + lane) & (kR - 1)) * E);
          cnt[r] = __popc(m);
        }
      }
      unsigned lane_pre = 0;  // lane chunks: selections of the warp's lanes before this one
      if constexpr (LANE) {
        const unsigned c = __popc(lm);
        const unsigned incl = warp_incl_scan(c, lane);
        lane_pre = incl - c;
        acc = __shfl_sync(0xffffffffu, incl, 31);
      } else {
        // Ranks of the selections: a lane's count per uint4 is at most 4 and a
        // warp's sum at most 128, so four uint4s share one 32-bit word as byte
        // lanes with no carries between them: one warp scan per four uint4s.
        constexpr int NW = (kR + 3) / 4;
        unsigned packed_c[NW], incl_w[NW], tot_w[NW];
#pragma unroll
        for (int w = 0; w < NW; ++w) packed_c[w] = 0;
#pragma unroll
        for (int r = 0; r < kR; ++r) packed_c[r / 4] |= cnt[r] << (8 * (r % 4));
#pragma unroll
        for (int w = 0; w < NW; ++w) {
          incl_w[w] = warp_incl_scan(packed_c[w], lane);
          tot_w[w] = __shfl_sync(0xffffffffu, incl_w[w], 31);
        }
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          const unsigned incl = (incl_w[r / 4] >> (8 * (r % 4))) & 0xffu;
          pre[r] = acc + incl - cnt[r];
          acc += (tot_w[r / 4] >> (8 * (r % 4))) & 0xffu;
        }
      }
      if (lane == 0) s_warp[grp][buf][warp] = acc;
      // The one barrier of a phase: the group has read the stage, and has its warps' counts.
      if (bar_or(1 + grp, kGroup, !ok)) {  // a failed wait stops the whole group here
        if (lane == 0) atomicExch(sc.error, 1u);
        return;
      }
      const unsigned wt = lane < WARPS ? s_warp[grp][buf][lane] : 0u;
      const unsigned wincl = warp_incl_scan(wt, lane);
      const unsigned woff = __shfl_sync(0xffffffffu, wincl - wt, warp);
      buf ^= 1u;
      if (warp == 0 && lane == 31) {
        s_cnt[st] = wincl;
        // the row's last readers are done (kSlots); if that wait runs out, the writers' waits do too
        if (p > (unsigned)kDefer) {
          const unsigned w = p - 1 - kDefer;
          mbar_wait(&s_written[w % kStages], (w / kStages) & 1u);
        }
        // publish this CTA's count of phase p, tagged with p + 1
        st_relaxed(sc.slots + (p % kSlots) * G + b, ((unsigned long long)(p + 1) << 32) | wincl);
      }
      // Packing starts together, also for the lane above: without this barrier a 2^28-element
      // copy_if is 3-10% slower (446 -> 497 us at 99 of 100 selected, one group).
      bar_sync(1 + grp, kGroup);
      // the CTA-local result, in place in the stage (every thread has read it)
      {
        O* packed = reinterpret_cast<O*>(stage);
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          if (!bits[r]) continue;  // nothing selected in this uint4: the common case for a sparse rule
          unsigned o;
          if constexpr (LANE) {
            const unsigned jb = ((r + lane) & (kR - 1)) * E;  // first bit of this uint4 in the lane's mask
            o = woff + lane_pre + __popc(lm & ((1u << jb) - 1u));
          } else {
            o = woff + pre[r];
          }
#pragma unroll
          for (int q = 0; q < E; ++q)
            if (bits[r] & (1u << q)) packed[o++] = hxs::project<T, O>(x[r][q]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_packed[st]);
      st += kGroups;
      if (st >= (unsigned)kStages) st -= kStages;
    }
    return;
  }

  // ---- the writing warps: loads ahead, pass 2 of one phase after the other ------
  const unsigned tid = threadIdx.x - kPack;
  const int warp = tid >> 5;
  unsigned issued[kStages];  // thread 0 of them: loads issued per stage
#pragma unroll
  for (int s = 0; s < kStages; ++s) issued[s] = 0;
  // Fill stage st with the slice of phase p: a whole slice by one bulk copy; the
  // ragged last slice and slices past n are read later with plain loads, so their
  // barrier phase completes with no bytes.
  auto issue = [&](unsigned st, unsigned p) {
    const uint64_t t = (uint64_t)p * G + b;
    if (t < full_slices) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // earlier reads of the stage come first
      mbar_expect_tx(&s_full[st], kSliceBytes);
      bulk_load(s_stage + (size_t)st * SU4, in + t * SE, kSliceBytes, &s_full[st]);
    } else {
      mbar_expect_tx(&s_full[st], 0);
    }
#pragma unroll
    for (int s = 0; s < kStages; ++s) issued[s] += (unsigned)(s == (int)st);
  };
  if (tid == 0)
    for (unsigned s = 0; s < (unsigned)kStages && s < phases; ++s) issue(s, s);
  // result count of the phases already written, after any elements placed before this pass
  unsigned long long base = done.base_from ? *done.base_from : 0ull;
  bool failed = false;
  unsigned st = 0, sl = 0, par = 0;
  unsigned long long pv[kSlotLoads];  // the counts of phase q, read ahead while phase q - 1 is written
#pragma unroll
  for (int k = 0; k < kSlotLoads; ++k) pv[k] = 0;  // no phase's tag: read when the wait is over
  for (unsigned q = 0; q < phases; ++q) {
    // Every CTA's count of phase q: the sum over CTAs before this one, and
    // the total. A phase holds at most kMaxGrid slices of at most 2^14
    // elements, so both fit 32 bits.
    const unsigned long long* row = sc.slots + sl * G;
    bool ok = mbar_wait(&s_packed[st], (par >> st) & 1u);
    par ^= 1u << st;
    unsigned before = 0, total = 0;
#pragma unroll
    for (int k = 0; k < kSlotLoads; ++k) {
      const unsigned c = tid + k * kWrite;
      if (c >= G) break;
      unsigned long long v = pv[k];
      if (ok && (unsigned)(v >> 32) != q + 1) v = ld_relaxed(row + c);
      if (ok && (unsigned)(v >> 32) != q + 1) {
        const unsigned long long t0 = globaltimer();
        unsigned i = 0;
        while ((unsigned)(v >> 32) != q + 1) {
          if ((++i & 63) == 0) {
            if (ld_relaxed_u32(sc.error) || globaltimer() - t0 > kWaitNs) {
              ok = false;
              break;
            }
            __nanosleep(64);
          }
          v = ld_relaxed(row + c);
        }
      }
      const unsigned cnt = (unsigned)v;
      total += cnt;
      if (c < b) before += cnt;
    }
    // only the warps that read a slot reduce; the others hold zeros
    const unsigned nw = G >= (unsigned)kWrite ? (unsigned)WWARPS : (G + 31) / 32;
    if ((unsigned)warp < nw) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        before += __shfl_xor_sync(0xffffffffu, before, o);
        total += __shfl_xor_sync(0xffffffffu, total, o);
      }
      if (lane == 0) s_red[warp] = make_uint2(before, total);
    }
    if (bar_or(kWriteBar, kWrite, !ok)) {
      failed = true;
      break;
    }
    next(sl, kSlots);
    if (q + 1 < phases) {
      const unsigned long long* ahead = sc.slots + sl * G;
#pragma unroll
      for (int k = 0; k < kSlotLoads; ++k) {
        const unsigned c = tid + k * kWrite;
        if (c < G) pv[k] = ld_relaxed(ahead + c);
      }
    }
    before = 0;
    total = 0;
    for (unsigned w = 0; w < nw; ++w) {
      const uint2 r = s_red[w];
      before += r.x;
      total += r.y;
    }
    const unsigned long long prefix = base + before;
    const uint4* stage = s_stage + (size_t)st * SU4;
    {
      const O* packed = reinterpret_cast<const O*>(stage);
      unsigned cnt = s_cnt[st];
      if (prefix >= capacity) cnt = 0;
      else if (capacity - prefix < cnt) cnt = (unsigned)(capacity - prefix);
      O* to = out + prefix;
#pragma unroll 8
      for (unsigned i = tid; i < cnt; i += kWrite) to[i] = packed[i];
    }
    base += total;
    bar_sync(kWriteBar, kWrite);  // stage st is written out, s_red is read
    if (tid == 0) {
      mbar_arrive(&s_written[st]);
      if (q + kStages < phases) issue(st, q + kStages);
    }
    next(st, kStages);
  }
  if (failed) {
    if (tid == 0) {
      atomicExch(sc.error, 1u);
      // no copy is issued after a failure: give each one still in flight a
      // bounded wait before the CTA exits
#pragma unroll
      for (int s = 0; s < kStages; ++s)
        if (issued[s]) mbar_wait(&s_full[s], (issued[s] - 1) & 1u);
    }
    return;
  }
  if (b == 0 && tid == 0) {
    if (done.d_count) *done.d_count = base < done.count_max ? base : done.count_max;
  }
}

// ---------------------------------------------------------------------------
// The scan: out[i] = sum of in[0..i) mod 2^32. The same phases, with every
// thread in both passes: it writes as much as it reads and is bound by memory,
// and the split of the compaction below costs it more than it saves (2^28 - 57
// elements, 342 us; with selecting groups and writers apart 347-380 us).
// ---------------------------------------------------------------------------
namespace scan {
constexpr int kR = 8, kStages = 3, kDefer = 1, kSlots = 2 * kDefer + 2;
constexpr unsigned kSliceBytes = 512 * kR * 16;
constexpr int kMaxGrid = 1024;
constexpr int kSlotLoads = (kMaxGrid + 511) / 512;  // count slots each thread reads per phase
}  // namespace scan
template <int kBlock = 512>  // a template only so that every unit that includes this may define it
__global__ void __launch_bounds__(kBlock, 1) k_scan(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                    uint64_t n, Scratch sc) {
  constexpr int E = 4;
  constexpr int WARPS = kBlock / 32;
  constexpr unsigned SU4 = kBlock * scan::kR;  // uint4 per slice
  constexpr unsigned SE = SU4 * E;       // elements per slice
  extern __shared__ __align__(128) uint4 s_stage[];  // scan::kStages x SU4
  __shared__ __align__(8) uint64_t s_bar[scan::kStages];
  __shared__ unsigned s_warp[WARPS];
  __shared__ uint2 s_red[WARPS];  // per warp: (count before this CTA, phase total), both < 2^32
  __shared__ int s_abort;

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned G = gridDim.x, b = blockIdx.x;
  const uint64_t full_slices = n / SE;  // slices wholly inside [0, n)
  const unsigned phases = (unsigned)(((n + SE - 1) / SE + G - 1) / G);  // below 2^32 - scan::kDefer (launch)
  unsigned pend = 0;                    // thread 0: stages with a bulk copy not yet seen complete
  unsigned par = 0;                     // parity of the next wait, bit per stage

  // Fill stage st with the slice of phase p (thread 0): a whole slice by one
  // bulk copy; the ragged last slice and slices past n are read later with
  // plain loads, so their barrier phase completes with no bytes.
  auto issue = [&](int st, unsigned p) {
    const uint64_t t = (uint64_t)p * G + b;
    if (t < full_slices) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // earlier reads of the stage come first
      mbar_expect_tx(&s_bar[st], scan::kSliceBytes);
      bulk_load(s_stage + (size_t)st * SU4, in + t * SE, scan::kSliceBytes, &s_bar[st]);
    } else {
      mbar_expect_tx(&s_bar[st], 0);
    }
    pend |= 1u << st;
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < scan::kStages; ++s) mbar_init(&s_bar[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_abort = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int s = 0; s < scan::kStages && (unsigned)s < phases; ++s) issue(s, s);

  unsigned long long base = 0;  // sum of the phases already written
  bool failed = false;
  // stage and count-slot row of phase p (pass 1) and of phase p - scan::kDefer
  // (pass 2), advanced by one each phase instead of computed by division
  unsigned st1 = 0, st2 = 0, sl1 = 0, sl2 = 0;
  auto next = [](unsigned& i, unsigned m) { i = i + 1 == m ? 0u : i + 1; };
  for (unsigned p = 0; p < phases + scan::kDefer; ++p) {
    // The count slots that pass 2 reads below were published scan::kDefer phases
    // ago: load them now, so that their latency overlaps pass 1.
    unsigned long long pv[scan::kSlotLoads];
    if (p >= (unsigned)scan::kDefer) {
      const unsigned long long* row = sc.slots + sl2 * G;
#pragma unroll
      for (int k = 0; k < scan::kSlotLoads; ++k) {
        const unsigned c = threadIdx.x + k * kBlock;
        pv[k] = c < G ? ld_relaxed(row + c) : 0ull;
      }
    }
    // ---- pass 1: phase p -------------------------------------------------
    if (p < phases) {
      const unsigned st = st1;
      const bool ok = mbar_wait(&s_bar[st], (par >> st) & 1u);
      if (ok) {  // a failed wait leaves par and pend as they were, for the drain below
        par ^= 1u << st;
        pend &= ~(1u << st);
      }
      const uint64_t t = (uint64_t)p * G + b;
      const bool whole = t < full_slices;
      const uint64_t e0 = t * SE;
      uint32_t x[scan::kR][E];
      uint4* stage = s_stage + (size_t)st * SU4;
      const unsigned wbase = warp * 32 * scan::kR;  // this warp's first uint4 of the slice
#pragma unroll
      for (int r = 0; r < scan::kR; ++r) {
        const unsigned u = wbase + r * 32 + lane;
        if (whole) {
          const uint4 q = stage[u];
          memcpy(&x[r][0], &q, 16);
        } else {
#pragma unroll
          for (int q = 0; q < E; ++q) {
            const uint64_t e = e0 + (uint64_t)u * E + q;
            if (e < n) x[r][q] = in[e];
            else x[r][q] = 0;
          }
        }
      }
      if (__syncthreads_or(!ok)) {  // stage st is read; a failed wait stops every thread here
        failed = true;
        break;
      }
      unsigned pre[scan::kR];
      unsigned acc = 0;
#pragma unroll
      for (int r = 0; r < scan::kR; ++r) {
        const unsigned c = x[r][0] + x[r][1] + x[r][2] + x[r][3];
        const unsigned incl = warp_incl_scan(c, lane);
        pre[r] = acc + incl - c;
        acc += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) s_warp[warp] = acc;
      __syncthreads();
      if (warp == 0) {
        const unsigned wt = lane < WARPS ? s_warp[lane] : 0u;
        const unsigned wincl = warp_incl_scan(wt, lane);
        if (lane < WARPS) s_warp[lane] = wincl - wt;
        if (lane == 31) {
          // publish this CTA's sum of phase p (mod 2^32), tagged with p + 1
          st_relaxed(sc.slots + sl1 * G + b, ((unsigned long long)(p + 1) << 32) | wincl);
        }
      }
      __syncthreads();
      // the CTA-local result, in place in the stage (every thread has read it)
      const unsigned woff = s_warp[warp];
#pragma unroll
      for (int r = 0; r < scan::kR; ++r) {
        const unsigned o0 = woff + pre[r], o1 = o0 + x[r][0], o2 = o1 + x[r][1], o3 = o2 + x[r][2];
        stage[wbase + r * 32 + lane] = make_uint4(o0, o1, o2, o3);
      }
    }
    // ---- pass 2: phase p - D ---------------------------------------------
    if (p >= (unsigned)scan::kDefer) {
      const unsigned q = p - scan::kDefer;
      const unsigned st = st2;
      // Every CTA's sum of phase q, mod 2^32: of the CTAs before this one, and of all.
      unsigned before = 0, total = 0;
      bool ok = true;
#pragma unroll
      for (int k = 0; k < scan::kSlotLoads; ++k) {
        const unsigned c = threadIdx.x + k * kBlock;
        if (c >= G) break;
        const unsigned long long* slot = sc.slots + sl2 * G + c;
        unsigned long long v = pv[k];
        if ((unsigned)(v >> 32) != q + 1) {
          const unsigned long long t0 = globaltimer();
          unsigned i = 0;
          while ((unsigned)(v >> 32) != q + 1) {
            if ((++i & 63) == 0) {
              if (ld_relaxed_u32(sc.error) || globaltimer() - t0 > kWaitNs) {
                ok = false;
                break;
              }
              __nanosleep(64);
            }
            v = ld_relaxed(slot);
          }
          if (!ok) break;
        }
        const unsigned cnt = (unsigned)v;
        total += cnt;
        if (c < b) before += cnt;
      }
      // only the warps that read a slot reduce; the others hold zeros
      const unsigned nw = G >= (unsigned)kBlock ? (unsigned)WARPS : (G + 31) / 32;
      if ((unsigned)warp < nw) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          before += __shfl_xor_sync(0xffffffffu, before, o);
          total += __shfl_xor_sync(0xffffffffu, total, o);
        }
        if (lane == 0) s_red[warp] = make_uint2(before, total);
      }
      if (__syncthreads_or(!ok)) {
        failed = true;
        break;
      }
      before = 0;
      total = 0;
      for (unsigned w = 0; w < nw; ++w) {
        const uint2 r = s_red[w];
        before += r.x;
        total += r.y;
      }
      const unsigned long long prefix = base + before;
      const uint4* stage = s_stage + (size_t)st * SU4;
      const uint64_t t = (uint64_t)q * G + b;
      const uint64_t e0 = t * SE;
      const unsigned add = (unsigned)prefix;
      const bool whole = t < full_slices;
      for (unsigned u = threadIdx.x; u < SU4; u += kBlock) {
        const uint4 v = stage[u];
        const uint4 w = make_uint4(v.x + add, v.y + add, v.z + add, v.w + add);
        const uint64_t e = e0 + (uint64_t)u * 4;
        if (whole) {
          __stcs(reinterpret_cast<uint4*>(out + e), w);
        } else {
          const unsigned a[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (e + k < n) out[e + k] = a[k];
        }
      }
      base += total;
      __syncthreads();  // stage st is written out
      if (threadIdx.x == 0 && q + scan::kStages < phases) issue(st, q + scan::kStages);
      next(st2, scan::kStages);
      next(sl2, scan::kSlots);
    }
    next(st1, scan::kStages);
    next(sl1, scan::kSlots);
  }
  if (failed) {
    if (threadIdx.x == 0) {
      atomicExch(sc.error, 1u);
      // no copy is issued after a failure: give each one still in flight a
      // bounded wait before the CTA exits
      for (int s = 0; s < scan::kStages; ++s)
        if ((pend >> s) & 1u) mbar_wait(&s_bar[s], (par >> s) & 1u);
    }
  }
}
// ---- host side -------------------------------------------------------------
// Co-resident CTAs of one kernel on the current device (SMs x CTAs per SM,
// at most max_grid), with the kernel's shared-memory limit raised first.
// The limit is raised on every call (cheap, and it survives a device reset
// that would drop it); the occupancy query runs once per kernel and device.
// The cache is keyed by the kernel's host-side address, not by its template
// arguments alone: a kernel template instantiated in several translation
// units (libhx's, a caller's, the no-allocation scan's) is a separate
// function in each, while a static of an inline function is one object
// shared by all of them.
template <class Kern>
inline cudaError_t resident_grid(Kern kern, int block, size_t smem, int max_grid, unsigned* grid) {
  cudaError_t e = cudaSuccess;
  if (smem > 48 * 1024) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  int dev = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, unsigned> cache;
  const auto key = std::make_pair(reinterpret_cast<const void*>(kern), dev);
  {
    std::lock_guard<std::mutex> g(mu);
    const auto it = cache.find(key);
    if (it != cache.end()) {
      *grid = it->second;
      return cudaSuccess;
    }
  }
  int per_sm = 0, sms = 0;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, smem)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  long g = (long)per_sm * sms;
  if (g < 1) return cudaErrorInvalidConfiguration;
  if (g > max_grid) g = max_grid;
  {
    std::lock_guard<std::mutex> lk(mu);
    cache[key] = (unsigned)g;
  }
  *grid = (unsigned)g;
  return cudaSuccess;
}

// Launches `kern`, one CTA of `block` threads per slice and at most as many as are
// resident together, with `rows` rows of count slots (fewer if there are fewer phases)
// and the error word zeroed first, on the stream.
template <class Kern, class... Args>
inline cudaError_t launch_phases(Kern kern, int block, size_t smem, int max_grid, uint64_t slices, unsigned rows,
                                 void* scratch, cudaStream_t s, Args... args) {
  unsigned grid = 0;
  cudaError_t e = resident_grid(kern, block, smem, max_grid, &grid);
  if (e != cudaSuccess) return e;
  if (slices < grid) grid = (unsigned)slices;
  if (slices / grid >= 0xffff0000ull) return cudaErrorInvalidValue;  // phases are counted in 32 bits
  const uint64_t phases = (slices + grid - 1) / grid;
  e = cudaMemsetAsync(scratch, 0, 256 + 8ull * (phases < rows ? phases : rows) * grid, s);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args..., carve(scratch));
}

// Launches one pass over n > 0 elements of a 16-byte-aligned `in` (and, for
// the scan, a 16-byte-aligned `out`). scratch: scratch_need(n, sizeof(T))
// bytes of device memory; the part this launch uses is zeroed here, on the
// stream. With done.n_from, n is an upper bound of the device-side count.
template <class T, class O, class Sel, bool SCAN>
inline cudaError_t launch(const T* in, O* out, uint64_t n, const Sel& sel, uint64_t capacity, Done done,
                          void* scratch, cudaStream_t s) {
  if constexpr (SCAN) {
    constexpr uint64_t SE = scan::kSliceBytes / 4;
    return launch_phases(k_scan<512>, 512, (size_t)scan::kStages * scan::kSliceBytes, scan::kMaxGrid,
                         (n + SE - 1) / SE, scan::kSlots, scratch, s, in, out, n);
  } else {
    constexpr uint64_t SE = kSliceBytes / sizeof(T);
    return launch_phases(k_compact<T, O, Sel>, kBlock, (size_t)kStages * kSliceBytes, kMaxGrid, (n + SE - 1) / SE,
                         kSlots, scratch, s, in, out, n, sel, capacity, done);
  }
}

}  // namespace hxs
