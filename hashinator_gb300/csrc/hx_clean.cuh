// hx_clean.cuh — clean_tombstones in one pass over the table.
//
// Every key that does not sit in its home bucket is taken out, every TOMBSTONE
// becomes EMPTY, and the keys taken out go back in (hashinator.h:1262-1315). What a
// slice of the table looks like when all keys are out depends on that slice alone, so
// one CTA does both for its slice in shared memory: it keeps the keys that are at home,
// queues the others, and gives each of those the first EMPTY bucket from its home on,
// found in a bitmap (32 buckets at a look; a key occurs once, so nothing has to be
// compared). The slice is read once and written once. A key whose home lies in the
// slice before (its run crossed the slice's end), or that finds its slice full, goes to
// a list and is inserted when all slices are done; a table of one slice wraps instead.
// Bound by instructions (about 40 a bucket and 100 a moved key; DRAM at a quarter of
// its rate). 2^27 u32 buckets at load factor 0.5 / 0.9 with 30 % erased: 0.65 / 0.73 ms;
// a compaction pass, a list of all moved keys and their re-insertion at random took
// 0.76 / 1.25 ms. A persistent grid (0.75 / 0.91 ms, its loop spills) and fetching
// slices ahead into L2 (0.68 / 0.71 ms) gave nothing.
#pragma once
#include "hx_probe.cuh"
#include "../../include/hx_stream.cuh"

namespace hx {

constexpr unsigned kCleanThreads = 512;
template <class P>
__host__ __device__ constexpr unsigned clean_slice() {  // buckets: 32 KiB
  return 32768 / sizeof(P);
}
// Shared memory of a slice of `slots` buckets: the result and the queue.
template <class P>
constexpr unsigned clean_smem(unsigned slots) {
  return 2 * slots * (unsigned)sizeof(P) + 16;
}

// B: buckets per load, slots a multiple of it.
template <class P, int B>
__global__ void __launch_bounds__(kCleanThreads, 3) k_clean(P* table, unsigned slots, int sp, DInfo* info, P* left,
                                                           uint64_t left_cap) {
  using K = typename PairTraits<P>::K;
  using V = typename PairTraits<P>::V;
  constexpr K EMPTY = PairTraits<P>::EMPTY, TOMB = PairTraits<P>::TOMB;
  constexpr unsigned T = kCleanThreads, N = clean_slice<P>() / B / T > 0 ? clean_slice<P>() / B / T : 1;
  extern __shared__ __align__(16) unsigned char s_clean[];
  P* s_out = reinterpret_cast<P*>(s_clean);
  P* s_queue = s_out + slots;
  __shared__ unsigned s_free[clean_slice<P>() / 32];  // bit set: nothing is there yet
  __shared__ unsigned s_queued, s_away, s_over, s_max;
  __shared__ unsigned long long s_left0;
  const unsigned tid = threadIdx.x, lane = tid & 31;
  const uint32_t base = blockIdx.x * slots;
  const bool whole = gridDim.x == 1;  // the slice is the table: probes wrap inside it
  // Nobody changes this count before every CTA has counted itself done below.
  if (*reinterpret_cast<volatile unsigned long long*>(&info->tombstones) == 0) {
    if (blockIdx.x == 0 && tid == 0) info->moved = info->left = 0;
    return;
  }
  K k[N][B];
  V v[N][B];
#pragma unroll
  for (unsigned j = 0; j < N; ++j) {
    const unsigned b0 = (j * T + tid) * B;
    if (b0 < slots) load_buckets<B>(table + base + b0, k[j], v[j]);
    else
#pragma unroll
      for (int q = 0; q < B; ++q) k[j][q] = EMPTY;
  }
  for (unsigned i = tid; i < (slots + 31) / 32; i += T) s_free[i] = 0;
  if (tid == 0) s_queued = s_away = s_over = s_max = 0;
  __syncthreads();
  // ---- what stays, what is queued, what belongs to another slice ---------------
  unsigned moves = 0, away = 0;  // bit j * B + q: not at home; and home in another slice
#pragma unroll
  for (unsigned j = 0; j < N; ++j) {
    const unsigned b0 = (j * T + tid) * B;
    unsigned free = 0;
    alignas(16) P kept[B];
#pragma unroll
    for (int q = 0; q < B; ++q) {
      const K key = k[j][q];
      const uint32_t h = home_slot(key, sp) - base;  // wraps to a large number before the slice
      const bool there = key != EMPTY && key != TOMB, stays = there && h == b0 + q;
      kept[q].first = stays ? key : EMPTY;
      kept[q].second = stays ? v[j][q] : V(0);
      free |= (unsigned)!stays << q;
      moves |= (unsigned)(there && !stays) << (j * B + q);
      away |= (unsigned)(there && h >= slots) << (j * B + q);
    }
    if (b0 < slots) {
      if constexpr (B * sizeof(P) == 32) {
        uint4 w[2];
        memcpy(w, kept, 32);
        reinterpret_cast<uint4*>(s_out + b0)[0] = w[0];
        reinterpret_cast<uint4*>(s_out + b0)[1] = w[1];
      } else {
        s_out[b0] = kept[0];
      }
      if (free) atomicOr(&s_free[b0 / 32], free << (b0 % 32));
    }
  }
  // ---- the queue: one scan of the counts per warp ----------------------------
  {
    const unsigned c = __popc(moves & ~away) | (unsigned)__popc(away) << 16;
    const unsigned incl = hxs::warp_incl_scan(c, lane);
    unsigned q0 = 0, a0 = 0;
    if (lane == 31) {
      if (incl & 0xffffu) q0 = atomicAdd(&s_queued, incl & 0xffffu);
      if (incl >> 16) a0 = atomicAdd(&s_away, incl >> 16);
    }
    q0 = __shfl_sync(0xffffffffu, q0, 31) + ((incl - c) & 0xffffu);
    a0 = __shfl_sync(0xffffffffu, a0, 31) + ((incl - c) >> 16);
    // the keys of other slices wait at the queue's far end: a bucket holds at most one key, so the two never meet
#pragma unroll
    for (unsigned j = 0; j < N; ++j) {
#pragma unroll
      for (int q = 0; q < B; ++q) {
        if (!(moves >> (j * B + q) & 1u)) continue;
        P pr;
        pr.first = k[j][q];
        pr.second = v[j][q];
        s_queue[away >> (j * B + q) & 1u ? slots - 1 - a0++ : q0++] = pr;
      }
    }
  }
  __syncthreads();
  // ---- each queued key to the first free bucket from its home on ---------------
  const unsigned queued = s_queued, words = (slots + 31) / 32, tmask = slots - 1;
  const unsigned moved = queued + s_away;
  unsigned maxd = 0, over = 0, turn = 0;  // over: bit t, the key of the thread's turn t found its slice full
  for (unsigned i = tid; i < queued; i += T, ++turn) {
    const P pr = s_queue[i];
    const unsigned h = home_slot(pr.first, sp) - base;
    unsigned w = h / 32, mask = ~0u << (h % 32);
    for (;;) {
      const unsigned free = *const_cast<volatile unsigned*>(&s_free[w]) & mask;
      if (free) {
        const unsigned bit = free & (0u - free);
        if (atomicAnd(&s_free[w], ~bit) & bit) {
          const unsigned at = w * 32 + __ffs(bit) - 1;
          s_out[at] = pr;
          maxd = max(maxd, ((at - h) & tmask) + 1);
          break;
        }
      } else {
        mask = ~0u;
        if (++w == words) {
          if (!whole) {
            over |= 1u << turn;
            break;
          }
          w = 0;  // there is room: as many buckets were freed as keys are queued
        }
      }
    }
  }
  maxd = __reduce_max_sync(0xffffffffu, maxd);
  if (lane == 0 && maxd) atomicMax(&s_max, maxd);
  if (over) atomicAdd(&s_over, (unsigned)__popc(over));
  __syncthreads();
  const unsigned aways = s_away;
  if (tid == 0) {
    const unsigned n = aways + s_over;
    s_left0 = n ? atomicAdd(&info->left_next, (unsigned long long)n) : 0ull;
    if (s_left0 + n > left_cap) atomicExch(&info->err, HX_STATUS_FAIL);  // more keys than fill says: some are lost
    s_over = 0;
  }
  // ---- write back ----------------------------------------------------------
  constexpr unsigned V16 = 16 / sizeof(P);
  uint4* out = reinterpret_cast<uint4*>(table + base);
  for (unsigned i = tid; i < slots / V16; i += T) out[i] = reinterpret_cast<const uint4*>(s_out)[i];
  __syncthreads();
  for (unsigned i = tid; i < aways; i += T) {
    const uint64_t at = s_left0 + i;
    if (at < left_cap) left[at] = s_queue[slots - 1 - i];
  }
  for (unsigned i = tid; over; i += T, over >>= 1) {
    if (!(over & 1u)) continue;
    const uint64_t at = s_left0 + aways + atomicAdd(&s_over, 1u);
    if (at < left_cap) left[at] = s_queue[i];
  }
  // ---- counters; the last CTA closes the call ------------------------------------
  __syncthreads();
  if (tid == 0) {
    if (moved) atomicAdd(&info->moved_next, (unsigned long long)moved);
    if (s_max) atomicMax(&info->max_next, s_max);
    __threadfence();
    if (atomicAdd(&info->done, 1u) == gridDim.x - 1) {
      __threadfence();
      volatile DInfo* d = info;
      const unsigned long long gone = d->left_next;
      const unsigned probe = d->max_next;
      d->moved = d->moved_next;
      d->left = gone;
      d->max_probe = probe ? probe : (d->fill ? 1u : 0u);
      d->fill -= gone;  // their insertion counts them again
      d->tombstones = 0;
      d->done = 0;
      d->max_next = 0;
      d->moved_next = d->left_next = 0;
    }
  }
}

}  // namespace hx
