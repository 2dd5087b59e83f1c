// Join count over one tile of left keys, with the matching window of right
// keys staged in shared memory by a bulk (TMA) copy.
#pragma once

#include "vg_prims.cuh"
#include "vg_relops.h"

namespace vg {

constexpr int kJcBlock = 256;
constexpr int kJcKeys = kJoinGroup;             // left keys per thread, consecutive
constexpr int kJcTile = kJcBlock * kJcKeys;     // 2048 left keys per block
constexpr int kJcWindow = 11264;                // right keys staged per block (44 KiB)

struct JoinCountSmem {
  alignas(16) uint32_t keys[kJcWindow + 8];
  alignas(8) uint64_t bar;
  uint64_t w0, w1;
  uint32_t staged;   // 0: search global memory, 1: window loaded by threads, 2: bulk copy
  uint32_t failed;
};

// Searches over the staged window, in 32-bit offsets from its first key
// (s points at it in shared memory, n keys).  kUpper: first offset whose key
// is above `key`; otherwise first offset whose key is not below it.
template <bool kUpper, typename T>
__device__ __forceinline__ bool smem_below(const T* s, uint32_t i, T key) {
  const T a = s[i];
  return kUpper ? (a <= key) : (a < key);
}

// Binary search over [lo, n).
template <bool kUpper, typename T>
__device__ __forceinline__ uint32_t smem_search(const T* s, uint32_t lo, uint32_t n, T key) {
  uint32_t len = n - lo;
  while (len > 0) {
    const uint32_t half = len >> 1;
    if (smem_below<kUpper>(s, lo + half, key)) {
      lo += half + 1;
      len -= half + 1;
    } else {
      len = half;
    }
  }
  return lo;
}

// The same answer at or after `from`, galloping from there (steps 1, 2, 4,
// ... then a binary search inside the last step): a thread's left keys are
// consecutive, so the next bound is usually a few keys further on.
template <bool kUpper, typename T>
__device__ __forceinline__ uint32_t smem_gallop(const T* s, uint32_t from, uint32_t n, T key) {
  if (from >= n || !smem_below<kUpper>(s, from, key)) return from;
  uint32_t lo = from, step = 1, hi = n;
  while (true) {
    const uint32_t nx = lo + step;
    if (nx >= n) break;
    if (!smem_below<kUpper>(s, nx, key)) {
      hi = nx;
      break;
    }
    lo = nx;
    step <<= 1;
  }
  // below(lo) holds and the answer lies in (lo, hi]
  return smem_search<kUpper>(s, lo + 1, hi, key);
}

// The keys of a relation sorted by its first column, or (PairKeys) by its
// first two, as 64-bit (column 0, column 1) words.
struct OneKeys {
  using T = uint32_t;
  const uint32_t* c0;
  __device__ __forceinline__ T operator()(uint64_t i) const { return __ldg(c0 + i); }
};
struct PairKeys {
  using T = uint64_t;
  const uint32_t* c0;
  const uint32_t* c1;
  __device__ __forceinline__ T operator()(uint64_t i) const {
    return (static_cast<uint64_t>(__ldg(c0 + i)) << 32) | __ldg(c1 + i);
  }
};

// First index in R[lo, hi) whose key is not below `key` (kUpper: above it),
// found by one warp: each round 31 lanes probe evenly spaced keys and the
// ballot of their comparisons narrows the range 32-fold, so a search over
// 10^8 keys takes six rounds of parallel loads instead of 27 dependent ones.
// Every lane of the warp must call it with the same arguments.
template <bool kUpper, typename T>
__device__ __forceinline__ uint64_t warp_bound(const T* __restrict__ R, uint64_t lo, uint64_t hi, T key) {
  const uint32_t lane = threadIdx.x & 31;
  while (hi - lo > 32) {
    const uint64_t step = (hi - lo + 31) >> 5;
    const uint64_t p = lo + static_cast<uint64_t>(lane + 1) * step;
    bool below = false;
    if (lane < 31 && p < hi) {
      const T a = __ldg(R + p);
      below = kUpper ? (a <= key) : (a < key);
    }
    const uint32_t c = __popc(__ballot_sync(0xffffffffu, below));
    const uint64_t nlo = c ? lo + static_cast<uint64_t>(c) * step + 1 : lo;
    const uint64_t cap = lo + static_cast<uint64_t>(c + 1) * step;
    hi = cap < hi ? cap : hi;
    lo = nlo;
  }
  bool below = false;
  if (lo + lane < hi) {
    const T a = __ldg(R + lo + lane);
    below = kUpper ? (a <= key) : (a < key);
  }
  return lo + __popc(__ballot_sync(0xffffffffu, below));
}

// Two bounds in R[0, n) by one warp at once: lanes 0-15 find the first
// index whose key is above ka (kUpperA) or not below it, lanes 16-31 the
// same for kb (kUpperB).  Each round every half-warp probes 15 evenly spaced
// keys of its range and the ballot of its comparisons narrows the range
// 16-fold.  Every lane of the warp must call it with the same arguments;
// every lane gets both bounds.
template <bool kUpperA, bool kUpperB, typename Keys, typename T>
__device__ __forceinline__ void warp_bound_pair_of(const Keys& keys, uint64_t n, T ka, T kb, uint64_t& ra,
                                                   uint64_t& rb) {
  const uint32_t lane = threadIdx.x & 31, sl = lane & 15;
  const bool second = lane >= 16;
  const bool upper = second ? kUpperB : kUpperA;
  const uint32_t half = second ? 0xffff0000u : 0x0000ffffu;
  const T key = second ? kb : ka;
  uint64_t lo = 0, hi = n;
  while (true) {
    const bool wide = hi - lo > 16;
    if (__ballot_sync(0xffffffffu, wide) == 0) break;
    uint64_t step = 0;
    bool below = false;
    if (wide) {
      step = (hi - lo + 15) >> 4;
      const uint64_t p = lo + static_cast<uint64_t>(sl + 1) * step;
      if (sl < 15 && p < hi) {
        const T a = keys(p);
        below = upper ? (a <= key) : (a < key);
      }
    }
    const uint32_t c = __popc(__ballot_sync(0xffffffffu, below) & half);
    if (wide) {
      const uint64_t nlo = c ? lo + static_cast<uint64_t>(c) * step + 1 : lo;
      const uint64_t cap = lo + static_cast<uint64_t>(c + 1) * step;
      hi = cap < hi ? cap : hi;
      lo = nlo;
    }
  }
  bool below = false;
  if (lo + sl < hi) {
    const T a = keys(lo + sl);
    below = upper ? (a <= key) : (a < key);
  }
  const uint64_t res = lo + __popc(__ballot_sync(0xffffffffu, below) & half);
  ra = __shfl_sync(0xffffffffu, res, 0);
  rb = __shfl_sync(0xffffffffu, res, 16);
}

template <bool kUpperA, bool kUpperB, typename T>
__device__ __forceinline__ void warp_bound_pair(const T* __restrict__ R, uint64_t n, T ka, T kb, uint64_t& ra,
                                                uint64_t& rb) {
  warp_bound_pair_of<kUpperA, kUpperB>([R](uint64_t i) { return __ldg(R + i); }, n, ka, kb, ra, rb);
}

// A tile's right-key window: the lower bound of klo and the upper bound of
// khi in R[0, nr), by one warp.
__device__ __forceinline__ void warp_window(const uint32_t* __restrict__ R, uint64_t nr, uint32_t klo,
                                            uint32_t khi, uint64_t& w0, uint64_t& w1) {
  warp_bound_pair<false, true, uint32_t>(R, nr, klo, khi, w0, w1);
}

// Lower and upper bounds of K keys in the right keys [w0, w1) at once:
// branchless binary searches advanced in lockstep, so each round has 2K
// independent loads in flight instead of one dependent chain per key.
// Positions have 32 bits (every join side has fewer than 2^32 rows), which
// halves the registers the bounds hold.
template <int K, typename Keys>
__device__ __forceinline__ void lockstep_bounds_of(const Keys& keys, uint32_t w0, uint32_t w1,
                                                   const typename Keys::T (&key)[K], uint32_t (&lo)[K],
                                                   uint32_t (&hi)[K]) {
  using T = typename Keys::T;
#pragma unroll
  for (int j = 0; j < K; ++j) lo[j] = hi[j] = w0;
  if (w1 <= w0) return;
  uint32_t n = w1 - w0;
  while (n > 1) {
    const uint32_t half = n >> 1;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const T a = keys(static_cast<uint64_t>(lo[j]) + half);
      const T b = keys(static_cast<uint64_t>(hi[j]) + half);
      lo[j] = (a < key[j]) ? lo[j] + half : lo[j];
      hi[j] = (b <= key[j]) ? hi[j] + half : hi[j];
    }
    n -= half;
  }
#pragma unroll
  for (int j = 0; j < K; ++j) {
    lo[j] += (keys(lo[j]) < key[j]) ? 1 : 0;
    hi[j] += (keys(hi[j]) <= key[j]) ? 1 : 0;
  }
}

template <int K>
__device__ __forceinline__ void lockstep_bounds32(const uint32_t* __restrict__ R, uint32_t w0, uint32_t w1,
                                                  const uint32_t (&key)[K], uint32_t (&lo)[K], uint32_t (&hi)[K]) {
  lockstep_bounds_of<K>(OneKeys{R}, w0, w1, key, lo, hi);
}

// Thread 0 of the block: records the tile's right-key window [w0, w1) and
// decides how it is staged in shared memory (sm.staged: 0 not staged, 1 by
// the block's threads, 2 its 16-byte aligned middle by one cp.async.bulk
// completed on sm.bar, its ragged ends by the threads).  The block must pass
// a barrier before jc_count_staged.
__device__ __forceinline__ void jc_issue_window(const uint32_t* __restrict__ R, uint64_t w0, uint64_t w1,
                                                JoinCountSmem& sm) {
  sm.w0 = w0;
  sm.w1 = w1;
  sm.staged = 0;
  sm.failed = 0;
  // R may start at any 4-byte boundary (a view of an index slice): element e
  // sits on a 16-byte boundary when (e + mis) % 4 == 0, and the window is laid
  // out in shared memory from `base`, the aligned element at or below w0
  // (index arithmetic is modulo 2^64, so base may lie below element 0).
  const uint64_t mis = (reinterpret_cast<uintptr_t>(R) >> 2) & 3u;
  if (w1 > w0 && w1 - w0 <= kJcWindow) {
    const uint64_t base = ((w0 + mis) & ~3ull) - mis;
    const uint64_t a0 = ((w0 + mis + 3) & ~3ull) - mis, a1 = ((w1 + mis) & ~3ull) - mis;
    if (a1 > a0 && a1 <= w1) {
      mbar_init(&sm.bar, 1);
      const uint32_t bytes = static_cast<uint32_t>((a1 - a0) * 4);
      mbar_arrive_expect_tx(&sm.bar, bytes);
      bulk_copy_g2s(&sm.keys[a0 - base], R + a0, bytes, &sm.bar);
      sm.staged = 2;
    } else {
      sm.staged = 1;
    }
  }
}

// The thread's keys (of left rows i0 + 8 * thread, up to i_end; ascending, the
// last repeated past the end) in a staged window of n right keys, whose first
// is right row w0.  The lower bounds of the first and last key are searched in
// lockstep over the window (a number of steps that the block shares), the
// others in lockstep between those two, and then the upper bounds of the keys
// that match, each before the next key's lower bound (both as many steps as
// the warp's widest range takes; every lane of the warp calls this): no lane
// waits for another's loop, where galloping from key to key left 18 of 32
// lanes active.  Equal keys share their bounds.  A key that the next thread
// has too, and the warp's last, gallop to their upper bound.
template <typename T>
__device__ __forceinline__ void jc_search_staged(const T* win, uint32_t n, uint64_t w0, uint64_t i0, uint64_t i_end,
                                                 const T (&key)[kJcKeys], uint32_t (&lov)[kJcKeys],
                                                 uint32_t (&cnt)[kJcKeys]) {
  const uint64_t first = i0 + static_cast<uint64_t>(threadIdx.x) * kJcKeys;
  uint32_t lo[kJcKeys];
  {
    uint32_t a = 0, b = 0, len = n;
    while (len > 1) {
      const uint32_t half = len >> 1;
      a = win[a + half - 1] < key[0] ? a + half : a;
      b = win[b + half - 1] < key[kJcKeys - 1] ? b + half : b;
      len -= half;
    }
    if (n) {
      a += win[a] < key[0] ? 1 : 0;
      b += win[b] < key[kJcKeys - 1] ? 1 : 0;
    }
    lo[0] = a;
    lo[kJcKeys - 1] = b;
  }
  // positions in [a, b]: b - a right keys to compare with (none where keys do
  // not ascend, so that nothing outside the window is ever read)
  uint32_t len = lo[kJcKeys - 1] > lo[0] ? lo[kJcKeys - 1] - lo[0] : 0u;
#pragma unroll
  for (int j = 1; j < kJcKeys - 1; ++j) lo[j] = lo[0];
  for (uint32_t most = __reduce_max_sync(0xffffffffu, len); most > 0; most >>= 1) {
    const uint32_t half = (len + 1) >> 1;
#pragma unroll
    for (int j = 1; j < kJcKeys - 1; ++j)
      if (half) lo[j] = win[lo[j] + half - 1] < key[j] ? lo[j] + half : lo[j];
    len -= half;
  }
  // upper bounds: range[j] right keys from lo[j] on may equal key j
  uint32_t hi[kJcKeys], most = 0;
#pragma unroll
  for (int j = 0; j < kJcKeys; ++j) hi[j] = lo[j];
  const T next_key = __shfl_down_sync(0xffffffffu, key[0], 1);
  const uint32_t next_lo = __shfl_down_sync(0xffffffffu, lo[0], 1);
  const bool last_own = lane_id() < 31 && next_key != key[kJcKeys - 1];
  uint32_t match = 0;   // keys whose upper bound the lockstep finds
#pragma unroll
  for (int j = 0; j < kJcKeys; ++j) {
    const uint32_t to = j + 1 < kJcKeys ? lo[j + 1] : next_lo;
    const bool own = j + 1 < kJcKeys ? key[j + 1] != key[j] : last_own;
    if (own && to > lo[j] && win[lo[j]] == key[j]) {
      match |= 1u << j;
      hi[j] = lo[j] + 1;
      most = max(most, to - lo[j] - 1);
    }
  }
  for (most = __reduce_max_sync(0xffffffffu, most); most > 0;) {
    const uint32_t half = (most + 1) >> 1;
#pragma unroll
    for (int j = 0; j < kJcKeys; ++j) {
      const uint32_t at = hi[j] + half - 1;
      if ((match >> j & 1u) && at < n && win[at] <= key[j]) hi[j] += half;
    }
    most -= half;
  }
  if (!last_own) hi[kJcKeys - 1] = smem_gallop<true, T>(win, lo[kJcKeys - 1], n, key[kJcKeys - 1]);
#pragma unroll
  for (int j = kJcKeys - 2; j >= 0; --j)
    if (key[j] == key[j + 1]) hi[j] = hi[j + 1];
#pragma unroll
  for (int j = 0; j < kJcKeys; ++j)
    if (first + j < i_end) {
      lov[j] = static_cast<uint32_t>(w0 + lo[j]);
      cnt[j] = max(hi[j], lo[j]) - lo[j];   // (keys out of order match nothing rather than 2^32 rows)
    }
}

// The thread's left keys: L[first, first + kJcKeys), the last of the tile
// repeated past its end.
__device__ __forceinline__ void jc_load_keys(const uint32_t* __restrict__ L, uint64_t first, uint64_t i_end,
                                             uint32_t (&key)[kJcKeys]) {
  static_assert(kJcKeys == 8, "the vector loads take 8 keys");
  if (first + kJcKeys <= i_end && (reinterpret_cast<uintptr_t>(L + first) & 15u) == 0) {
    const uint4 a = *reinterpret_cast<const uint4*>(L + first);
    const uint4 b = *reinterpret_cast<const uint4*>(L + first + 4);
    key[0] = a.x, key[1] = a.y, key[2] = a.z, key[3] = a.w;
    key[4] = b.x, key[5] = b.y, key[6] = b.z, key[7] = b.w;
  } else {
#pragma unroll
    for (int j = 0; j < kJcKeys; ++j) key[j] = L[first + j < i_end ? first + j : i_end - 1];
  }
}
__device__ __forceinline__ void jc_load_keys(const PairKeys& L, uint64_t first, uint64_t i_end,
                                             uint64_t (&key)[kJcKeys]) {
#pragma unroll
  for (int j = 0; j < kJcKeys; ++j) key[j] = L(first + j < i_end ? first + j : i_end - 1);
}
__device__ __forceinline__ void jc_load_keys(const OneKeys& L, uint64_t first, uint64_t i_end,
                                             uint32_t (&key)[kJcKeys]) {
  jc_load_keys(L.c0, first, i_end, key);
}

// Lower bound (in R) and match count of L[i0, min(i0 + kJcTile, nl)), given
// the window that jc_issue_window recorded: every left key of the tile lies
// in it.  A staged window is searched in shared memory; one that does not
// fit (a heavy key, or a right side much longer than the left) is searched in
// global memory with lockstep bounds instead.
// Thread t holds left keys i0 + 8t .. i0 + 8t + 7 in key[] (jc_load_keys, before
// the barrier, so that their loads are in flight with the window's), and gets
// their counts in cnt[] and lower bounds in lov[] (zero past the end).  Every thread of the block must call it.
__device__ __forceinline__ void jc_count_staged(const uint32_t (&key)[kJcKeys], uint64_t nl,
                                                const uint32_t* __restrict__ R, uint64_t i0,
                                                uint32_t (&lov)[kJcKeys], uint32_t (&cnt)[kJcKeys],
                                                JoinCountSmem& sm, DeviceErrors* err) {
#pragma unroll
  for (int j = 0; j < kJcKeys; ++j) cnt[j] = lov[j] = 0;
  const uint32_t tid = threadIdx.x;
  const uint64_t i_end = (i0 + kJcTile < nl) ? i0 + kJcTile : nl;
  const uint64_t mis = (reinterpret_cast<uintptr_t>(R) >> 2) & 3u;
  const uint64_t w0 = sm.w0, w1 = sm.w1 > sm.w0 ? sm.w1 : sm.w0;
  const uint32_t staged = sm.staged;
  const uint64_t base = ((w0 + mis) & ~3ull) - mis;
  const uint64_t first = i0 + static_cast<uint64_t>(tid) * kJcKeys;
  if (staged) {
    const uint64_t a0 = (staged == 2) ? ((w0 + mis + 3) & ~3ull) - mis : w1;
    const uint64_t a1 = (staged == 2) ? ((w1 + mis) & ~3ull) - mis : w1;
    for (uint64_t e = w0 + tid; e < a0; e += kJcBlock) sm.keys[e - base] = R[e];
    for (uint64_t e = a1 + tid; e < w1; e += kJcBlock) sm.keys[e - base] = R[e];
  }
  if (staged == 2) {
    // every consumer observes the barrier phase itself (bounded)
    if (!mbar_wait_bounded(&sm.bar, 0, err)) {
      sm.failed = 1;
      mbar_wait_bounded(&sm.bar, 0, err);  // a late copy gets a second bounded chance to land
    }
  }
  __syncthreads();
  const bool use_smem = staged != 0 && sm.failed == 0;
  if (!use_smem) {
    if (first >= i_end) return;   // counts stay zero
    uint32_t lo[kJcKeys], hi[kJcKeys];
    lockstep_bounds32<kJcKeys>(R, static_cast<uint32_t>(w0), static_cast<uint32_t>(w1), key, lo, hi);
#pragma unroll
    for (int j = 0; j < kJcKeys; ++j) {
      const uint64_t i = first + j;
      if (i < i_end) {
        lov[j] = static_cast<uint32_t>(lo[j]);
        cnt[j] = static_cast<uint32_t>(hi[j] - lo[j]);
      }
    }
    return;
  }
  const uint32_t* win = sm.keys + (w0 - base);
  jc_search_staged<uint32_t>(win, static_cast<uint32_t>(w1 - w0), w0, i0, i_end, key, lov, cnt);
}

// Called by one thread after the block's last use of the window: a bulk copy
// whose wait gave up may still be in flight into this block's shared memory,
// and must land before the block exits (bounded again; a copy that still has
// not landed is recorded as one more timeout).
__device__ __forceinline__ void jc_drain_window(JoinCountSmem& sm, DeviceErrors* err) {
  if (sm.staged == 2 && sm.failed) (void)mbar_wait_bounded(&sm.bar, 0, err);
}

// Staging of a PairKeys window: as 64-bit words, by the block's threads.
constexpr uint32_t kJcPairWindow = kJcWindow / 2;
__device__ __forceinline__ void jc_issue_pair_window(uint64_t w0, uint64_t w1, JoinCountSmem& sm) {
  sm.w0 = w0;
  sm.w1 = w1;
  sm.staged = (w1 > w0 && w1 - w0 <= kJcPairWindow) ? 1 : 0;
  sm.failed = 0;
}

struct SmemPairs {
  using T = uint64_t;
  const uint64_t* s;
  __device__ __forceinline__ T operator()(uint64_t i) const { return s[i]; }
};

// jc_count_staged for keys of two columns.  A window that does not fit shared
// memory is sampled: as many evenly spaced keys of it as fit, which bring every
// bound to within two of them before global memory is searched.  A right side
// much longer than the left has few tiles, and each one's block is bound by its
// scattered reads: the count of 10,285 left and 343,445 right rows took 51 us with
// the whole search in global memory and takes 32, that of 32,799 and 2M 53 and 41.
__device__ __forceinline__ void jc_count_staged_pairs(const uint64_t (&key)[kJcKeys], uint64_t nl, const PairKeys& R,
                                                      uint64_t i0, uint32_t (&lov)[kJcKeys], uint32_t (&cnt)[kJcKeys],
                                                      JoinCountSmem& sm) {
#pragma unroll
  for (int j = 0; j < kJcKeys; ++j) cnt[j] = lov[j] = 0;
  const uint32_t tid = threadIdx.x;
  const uint64_t i_end = (i0 + kJcTile < nl) ? i0 + kJcTile : nl;
  const uint64_t w0 = sm.w0, w1 = sm.w1 > sm.w0 ? sm.w1 : sm.w0;
  const uint64_t first = i0 + static_cast<uint64_t>(tid) * kJcKeys;
  uint64_t* win = reinterpret_cast<uint64_t*>(sm.keys);
  const uint32_t n = static_cast<uint32_t>(w1 - w0);
  const uint32_t step = sm.staged ? 1u : (n + kJcPairWindow - 1) / kJcPairWindow;   // (0: an empty window)
  const uint32_t samples = step ? (n + step - 1) / step : 0u;
  for (uint32_t e = tid; e < samples; e += kJcBlock) win[e] = R(w0 + static_cast<uint64_t>(e) * step);
  __syncthreads();
  if (sm.staged) {
    jc_search_staged<uint64_t>(win, n, w0, i0, i_end, key, lov, cnt);
    return;
  }
  if (first >= i_end || n == 0) return;   // counts stay zero
  uint32_t lo[kJcKeys], hi[kJcKeys];
  lockstep_bounds_of<kJcKeys>(SmemPairs{win}, 0u, samples, key, lo, hi);
  // a bound lies after the last sample below it, and at the next one at most
#pragma unroll
  for (int j = 0; j < kJcKeys; ++j) {
    lo[j] = lo[j] ? (lo[j] - 1) * step + 1 : 0u;
    hi[j] = hi[j] ? (hi[j] - 1) * step + 1 : 0u;
  }
  for (uint32_t len = step - 1; len > 0;) {
    const uint32_t half = (len + 1) >> 1;
#pragma unroll
    for (int j = 0; j < kJcKeys; ++j) {
      if (half <= n - lo[j] && R(w0 + lo[j] + half - 1) < key[j]) lo[j] += half;
      if (half <= n - hi[j] && R(w0 + hi[j] + half - 1) <= key[j]) hi[j] += half;
    }
    len -= half;
  }
#pragma unroll
  for (int j = 0; j < kJcKeys; ++j)
    if (first + j < i_end) {
      lov[j] = static_cast<uint32_t>(w0 + lo[j]);
      cnt[j] = hi[j] - lo[j];
    }
}

constexpr uint32_t kJcTileGroups = kJcTile / kJcKeys;

// What follows a tile's count: a block scan gives every left row its output
// offset from the tile's first, and base[tile] becomes the tile's first output
// row: the join's last tile to arrive scans the tiles' totals and writes the
// join's.  No tile waits for another (a look-back over the earlier tiles'
// totals kept the block's warps at a barrier for 8.3 of 18 stall cycles an
// instruction; 16M left rows took 163 us, 109 us without it).
// c and done (zero at first) are the join's own; left row i0 is the tile's
// first.  Every thread of the block calls it.
template <typename Off>
__device__ __forceinline__ void jc_finish_tile(uint64_t i0, const uint32_t (&lov)[kJcKeys], const uint32_t (&cnt)[kJcKeys],
                                               JoinCountSmem& sm, uint64_t* s_scan, uint32_t tile, uint32_t tiles,
                                               uint64_t nl, const JoinCounts<Off>& c, uint32_t* done, uint64_t* total,
                                               DeviceErrors* err) {
  __shared__ uint32_t s_last;
  uint64_t sum = 0;
#pragma unroll
  for (int k = 0; k < kJcKeys; ++k) sum += cnt[k];
  uint64_t tot;
  const uint64_t e = block_excl_scan64<kJcBlock>(sum, tot, s_scan);   // every thread is past its search
  const uint32_t tid = threadIdx.x;
  if (tid == 0) {
    jc_drain_window(sm, err);
    if (tiles == 1) {
      c.base[0] = 0;
      *total = tot;
    } else {   // (before the thread's stores of rows, which the fence would wait for)
      __stcg(reinterpret_cast<unsigned long long*>(c.base + tile), static_cast<unsigned long long>(tot));
      __threadfence();
      s_last = atomicAdd(done, 1u) == tiles - 1;
    }
  }
  const uint64_t first = i0 + static_cast<uint64_t>(tid) * kJcKeys, group = first / kJcKeys;
  if (first < nl) {
    uint32_t match = 0;
#pragma unroll
    for (int k = 0; k < kJcKeys; ++k) match |= (cnt[k] ? 1u : 0u) << k;
    c.start[group] = static_cast<Off>(e);
    c.match[group] = static_cast<uint8_t>(match);
    if (match) {
      static_assert(kJcKeys == 8, "the vector stores take 8 rows");
      uint4* lo4 = reinterpret_cast<uint4*>(c.lo + first);
      lo4[0] = make_uint4(lov[0], lov[1], lov[2], lov[3]);
      lo4[1] = make_uint4(lov[4], lov[5], lov[6], lov[7]);
      union {
        Off v[kJcKeys];
        uint4 w[kJcKeys * sizeof(Off) / 16];
      } o;
      Off run = static_cast<Off>(e);
#pragma unroll
      for (int k = 0; k < kJcKeys; ++k) {
        o.v[k] = run;
        run += cnt[k];
      }
#pragma unroll
      for (size_t k = 0; k < kJcKeys * sizeof(Off) / 16; ++k) reinterpret_cast<uint4*>(c.offs + first)[k] = o.w[k];
    }
  }
  if (tiles == 1) return;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  constexpr uint32_t kEach = 8;
  uint64_t before = 0;
  for (uint32_t t0 = 0; t0 < tiles; t0 += kJcBlock * kEach) {
    uint64_t v[kEach], mine = 0, all;
#pragma unroll
    for (uint32_t k = 0; k < kEach; ++k) {
      const uint32_t t = t0 + tid * kEach + k;
      v[k] = t < tiles ? __ldcg(reinterpret_cast<const unsigned long long*>(c.base + t)) : 0ull;
      mine += v[k];
    }
    uint64_t at = before + block_excl_scan64<kJcBlock>(mine, all, s_scan);
#pragma unroll
    for (uint32_t k = 0; k < kEach; ++k) {
      const uint32_t t = t0 + tid * kEach + k;
      if (t < tiles) c.base[t] = at;
      at += v[k];
    }
    before += all;
  }
  if (tid == 0) *total = before;
}

// The groups' first output rows (ascending), for searches.
template <typename Off>
struct JoinGroups {
  using T = Off;
  const Off* start;
  const uint64_t* base;
  __device__ __forceinline__ T operator()(uint64_t g) const {
    return static_cast<Off>(__ldg(base + g / kJcTileGroups)) + __ldg(start + g);
  }
};

// A join to write: its count, source and output columns (lc: the key columns
// and the other left ones, rc: the right ones without the keys).
template <typename Off>
struct JoinOutOf {
  JoinCounts<Off> cnt;
  uint64_t nl, total;
  const uint32_t* lc[VG_MAX_COLS];
  const uint32_t* rc[VG_MAX_COLS];
  uint32_t* oc[VG_MAX_COLS];
  uint32_t nlc, nrc;

  __host__ __device__ __forceinline__ JoinGroups<Off> groups() const { return {cnt.start, cnt.base}; }
  __host__ __device__ __forceinline__ uint64_t ngroups() const { return (nl + kJcKeys - 1) / kJcKeys; }
};
using JoinOut = JoinOutOf<uint32_t>;

constexpr int kJwBlock = 256;

// A tile's output rows that start a left row's ("heads"): the left row plus 1
// (0: not a head), and the right row that output row 0 of the tile would have
// from that head on (so that row k's is right + k).  heads: a bit per row.
template <int ROWS>
struct JwStage {
  static constexpr uint32_t kTile = kJwBlock * ROWS;
  alignas(16) uint32_t left[kTile];
  uint32_t right[kTile];
  uint32_t heads[kTile / 32];
};

// The block's threads clear a tile's heads; a barrier before jw_write_tile.
template <int ROWS>
__device__ __forceinline__ void jw_clear(JwStage<ROWS>& st) {
  for (uint32_t k = threadIdx.x; k < st.kTile / 4; k += kJwBlock)
    reinterpret_cast<uint4*>(st.left)[k] = make_uint4(0u, 0u, 0u, 0u);
}

// Marks the heads of a group's rows with matches among output rows [kb, kend).
template <int ROWS, typename Off>
__device__ __forceinline__ void jw_mark_group(const JoinOutOf<Off>& o, uint64_t g, uint32_t match, uint64_t kb,
                                              uint64_t kend, JwStage<ROWS>& st) {
  union {
    Off v[kJcKeys];
    uint4 w[kJcKeys * sizeof(Off) / 16];
  } f;
  union {
    uint32_t v[kJcKeys];
    uint4 w[2];
  } r;
  const uint64_t first = g * kJcKeys;
#pragma unroll
  for (size_t k = 0; k < kJcKeys * sizeof(Off) / 16; ++k) f.w[k] = __ldg(reinterpret_cast<const uint4*>(o.cnt.offs + first) + k);
#pragma unroll
  for (int k = 0; k < 2; ++k) r.w[k] = __ldg(reinterpret_cast<const uint4*>(o.cnt.lo + first) + k);
  const uint64_t base = __ldg(o.cnt.base + g / kJcTileGroups);
#pragma unroll
  for (int q = 0; q < kJcKeys; ++q) {
    const uint64_t at = base + f.v[q];
    if ((match >> q & 1u) && at < kend) {
      // of the rows that start at or before kb the last one, which covers it,
      // is marked last
      const uint32_t p = at > kb ? static_cast<uint32_t>(at - kb) : 0u;
      st.left[p] = static_cast<uint32_t>(first) + q + 1;
      st.right[p] = r.v[q] + static_cast<uint32_t>(kb - at);
    }
  }
}

// The left and right row of each of the thread's output rows, to st.left and
// st.right, for a tile whose groups lie far apart: every row's group is
// searched for, all of the thread's rows in lockstep (the last group that
// starts at or before a row has it: what follows starts after it).
template <int ROWS, typename Off>
__device__ __forceinline__ void jw_search_rows(const JoinOutOf<Off>& o, uint64_t kb, uint64_t kend, uint64_t ga, uint64_t gb,
                                            JwStage<ROWS>& st) {
  const JoinGroups<Off> starts = o.groups();
  uint32_t lo[ROWS];
#pragma unroll
  for (int it = 0; it < ROWS; ++it) lo[it] = 0;
  for (uint32_t n = static_cast<uint32_t>(gb - ga); n > 1;) {
    const uint32_t half = n >> 1;
#pragma unroll
    for (int it = 0; it < ROWS; ++it) {
      const Off k = static_cast<Off>(kb) + it * kJwBlock + threadIdx.x;
      if (starts(ga + lo[it] + half) <= k) lo[it] += half;
    }
    n -= half;
  }
#pragma unroll
  for (int it = 0; it < ROWS; ++it) st.left[it * kJwBlock + threadIdx.x] = lo[it];
#pragma unroll 1
  for (int it = 0; it < ROWS; ++it) {
    const uint32_t p = it * kJwBlock + threadIdx.x;
    if (kb + p >= kend) break;
    const uint64_t g = ga + st.left[p], first = g * kJcKeys;
    const uint32_t match = __ldg(o.cnt.match + g);
    const Off k = static_cast<Off>(kb) + p, base = static_cast<Off>(__ldg(o.cnt.base + g / kJcTileGroups));
    uint32_t q = 0;
    Off at = 0;
#pragma unroll
    for (uint32_t x = 0; x < kJcKeys; ++x) {
      const Off f = base + __ldg(o.cnt.offs + first + x);   // (not set where no row of the group matches)
      if ((match >> x & 1u) && f <= k) {
        q = x;
        at = f;
      }
    }
    st.left[p] = static_cast<uint32_t>(first) + q;
    st.right[p] = __ldg(o.cnt.lo + first + q) + static_cast<uint32_t>(k - at);
  }
}

// Output rows [kb, kend) (at most kJwBlock * ROWS) of a join, by one block;
// they come from the groups [ga, gb) of left rows.  Each left row with matches
// marks its first output row as a head; an output row's left row is the
// nearest head at or before it (a bit mask, one ballot per warp and 32 rows,
// and a maximum scan over the words): about 12 instructions a row, where
// galloping each row from the thread's previous one took over 100 (13.4M rows
// from 16M left rows: 199 -> 108 us; the six joins of a hub query 968 -> 770).
// Left rows without matches cost a bit, up to kFar groups: passes over them
// (about 1 us each of 256 groups) take longer than the searches of a tile's
// rows (some 15 us whatever the range) from there on.  1,000 output rows of 1M
// left ones took 135 us without the searches and 56 with them, 3,000 of 3M 239
// and 80; with the line at 32 passes 30,000 of 1M take 68 us for 62, at 64 passes
// 77.  Consecutive threads write consecutive rows, so loads and stores coalesce;
// hub keys spread over many blocks.
template <int ROWS, typename Off>
__device__ __forceinline__ void jw_write_tile(const JoinOutOf<Off>& o, uint64_t kb, uint64_t kend, uint64_t ga, uint64_t gb,
                                              JwStage<ROWS>& st) {
  constexpr uint32_t kTile = kJwBlock * ROWS;
  uint32_t li[ROWS], ri[ROWS];   // 1. the left and right row of each of the thread's output rows
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  constexpr uint32_t kFar = 16 * kJwBlock;
  if (gb - ga > kFar) {
    jw_search_rows<ROWS>(o, kb, kend, ga, gb, st);
#pragma unroll
    for (int it = 0; it < ROWS; ++it) {   // (each thread's own)
      li[it] = st.left[it * kJwBlock + threadIdx.x];
      ri[it] = st.right[it * kJwBlock + threadIdx.x];
    }
  } else {
    const uint8_t* match = o.cnt.match;
    for (uint64_t g = ga + threadIdx.x; g < gb; g += kJwBlock) {
      const uint32_t m = __ldg(match + g);
      if (m) jw_mark_group(o, g, m, kb, kend, st);
    }
    __syncthreads();
    uint32_t heads[ROWS];
#pragma unroll
    for (int it = 0; it < ROWS; ++it) {
      heads[it] = __ballot_sync(0xffffffffu, st.left[it * kJwBlock + threadIdx.x] != 0);
      if (lane == 0) st.heads[it * (kJwBlock / 32) + warp] = heads[it];
    }
    __syncthreads();
    // upto[g]: in lane l, the last head up to word 32 * g + l (row 0 is one)
    constexpr uint32_t kWords = kTile / 32, kGroups = (kWords + 31) / 32;
    uint32_t upto[kGroups];
#pragma unroll
    for (uint32_t g = 0; g < kGroups; ++g) {
      const uint32_t w = g * 32 + lane, x = w < kWords ? st.heads[w] : 0u;
      upto[g] = x ? w * 32 + 31 - __clz(x) : 0u;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, upto[g], d);
        if (static_cast<int>(lane) >= d) upto[g] = max(upto[g], y);
      }
      if (g) upto[g] = max(upto[g], __shfl_sync(0xffffffffu, upto[g - 1], 31));
    }
#pragma unroll
    for (int it = 0; it < ROWS; ++it) {
      const uint32_t k = it * kJwBlock + threadIdx.x, w = it * (kJwBlock / 32) + warp;
      uint32_t h = 0;
#pragma unroll
      for (uint32_t g = 0; g < kGroups; ++g) {   // the last head before word w
        const uint32_t y = __shfl_sync(0xffffffffu, upto[g], (w - 1) & 31);
        if (w > g * 32) h = y;
      }
      const uint32_t mine = heads[it] & (0xffffffffu >> (31 - lane));
      if (mine) h = w * 32 + 31 - __clz(mine);
      li[it] = st.left[h] - 1;
      ri[it] = st.right[h] + k;
    }
  }
  // 2. column by column: each thread's ROWS loads of a column are in flight
  // together (read-only path), each store instruction writes consecutive
  // rows, and one column's pointers are live at a time
  const uint32_t nlc = o.nlc, ncols = o.nlc + o.nrc;
  for (uint32_t c = 0; c < ncols; ++c) {
    const bool left = c < nlc;
    const uint32_t* src = left ? o.lc[c] : o.rc[c - nlc];
    uint32_t* dst = o.oc[c];
    uint32_t v[ROWS];
#pragma unroll
    for (int it = 0; it < ROWS; ++it) {
      const uint64_t k = kb + static_cast<uint64_t>(it) * kJwBlock + threadIdx.x;
      if (k < kend) v[it] = __ldg(src + (left ? li[it] : ri[it]));
    }
#pragma unroll
    for (int it = 0; it < ROWS; ++it) {
      const uint64_t k = kb + static_cast<uint64_t>(it) * kJwBlock + threadIdx.x;
      if (k < kend) dst[k] = v[it];
    }
  }
}

}  // namespace vg
