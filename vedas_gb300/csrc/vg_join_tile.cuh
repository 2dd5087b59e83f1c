// Join count over one tile of left keys, with the matching window of right
// keys staged in shared memory by a bulk (TMA) copy.
#pragma once

#include "vg_prims.cuh"

namespace vg {

constexpr int kJcBlock = 256;
constexpr int kJcKeys = 8;                      // left keys per thread, consecutive
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
// others in lockstep between those two (as many steps as the warp's widest
// range takes; every lane of the warp calls this): no lane waits for another's loop, where galloping from key to
// key left 18 of 32 lanes active.  The upper bound of a key that matches
// gallops from its lower bound; equal keys share both.
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
  uint32_t phi = 0;
#pragma unroll
  for (int j = 0; j < kJcKeys; ++j) {
    if (first + j < i_end) {
      const uint32_t hi = (j > 0 && key[j] == key[j - 1]) ? phi : smem_gallop<true, T>(win, lo[j], n, key[j]);
      lov[j] = static_cast<uint32_t>(w0 + lo[j]);
      cnt[j] = hi - lo[j];
      phi = hi;
    }
  }
}

// Lower bound (in R) and match count of L[i0, min(i0 + kJcTile, nl)), given
// the window that jc_issue_window recorded: every left key of the tile lies
// in it.  A staged window is searched in shared memory; one that does not
// fit (a heavy key, or a right side much longer than the left) is searched in
// global memory with lockstep bounds instead.
// The tile's counts stay in registers: thread t holds the counts of left
// keys i0 + 8t .. i0 + 8t + 7 in cnt[] and their lower bounds in lov[] (zero
// past the end).  Every thread of the block must call it.
__device__ __forceinline__ void jc_count_staged(const uint32_t* __restrict__ L, uint64_t nl,
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
  // the thread's left keys are loaded while the window's bulk copy is in flight
  const uint64_t first = i0 + static_cast<uint64_t>(tid) * kJcKeys;
  uint32_t key[kJcKeys];
  if (first + kJcKeys <= i_end && (reinterpret_cast<uintptr_t>(L + first) & 15u) == 0) {
    // two 16-byte loads (the thread's keys are consecutive)
    const uint4 a = *reinterpret_cast<const uint4*>(L + first);
    const uint4 b = *reinterpret_cast<const uint4*>(L + first + 4);
    key[0] = a.x, key[1] = a.y, key[2] = a.z, key[3] = a.w;
    key[4] = b.x, key[5] = b.y, key[6] = b.z, key[7] = b.w;
  } else {
#pragma unroll
    for (int j = 0; j < kJcKeys; ++j) {
      const uint64_t i = first + j;
      key[j] = L[i < i_end ? i : i_end - 1];
    }
  }
  static_assert(kJcKeys == 8, "the vector loads above take 8 keys");
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

// A tile's lower bounds and output offsets (from the tile's first), staged in
// the window's shared memory after the search so that they leave in coalesced
// stores: element e of the tile (thread e / 8's key e % 8) sits at e + e / 32
// of the 32-bit lower bounds, and at e + e / 32 (32-bit) or e + e / 16 (64-bit)
// of the offsets, which keeps both the per-thread writes and the row-order
// reads free of bank conflicts.
constexpr uint32_t kJcStageLoWords = kJcTile + kJcTile / 32;
__device__ __forceinline__ uint32_t* jc_stage_lo(JoinCountSmem& sm) { return sm.keys; }
template <typename Off>
__device__ __forceinline__ Off* jc_stage_off(JoinCountSmem& sm) {
  return reinterpret_cast<Off*>(sm.keys + kJcStageLoWords);
}
template <typename Off>
__device__ __forceinline__ uint32_t jc_stage_at(uint32_t e) {
  return e + e / (sizeof(Off) == 8 ? 16 : 32);
}
static_assert(kJcStageLoWords % 2 == 0, "the 64-bit staging area starts 8-byte aligned");
static_assert(kJcStageLoWords + 2 * (kJcTile + kJcTile / 16) <= kJcWindow, "staging fits in the window");

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

// jc_count_staged for keys of two columns.
__device__ __forceinline__ void jc_count_staged_pairs(const PairKeys& L, uint64_t nl, const PairKeys& R, uint64_t i0,
                                                      uint32_t (&lov)[kJcKeys], uint32_t (&cnt)[kJcKeys],
                                                      JoinCountSmem& sm) {
#pragma unroll
  for (int j = 0; j < kJcKeys; ++j) cnt[j] = lov[j] = 0;
  const uint32_t tid = threadIdx.x;
  const uint64_t i_end = (i0 + kJcTile < nl) ? i0 + kJcTile : nl;
  const uint64_t w0 = sm.w0, w1 = sm.w1 > sm.w0 ? sm.w1 : sm.w0;
  const uint64_t first = i0 + static_cast<uint64_t>(tid) * kJcKeys;
  uint64_t key[kJcKeys];
#pragma unroll
  for (int j = 0; j < kJcKeys; ++j) {
    const uint64_t i = first + j;
    key[j] = L(i < i_end ? i : i_end - 1);
  }
  uint64_t* win = reinterpret_cast<uint64_t*>(sm.keys);
  if (sm.staged)
    for (uint64_t e = w0 + tid; e < w1; e += kJcBlock) win[e - w0] = R(e);
  __syncthreads();
  if (sm.staged) {
    jc_search_staged<uint64_t>(win, static_cast<uint32_t>(w1 - w0), w0, i0, i_end, key, lov, cnt);
    return;
  }
  if (first >= i_end) return;   // counts stay zero
  uint32_t lo[kJcKeys], hi[kJcKeys];
  lockstep_bounds_of<kJcKeys>(R, static_cast<uint32_t>(w0), static_cast<uint32_t>(w1), key, lo, hi);
#pragma unroll
  for (int j = 0; j < kJcKeys; ++j)
    if (first + j < i_end) {
      lov[j] = lo[j];
      cnt[j] = hi[j] - lo[j];
    }
}

// What follows a tile's count: a block scan and a look-back over the same
// join's tiles [first_tile, tile) give every left row its output offset; the
// join's last tile writes its total.  lo and offs are the join's own arrays
// (left row i0 is the tile's first).  Off: 32 bits hold every offset of a join
// that is written (one with 2^32 rows or more is refused, by its 64-bit total);
// 64 bits for the join that takes any.  Every thread of the block calls it.
template <typename Off>
__device__ __forceinline__ void jc_finish_tile(uint64_t nl, uint64_t i0, const uint32_t (&lov)[kJcKeys],
                                               const uint32_t (&cnt)[kJcKeys], JoinCountSmem& sm, uint64_t* s_scan,
                                               uint64_t* s_b, uint64_t tile, uint64_t first_tile, bool last_tile,
                                               uint32_t* __restrict__ lo, Off* __restrict__ offs,
                                               uint64_t* status, uint64_t* total, DeviceErrors* err) {
  uint64_t sum = 0;
#pragma unroll
  for (int k = 0; k < kJcKeys; ++k) sum += cnt[k];
  uint64_t tot;
  const uint64_t e = block_excl_scan64<kJcBlock>(sum, tot, s_scan);   // every thread is past its search
  const uint32_t tid = threadIdx.x;
  const uint64_t first = i0 + static_cast<uint64_t>(tid) * kJcKeys;
  const uint32_t tile_n = static_cast<uint32_t>(nl - i0 < kJcTile ? nl - i0 : kJcTile);
  // a bulk copy that gave up may still land in the window: no staging there
  const bool stage = !(sm.staged == 2 && sm.failed);
  if (stage) {
    // lower bounds and tile-relative offsets staged in the window while warp 0
    // looks back; the tile's prefix is added when they are stored
    uint32_t* s_lo = jc_stage_lo(sm);
    Off* s_off = jc_stage_off<Off>(sm);
    uint64_t run = e;
#pragma unroll
    for (int k = 0; k < kJcKeys; ++k) {
      const uint32_t q = tid * kJcKeys + k;
      s_lo[q + q / 32] = lov[k];
      s_off[jc_stage_at<Off>(q)] = static_cast<Off>(run);
      run += cnt[k];
    }
  }
  if (threadIdx.x < 32) {
    const uint64_t p = warp_lookback_seg(status, tile, first_tile, tot, err);
    if (threadIdx.x == 0) *s_b = p;
  }
  __syncthreads();
  const uint64_t base = *s_b;
  if (last_tile && tid == 0) *total = base + tot;
  if (!stage) {
    uint64_t run = base + e;
#pragma unroll
    for (int k = 0; k < kJcKeys; ++k) {
      if (first + k < nl) {
        offs[first + k] = static_cast<Off>(run);
        lo[first + k] = lov[k];
      }
      run += cnt[k];
    }
    if (tid == 0) jc_drain_window(sm, err);
    return;
  }
  const uint32_t* s_lo = jc_stage_lo(sm);
  const Off* s_off = jc_stage_off<Off>(sm);
  for (uint32_t q = tid; q < tile_n; q += kJcBlock) {
    lo[i0 + q] = s_lo[q + q / 32];
    offs[i0 + q] = static_cast<Off>(base) + s_off[jc_stage_at<Off>(q)];
  }
}

// A join to write: left rows' lower bounds and output offsets, source and
// output columns (lc: the key columns and the other left ones, rc: the right
// ones without the keys).
template <typename Off>
struct JoinOutOf {
  using Offset = Off;
  const Off* offs;
  const uint32_t* lo;
  uint64_t nl, total;
  const uint32_t* lc[VG_MAX_COLS];
  const uint32_t* rc[VG_MAX_COLS];
  uint32_t* oc[VG_MAX_COLS];
  uint32_t nlc, nrc;
};
using JoinOut = JoinOutOf<uint32_t>;

constexpr int kJwBlock = 256;

// Left rows that a tile of kJwBlock * ROWS output rows stages: twice as many,
// since rows without matches lie between the others (16M left rows with 13M
// output rows had no tile staged when only as many fitted: 0.26 ms).
template <int ROWS>
struct JwStage {
  static constexpr uint32_t kMost = 2 * kJwBlock * ROWS;
  uint32_t off[kMost];   // first output row, from the tile's first (0 where it lies before)
  uint32_t lo[kMost];    // the right row that output row off comes from
};

// Output rows [kb, kend) (at most kJwBlock * ROWS) of a join, by one block.
// Output row k comes from the left row i with offs[i] <= k < offs[i + 1] and
// the right row lo[i] + (k - offs[i]); the rows come from left rows [ib, ie).
// When those fit the stage, their offsets and lower bounds lie in shared
// memory and each thread walks its rows (k increasing, consecutive threads on
// consecutive rows, so loads and stores coalesce) from the previous one's left
// row.  Hub keys thus spread over many blocks.
template <int ROWS, typename Off>
__device__ __forceinline__ void jw_write_tile(const JoinOutOf<Off>& o, uint64_t kb, uint64_t kend, uint64_t ib, uint64_t ie,
                                              JwStage<ROWS>& st) {
  const uint64_t m64 = ie - ib;
  const bool staged = m64 <= JwStage<ROWS>::kMost;
  const uint32_t m = static_cast<uint32_t>(staged ? m64 : 0);
  for (uint32_t e = threadIdx.x; e < m; e += kJwBlock) {
    const uint64_t f = o.offs[ib + e];
    const uint32_t r = o.lo[ib + e];
    st.off[e] = f > kb ? static_cast<uint32_t>(f - kb) : 0u;
    st.lo[e] = f > kb ? r : r + static_cast<uint32_t>(kb - f);
  }
  __syncthreads();
  // 1. the left and right row of each of the thread's output rows
  uint32_t li[ROWS], ri[ROWS];
  if (staged) {
    const uint32_t rows = static_cast<uint32_t>(kend - kb);
    uint32_t p = 0;   // the current left row, relative to ib
#pragma unroll
    for (int it = 0; it < ROWS; ++it) {
      const uint32_t k = it * kJwBlock + threadIdx.x;
      li[it] = ri[it] = 0;
      if (k < rows) {
        // last p with off[p] <= k, moving forward from the previous row's p
        uint32_t step = 1;
        while (p + step < m && st.off[p + step] <= k) {
          p += step;
          step <<= 1;
        }
        while (step > 1) {
          step >>= 1;
          if (p + step < m && st.off[p + step] <= k) p += step;
        }
        li[it] = static_cast<uint32_t>(ib) + p;
        ri[it] = st.lo[p] + (k - st.off[p]);
      }
    }
  } else {
    // a sparse tile (more left rows than the stage holds, most without matches): the
    // left rows of kGroup of the thread's output rows at a time come from
    // kGroup binary searches of the offsets advanced in lockstep, so each
    // round has kGroup independent loads in flight
    constexpr int kGroup = ROWS < 4 ? ROWS : 4;
#pragma unroll
    for (int g0 = 0; g0 < ROWS; g0 += kGroup) {
      uint64_t lq[kGroup], kk[kGroup];
#pragma unroll
      for (int q = 0; q < kGroup; ++q) {
        const uint64_t k = kb + static_cast<uint64_t>(g0 + q) * kJwBlock + threadIdx.x;
        kk[q] = k < kend ? k : kend - 1;
        lq[q] = ib;
      }
      uint64_t n = ie - ib;                     // last i in [ib, ie) with offs[i] <= k
      while (n > 1) {
        const uint64_t half = n >> 1;
#pragma unroll
        for (int q = 0; q < kGroup; ++q) lq[q] = (o.offs[lq[q] + half] <= kk[q]) ? lq[q] + half : lq[q];
        n -= half;
      }
#pragma unroll
      for (int q = 0; q < kGroup; ++q) {
        li[g0 + q] = static_cast<uint32_t>(lq[q]);
        ri[g0 + q] = static_cast<uint32_t>(o.lo[lq[q]] + (kk[q] - o.offs[lq[q]]));
      }
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
