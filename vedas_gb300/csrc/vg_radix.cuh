// Digit counts of a radix sort, for kernels that read (or make) the keys
// anyway: shared-memory counters per digit, added to global counts at the
// end; the last block to finish turns them into bucket bases.
#pragma once

#include "vg_prims.cuh"
#include "vg_sort.h"

namespace vg {

constexpr int kRadixValues = 256;   // counts and bases are kept for 256 values whatever a digit's width

struct DigitList {
  uint32_t n;
  RadixDigit d[kRadixMaxPasses];
};

// Device memory of the counts of a digit list: zeroed counts and block counter,
// and the bases.
struct RadixCounts {
  Scratch<char> mem;
  size_t bytes;
  static constexpr size_t kHead = 128;
  RadixCounts(Ctx& ctx, const DigitList& dl)
      : mem(ctx, 2 * dl.n * kRadixValues * sizeof(uint64_t) + kHead), bytes(dl.n * kRadixValues * sizeof(uint64_t)) {
    VG_CUDA(cudaMemsetAsync(mem.get(), 0, kHead + bytes, ctx.stream));
  }
  unsigned long long* hist() const { return reinterpret_cast<unsigned long long*>(mem.get() + kHead); }
  uint64_t* bases(uint32_t digit = 0) const {
    return reinterpret_cast<uint64_t*>(mem.get() + kHead + bytes) + static_cast<size_t>(digit) * kRadixValues;
  }
  uint32_t* done() const { return reinterpret_cast<uint32_t*>(mem.get()); }
};

// s: dl.n * kRadixValues words of shared memory.
template <int BLOCK>
__device__ __forceinline__ void digit_counts_init(const DigitList& dl, uint32_t* s) {
  for (uint32_t i = threadIdx.x; i < dl.n * kRadixValues; i += BLOCK) s[i] = 0;
  __syncthreads();
}

template <typename K>
__device__ __forceinline__ void digit_counts_add(const DigitList& dl, uint32_t* s, K key) {
  for (uint32_t p = 0; p < dl.n; ++p)
    atomicAdd(&s[p * kRadixValues + (static_cast<uint32_t>(key >> dl.d[p].shift) & ((1u << dl.d[p].bits) - 1u))], 1u);
}

// Every thread of every block calls it once, after its last key.  hist (zeroed
// before the launch) receives the counts, bases[p][v] the first output row of
// value v; done counts the blocks (zeroed).  whole (nullable, page-locked): bit
// p set where all n keys have one value of digit p.
template <int BLOCK>
__device__ __forceinline__ void digit_counts_finish(const DigitList& dl, const uint32_t* s,
                                                    unsigned long long* hist, uint64_t* bases, uint32_t* done,
                                                    uint64_t n = 0, uint32_t* whole = nullptr) {
  static_assert(BLOCK == kRadixValues, "one thread per digit value");
  static_assert(kRadixMaxPasses <= 32, "a bit per digit");
  __shared__ uint64_t s_scan[BLOCK / 32 + 1];
  __shared__ bool s_last;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < dl.n * kRadixValues; i += BLOCK)
    if (s[i]) atomicAdd(&hist[i], static_cast<unsigned long long>(s[i]));
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  uint32_t one = 0;
  for (uint32_t p = 0; p < dl.n; ++p) {
    const uint64_t c = ld_status_u64(reinterpret_cast<const uint64_t*>(&hist[p * kRadixValues + threadIdx.x]));
    uint64_t tot;
    bases[p * kRadixValues + threadIdx.x] = block_excl_scan64<BLOCK>(c, tot, s_scan);
    if (whole && __syncthreads_or(c == n)) one |= 1u << p;
  }
  if (whole && threadIdx.x == 0) *whole = one;
}

}  // namespace vg
