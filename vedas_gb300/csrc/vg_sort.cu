// Stable LSD radix sort, onesweep style (one upfront histogram pass, then one
// pass per digit of at most 8 bits whose tile offsets come from a decoupled
// look-back).
//
// A tile is 256 threads x 16, 12, 8 or 4 keys; tiles take their index from an
// atomic ticket in launch order, which guarantees that every look-back
// predecessor is running.  Passes whose digit is the same for every key are
// skipped (the permutation would be the identity) where this file counts the
// digits, at the price of a wait; sorts whose counts the caller made run every
// pass and wait for nothing.
#include "vg_sort.h"

#include <algorithm>

#include "vg_prims.cuh"
#include "vg_radix.cuh"

namespace vg {
namespace {

constexpr int kBlock = 256;
constexpr int kRadix = kRadixValues;
constexpr int kMaxPasses = kRadixMaxPasses;

// Digit counts and bases of every pass in one read of the keys (16-byte
// loads), and which digits are the same for every key (a bit each).
template <typename K>
__global__ void __launch_bounds__(kBlock) radix_hist_kernel(const K* __restrict__ keys, uint64_t n, DigitList dl,
                                                            unsigned long long* __restrict__ hist,
                                                            uint64_t* __restrict__ bases, uint32_t* done,
                                                            uint32_t* whole) {
  extern __shared__ uint32_t sh[];   // [dl.n][kRadix]
  digit_counts_init<kBlock>(dl, sh);
  constexpr uint32_t kVec = 16 / sizeof(K);
  const uint64_t t = static_cast<uint64_t>(blockIdx.x) * kBlock + threadIdx.x;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * kBlock;
  uint64_t nv = 0;
  if ((reinterpret_cast<uintptr_t>(keys) & 15u) == 0) {
    nv = n / kVec;
    for (uint64_t i = t; i < nv; i += stride) {
      const uint4 v = reinterpret_cast<const uint4*>(keys)[i];
      K k[kVec];
      if constexpr (sizeof(K) == 8) {
        k[0] = (static_cast<uint64_t>(v.y) << 32) | v.x;
        k[1] = (static_cast<uint64_t>(v.w) << 32) | v.z;
      } else {
        k[0] = v.x, k[1] = v.y, k[2] = v.z, k[3] = v.w;
      }
#pragma unroll
      for (uint32_t q = 0; q < kVec; ++q) digit_counts_add(dl, sh, k[q]);
    }
  }
  for (uint64_t i = nv * kVec + t; i < n; i += stride) digit_counts_add(dl, sh, keys[i]);
  digit_counts_finish<kBlock>(dl, sh, hist, bases, done, n, whole);
}

__global__ void iota_kernel(uint32_t* out, uint64_t n) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
    out[i] = static_cast<uint32_t>(i);
}

// Look-back words: 32 bits (two of them flags) while every prefix fits 30
// bits, else 64.
template <bool WIDE>
struct Status;
template <>
struct Status<false> {
  using T = uint32_t;
  static constexpr T kAgg = 1u << 30, kInc = 2u << 30, kValue = (1u << 30) - 1;
  static __device__ __forceinline__ T load(const T* p) {
    T v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
  }
  static __device__ __forceinline__ void store(T* p, T v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
  }
};
template <>
struct Status<true> {
  using T = uint64_t;
  static constexpr T kAgg = kFlagAgg, kInc = kFlagInc, kValue = kValueMask;
  static __device__ __forceinline__ T load(const T* p) { return ld_status_u64(p); }
  static __device__ __forceinline__ void store(T* p, T v) { st_status_u64(p, v); }
};

// One digit pass.  What bounds it is the ranking (about 100 instructions per
// key and warp, four blocks of 64 registers per SM), not memory: 100M 64-bit
// keys take 0.49 ms with 7-bit digits and 0.55 with 8-bit ones (3.3 and 2.9
// TB/s), where ranking with __match_any_sync took 0.89 (its cost grows with
// the number of distinct digits in the warp).
// 1. the warps count their digits with shared atomics, so the tile's counts
//    are published before anything is ranked and the look-back of later tiles
//    finds them (publishing after the ranking: 0.53 ms);
// 2. every key's place in the tile: the lanes with the same digit from one
//    ballot per digit bit, the first of them takes their places off the
//    warp's running counter (which starts at the warp's first place) with one
//    shared atomic, four keys' atomics in flight.  Lanes and keys are taken in
//    input order, so the sort is stable: a warp barrier after each key's atomic
//    keeps the next key's first lane, often another one, behind it;
// 3. keys (and values) go to their places in shared memory and leave from
//    there in digit order, mostly coalesced.
// Keys past the end are all ones: the tile's highest digit, placed after every
// real key, never stored, and counted only by the last tile.
template <typename K, bool HAS_V, bool IOTA, int BITS, int ITEMS, bool WIDE>
__global__ void __launch_bounds__(kBlock, HAS_V && sizeof(K) == 8 && ITEMS > 8 ? 3 : 4) onesweep_kernel(
    const K* __restrict__ kin, K* __restrict__ kout, const uint32_t* __restrict__ vin,
    uint32_t* __restrict__ vout, uint64_t n, uint32_t shift, uint32_t mask, uint32_t look,
    const uint64_t* __restrict__ bucket_base, typename Status<WIDE>::T* status, uint32_t* ticket,
    DeviceErrors* err) {
  using S = Status<WIDE>;
  using Word = typename S::T;
  constexpr int kTile = kBlock * ITEMS, kWarps = kBlock / 32, R = 1 << BITS, kGroup = 4;
  static_assert(R <= kBlock, "one thread per digit value");
  static_assert(ITEMS % kGroup == 0, "keys are ranked in groups");
  extern __shared__ __align__(16) unsigned char smem[];
  K* s_keys = reinterpret_cast<K*>(smem);
  uint32_t* s_vals = reinterpret_cast<uint32_t*>(smem + kTile * sizeof(K));
  __shared__ uint32_t s_whist[kWarps * R];
  __shared__ Word s_glob[R];
  __shared__ uint32_t s_scan[kWarps + 1];
  __shared__ uint32_t s_tile;

  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid == 0) s_tile = atomicAdd(ticket, 1u);
#pragma unroll
  for (int i = 0; i < kWarps * R / kBlock; ++i) s_whist[i * kBlock + tid] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint64_t base = static_cast<uint64_t>(tile) * kTile;
  const uint32_t tile_n = static_cast<uint32_t>(n - base < kTile ? n - base : kTile);
  const uint32_t w0 = warp * (32u * ITEMS) + lane;
  kin += base;
  if (HAS_V && !IOTA) vin += base;

  K key[ITEMS];
  uint32_t val[HAS_V ? ITEMS : 1];
  if (tile_n == kTile) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) key[i] = kin[w0 + i * 32u];
    if (HAS_V) {
#pragma unroll
      for (int i = 0; i < ITEMS; ++i)
        val[i] = IOTA ? static_cast<uint32_t>(base) + w0 + i * 32u : vin[w0 + i * 32u];
    }
  } else {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const uint32_t q = w0 + i * 32u;
      key[i] = q < tile_n ? kin[q] : ~K(0);
      if (HAS_V) val[i] = IOTA ? static_cast<uint32_t>(base) + q : (q < tile_n ? vin[q] : 0u);
    }
  }
  uint32_t* wh = s_whist + warp * R;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) atomicAdd(&wh[static_cast<uint32_t>(key[i] >> shift) & mask], 1u);
  __syncthreads();

  // Thread d owns digit value d: the tile's count, published for later tiles,
  // and each warp's first place.
  uint32_t run = 0, cnt[kWarps];
  Word* my = status + static_cast<uint64_t>(tile) * R + tid;
  if (tid < R) {
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      cnt[w] = s_whist[w * R + tid];
      run += cnt[w];
    }
    S::store(my, (tile == 0 ? S::kInc : S::kAgg) | run);
  }
  uint32_t tot;
  const uint32_t excl = block_excl_scan<kBlock>(run, tot, s_scan);
  if (tid < R) {
    uint32_t x = excl;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      s_whist[w * R + tid] = x;
      x += cnt[w];
    }
  }
  __syncthreads();

#pragma unroll
  for (int g = 0; g < ITEMS; g += kGroup) {
    uint32_t peers[kGroup], first[kGroup];
#pragma unroll
    for (int q = 0; q < kGroup; ++q) {
      const uint32_t d = static_cast<uint32_t>(key[g + q] >> shift) & mask;
      uint32_t p = 0xffffffffu;
#pragma unroll
      for (int b = 0; b < BITS; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t v = __ballot_sync(0xffffffffu, bit);
        p &= bit ? v : ~v;
      }
      peers[q] = p;
    }
#pragma unroll
    for (int q = 0; q < kGroup; ++q) {
      const uint32_t d = static_cast<uint32_t>(key[g + q] >> shift) & mask;
      first[q] = 0;
      if ((peers[q] & lanemask_lt()) == 0) first[q] = atomicAdd(&wh[d], __popc(peers[q]));
      __syncwarp();
    }
#pragma unroll
    for (int q = 0; q < kGroup; ++q) {
      const uint32_t pos =
          __shfl_sync(0xffffffffu, first[q], __ffs(peers[q]) - 1) + __popc(peers[q] & lanemask_lt());
      s_keys[pos] = key[g + q];
      if (HAS_V) s_vals[pos] = val[g + q];
    }
  }

  // Decoupled look-back for digit value d over earlier tiles ([tile][value]
  // layout): `look` (1 or 4) earlier tiles' words are loaded at once, then
  // summed in order until one holds an inclusive prefix (a word not yet
  // published is waited for, a bounded number of polls).
  if (tid < R) {
    Word prefix = 0;
    if (tile > 0) {
      constexpr int kLook = 4;
      int64_t j = static_cast<int64_t>(tile) - 1;
      bool found = false;
      while (!found) {
        Word w[kLook];
#pragma unroll
        for (int q = 0; q < kLook; ++q)
          w[q] = (j - q >= 0 && q < static_cast<int>(look)) ? S::load(status + static_cast<uint64_t>(j - q) * R + tid)
                                                            : S::kInc;
#pragma unroll
        for (int q = 0; q < kLook; ++q) {
          if (found || q >= static_cast<int>(look)) break;
          Word v = w[q];
          for (uint32_t spins = 0; (v & ~S::kValue) == 0;) {
            if (++spins > kSpinLimit) {
              atomicExch(&err->timeout, 1u);
              v = S::kInc;
              break;
            }
            __nanosleep(20);
            v = S::load(status + static_cast<uint64_t>(j - q) * R + tid);
          }
          prefix += v & S::kValue;
          found = (v & S::kInc) != 0;
        }
        j -= look;
      }
      S::store(my, S::kInc | (prefix + run));
    }
    // + a place in the tile gives the output row (modulo the word: n fits it)
    s_glob[tid] = static_cast<Word>(bucket_base[tid]) + prefix - excl;
  }
  __syncthreads();
  // (after a wait that gave up in an earlier pass the keys no longer match
  // the counts: the row is checked, the caller sees the recorded timeout)
  auto store = [&](uint32_t p) {
    const K k = s_keys[p];
    const Word o = s_glob[static_cast<uint32_t>(k >> shift) & mask] + p;
    if (o < static_cast<Word>(n)) {
      kout[o] = k;
      if (HAS_V) vout[o] = s_vals[p];
    }
  };
  if (tile_n == kTile) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) store(i * kBlock + tid);
  } else {
    for (uint32_t p = tid; p < tile_n; p += kBlock) store(p);
  }
}

struct PassArgs {
  const uint32_t* vin;
  uint32_t* vout;
  uint64_t n;
  RadixDigit digit;
  const uint64_t* bases;
  void* status;
  uint32_t* ticket;
};

template <typename K, bool HAS_V, bool IOTA, int BITS, int ITEMS, bool WIDE>
void launch_pass_as(Ctx& ctx, const K* kin, K* kout, const PassArgs& a) {
  constexpr int kTile = kBlock * ITEMS;
  const size_t smem = kTile * sizeof(K) + (HAS_V ? kTile * sizeof(uint32_t) : 0);
  auto kernel = onesweep_kernel<K, HAS_V, IOTA, BITS, ITEMS, WIDE>;
  // once per instantiation (thread-safe static initialisation)
  static const bool attr_set = [&] {
    VG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    // all of the unified L1/shared storage as shared memory: three or more
    // blocks of a tile's keys (and values) per SM
    VG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared));
    return true;
  }();
  (void)attr_set;
  const uint64_t tiles = div_up(a.n, kTile);
  const double bytes = static_cast<double>(a.n) * (2 * sizeof(K) + (HAS_V ? (IOTA ? 4 : 8) : 0));
  ctx.launch("radix_onesweep", bytes, [&] {
    kernel<<<static_cast<unsigned>(tiles), kBlock, smem, ctx.stream>>>(
        kin, kout, a.vin, a.vout, a.n, a.digit.shift, (1u << a.digit.bits) - 1u, ctx.tune.sort_lookback, a.bases,
        static_cast<typename Status<WIDE>::T*>(a.status), a.ticket, ctx.d_err);
  });
  VG_CUDA(cudaGetLastError());
}

// Digits of up to 7 bits have 128 counters a warp instead of 256 and one
// ballot a key less.
constexpr uint32_t status_row(uint32_t bits) { return bits <= 7 ? 128 : 256; }
// Prefixes of 2^30 rows and more take 64-bit look-back words.
constexpr bool wide_status(uint64_t n) { return n >= (1ull << 30); }

template <typename K, bool HAS_V, bool IOTA, int ITEMS, bool WIDE>
void launch_pass_bits(Ctx& ctx, const K* kin, K* kout, const PassArgs& a) {
  if (a.digit.bits <= 7) launch_pass_as<K, HAS_V, IOTA, 7, ITEMS, WIDE>(ctx, kin, kout, a);
  else launch_pass_as<K, HAS_V, IOTA, 8, ITEMS, WIDE>(ctx, kin, kout, a);
}

template <typename K, bool HAS_V, bool IOTA>
void launch_pass(Ctx& ctx, int items, const K* kin, K* kout, const PassArgs& a) {
  if (wide_status(a.n)) launch_pass_bits<K, HAS_V, IOTA, 16, true>(ctx, kin, kout, a);
  else if (items == 16) launch_pass_bits<K, HAS_V, IOTA, 16, false>(ctx, kin, kout, a);
  else if (items == 12) launch_pass_bits<K, HAS_V, IOTA, 12, false>(ctx, kin, kout, a);
  else if (items == 8) launch_pass_bits<K, HAS_V, IOTA, 8, false>(ctx, kin, kout, a);
  else launch_pass_bits<K, HAS_V, IOTA, 4, false>(ctx, kin, kout, a);
}

// Keys per thread: the context's choice (16 by default), or fewer while that
// leaves less than two tiles per SM.
int items_for(const Ctx& ctx, uint64_t n) {
  if (wide_status(n)) return 16;
  const int most = (ctx.tune.sort_items == 8 || ctx.tune.sort_items == 12) ? static_cast<int>(ctx.tune.sort_items) : 16;
  const uint64_t two = 2ull * ctx.num_sms * kBlock;
  if (n >= two * most) return most;
  return n >= two * 8 && most > 8 ? 8 : 4;
}

// Tickets and look-back words of a list of passes, to be zeroed before them:
// the tickets (and one more word for the caller), then the words of as many
// passes as half a byte a key holds (1 MiB in small sorts, and what that
// leaves of the arena's block): four passes of 7-bit digits in tiles of 4096
// keys, two of 8-bit ones, half of that from 2^30 keys on.  Later passes use
// them again, zeroed in between (one memset more, 2 us).  With the words of all
// passes at once a sort of 64-bit keys over eight digits held two bytes a key.
struct PassScratch {
  static constexpr size_t kHead = 128, kLeast = 1u << 20;
  static_assert((kMaxPasses + 1) * sizeof(uint32_t) <= kHead, "tickets and the caller's word");
  size_t bytes;       // to be zeroed
  size_t set = 0;     // bytes of a pass's words
  uint32_t sets = 1;  // passes whose words there are
  int items;
  // more: bytes that the caller puts behind them in the same block
  PassScratch(const Ctx& ctx, uint64_t n, const DigitList& dl, size_t more) : items(items_for(ctx, n)) {
    const uint64_t tiles = div_up(n, static_cast<uint64_t>(kBlock) * items);
    const size_t word = wide_status(n) ? sizeof(uint64_t) : sizeof(uint32_t);
    for (uint32_t p = 0; p < dl.n; ++p) set = std::max(set, tiles * status_row(dl.d[p].bits) * word);
    size_t room = std::max<size_t>(div_up(n, uint64_t{4096}) * 2048, kLeast);
    if (room <= Arena::kSmallMax) room = std::max(Arena::block_bytes(room), kHead + more) - kHead - more;
    if (set) sets = static_cast<uint32_t>(std::clamp<size_t>(room / set, 1, dl.n));
    bytes = kHead + sets * set;
  }
  // Where the words of the t-th pass lie, zeroed on the stream if they have
  // been used before.
  void* words(Ctx& ctx, char* zeroed, size_t t) const {
    if (t && t % sets == 0) VG_CUDA(cudaMemsetAsync(zeroed + kHead, 0, sets * set, ctx.stream));
    return zeroed + kHead + t % sets * set;
  }
};

DigitList digit_list(const std::vector<RadixDigit>& digits) {
  if (digits.size() > kMaxPasses) fail(VG_ERR_INVALID, "radix sort: too many digits");
  DigitList dl{};
  dl.n = static_cast<uint32_t>(digits.size());
  for (uint32_t p = 0; p < dl.n; ++p) dl.d[p] = digits[p];
  return dl;
}

// The passes (those of `todo`, in order) over zeroed scratch; returns whether
// the result is in the alternate buffers.
template <typename K>
bool run_passes(Ctx& ctx, K* keys, K* keys_alt, uint32_t* vals, uint32_t* vals_alt, uint64_t n, const DigitList& dl,
                const uint64_t* const* bases, const std::vector<uint32_t>& todo, const PassScratch& ps, char* zeroed,
                bool vals_iota) {
  const bool has_v = vals != nullptr;
  K* kin = keys;
  K* kout = keys_alt;
  uint32_t* vin = vals;
  uint32_t* vout = vals_alt;
  for (size_t t = 0; t < todo.size(); ++t) {
    const uint32_t p = todo[t];
    const PassArgs a{vin, vout, n, dl.d[p], bases[p], ps.words(ctx, zeroed, t), reinterpret_cast<uint32_t*>(zeroed) + p};
    if (!has_v) launch_pass<K, false, false>(ctx, ps.items, kin, kout, a);
    else if (t == 0 && vals_iota) launch_pass<K, true, true>(ctx, ps.items, kin, kout, a);
    else launch_pass<K, true, false>(ctx, ps.items, kin, kout, a);
    std::swap(kin, kout);
    std::swap(vin, vout);
  }
  return kin == keys_alt;
}

template <typename K>
bool radix_sort_impl(Ctx& ctx, K* keys, K* keys_alt, uint32_t* vals, uint32_t* vals_alt, uint64_t n,
                     const std::vector<RadixDigit>& digits, bool vals_iota) {
  const bool has_v = vals != nullptr;
  if (n == 0) return false;
  if (n > 0xFFFFFFFFull && has_v) fail(VG_ERR_OVERFLOW, "radix sort values are 32-bit row ids");
  const DigitList dl = digit_list(digits);
  const uint32_t passes = dl.n;
  // counts, tickets and the passes' look-back words in one block, zeroed by
  // one memset; the bases behind them
  const size_t hist_bytes = passes * kRadix * sizeof(uint64_t);
  const PassScratch ps(ctx, n, dl, 2 * hist_bytes);
  Scratch<char> scratch(ctx, ps.bytes + 2 * hist_bytes);
  char* sc = scratch.get();
  auto* hist = reinterpret_cast<unsigned long long*>(sc + ps.bytes);
  auto* bases = reinterpret_cast<uint64_t*>(sc + ps.bytes + hist_bytes);
  auto* done = reinterpret_cast<uint32_t*>(sc) + kMaxPasses;
  VG_CUDA(cudaMemsetAsync(sc, 0, ps.bytes + hist_bytes, ctx.stream));
  uint64_t grid = div_up(n, kBlock * 16);
  const uint64_t gmax = static_cast<uint64_t>(ctx.num_sms) * 8;
  if (grid > gmax) grid = gmax;
  if (grid < 1) grid = 1;
  auto* whole = reinterpret_cast<uint32_t*>(ctx.h_small);
  ctx.launch("radix_histogram", static_cast<double>(n) * sizeof(K), [&] {
    radix_hist_kernel<K><<<static_cast<unsigned>(grid), kBlock, (passes ? passes : 1) * kRadix * sizeof(uint32_t),
                           ctx.stream>>>(keys, n, dl, hist, bases, done, whole);
  });
  VG_CUDA(cudaGetLastError());
  std::vector<uint32_t> todo;
  // (the kernel stored the host's word: no copy, and nothing for a copy to be staged in)
  ctx.sync();
  for (uint32_t p = 0; p < passes; ++p)
    if (!(*whole >> p & 1u)) todo.push_back(p);
  if (todo.empty()) {
    if (has_v && vals_iota) fill_iota(ctx, vals, n);
    return false;
  }
  const uint64_t* pb[kMaxPasses];
  for (uint32_t p = 0; p < passes; ++p) pb[p] = bases + p * kRadix;
  return run_passes(ctx, keys, keys_alt, vals, vals_alt, n, dl, pb, todo, ps, sc, vals_iota);
}

}  // namespace

void radix_plan(std::vector<RadixDigit>& digits, int begin, int end) {
  const int passes = (end - begin + 7) / 8;
  for (int p = 0, at = begin; p < passes; ++p) {
    const int left = passes - p, bits = (end - at + left - 1) / left;
    digits.push_back({static_cast<uint32_t>(at), static_cast<uint32_t>(bits)});
    at += bits;
  }
}

bool radix_sort_u32(Ctx& ctx, uint32_t* keys, uint32_t* keys_alt, uint32_t* vals, uint32_t* vals_alt,
                    uint64_t n, int end_bit, bool vals_iota) {
  std::vector<RadixDigit> digits;
  radix_plan(digits, 0, end_bit);
  return radix_sort_impl<uint32_t>(ctx, keys, keys_alt, vals, vals_alt, n, digits, vals_iota);
}

bool radix_sort_u64(Ctx& ctx, uint64_t* keys, uint64_t* keys_alt, uint64_t n, int end_bit) {
  std::vector<RadixDigit> digits;
  radix_plan(digits, 0, end_bit);
  return radix_sort_impl<uint64_t>(ctx, keys, keys_alt, nullptr, nullptr, n, digits, false);
}

bool radix_sort_u64_counted(Ctx& ctx, uint64_t* keys, uint64_t* keys_alt, uint32_t* vals, uint32_t* vals_alt,
                            uint64_t n, const std::vector<RadixDigit>& digits,
                            const std::vector<const uint64_t*>& bases, bool vals_iota) {
  if (n == 0) return false;
  if (n > 0xFFFFFFFFull && vals) fail(VG_ERR_OVERFLOW, "radix sort values are 32-bit row ids");
  if (digits.empty()) {
    if (vals && vals_iota) fill_iota(ctx, vals, n);
    return false;
  }
  const DigitList dl = digit_list(digits);
  const PassScratch ps(ctx, n, dl, 0);
  Scratch<char> scratch(ctx, ps.bytes);
  VG_CUDA(cudaMemsetAsync(scratch.get(), 0, ps.bytes, ctx.stream));
  std::vector<uint32_t> todo(dl.n);
  for (uint32_t p = 0; p < dl.n; ++p) todo[p] = p;
  return run_passes<uint64_t>(ctx, keys, keys_alt, vals, vals_alt, n, dl, bases.data(), todo, ps, scratch.get(),
                              vals_iota);
}

void fill_iota(Ctx& ctx, uint32_t* out, uint64_t n) {
  if (n == 0) return;
  uint64_t grid = div_up(n, kBlock * 8);
  const uint64_t gmax = static_cast<uint64_t>(ctx.num_sms) * 8;
  if (grid > gmax) grid = gmax;
  ctx.launch("iota", 4.0 * n, [&] { iota_kernel<<<static_cast<unsigned>(grid), kBlock, 0, ctx.stream>>>(out, n); });
  VG_CUDA(cudaGetLastError());
}

}  // namespace vg
