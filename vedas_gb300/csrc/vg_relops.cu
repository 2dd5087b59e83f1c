// Relation kernels: select copies, adjacent-unique compaction, sort-merge
// join (count -> scan -> load-balanced write), gathers and relation sorts.
#include "vg_relops.h"

#include <algorithm>
#include <cstring>
#include <initializer_list>
#include <optional>
#include <utility>

#include "vg_join_tile.cuh"
#include "vg_prims.cuh"
#include "vg_radix.cuh"
#include "vg_sort.h"

namespace vg {
namespace {

constexpr int kBlock = 256;
constexpr int kRows = 8;
constexpr int kTileRows = kBlock * kRows;
constexpr uint64_t kGuessRows = 1u << 20;   // joins of at most so many left rows guess their output (join()),
constexpr uint64_t kWideGuess = (1u << 18) + 1;   // and from so many on as eight times those

unsigned grid_for(const Ctx& ctx, uint64_t n, int per_thread, int per_sm = 16) {
  uint64_t g = div_up(n, static_cast<uint64_t>(kBlock) * per_thread);
  const uint64_t gmax = static_cast<uint64_t>(ctx.num_sms) * per_sm;
  if (g > gmax) g = gmax;
  return static_cast<unsigned>(g < 1 ? 1 : g);
}

// ---------------------------------------------------------------------------
// Multi-piece copy: destination-aligned 128-bit stores, source loads
// vectorised when the source shares the destination's 16-byte phase.
// ---------------------------------------------------------------------------
struct CopyArgs {
  CopyPiece p[16];
  uint64_t start[17];  // prefix of vector-chunk counts per piece
  int np;
};

__global__ void __launch_bounds__(kBlock) multi_copy_kernel(CopyArgs a) {
  const uint64_t total = a.start[a.np];
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * kBlock;
  for (uint64_t q = static_cast<uint64_t>(blockIdx.x) * kBlock + threadIdx.x; q < total; q += stride) {
    int k = 0;
    while (q >= a.start[k + 1]) ++k;
    const CopyPiece& pc = a.p[k];
    const uint64_t c = q - a.start[k];
    // head: elements before the first 16-byte aligned destination address
    const uint64_t head = (4 - ((reinterpret_cast<uintptr_t>(pc.dst) >> 2) & 3)) & 3;
    const uint64_t h = head < pc.len ? head : pc.len;
    if (c == 0) {
      for (uint64_t e = 0; e < h; ++e) pc.dst[e] = pc.src[e];
      // tail after the last full vector
      const uint64_t body = (pc.len - h) / 4 * 4;
      for (uint64_t e = h + body; e < pc.len; ++e) pc.dst[e] = pc.src[e];
    }
    const uint64_t e0 = h + c * 4;
    if (e0 + 4 > pc.len) continue;
    uint4 v;
    const uint32_t* s = pc.src + e0;
    if (c > 0 && e0 + 8 <= pc.len) {
      v = load4_realigned(s);   // both aligned vectors inside the piece
    } else {
      v.x = s[0];
      v.y = s[1];
      v.z = s[2];
      v.w = s[3];
    }
    *reinterpret_cast<uint4*>(pc.dst + e0) = v;
  }
}

// Rooms taken for an output before its size is known, from the largest to the
// smallest: the output goes to the smallest one that holds it.
constexpr uint32_t kRooms = 4;
struct Rooms {
  uint32_t n;
  uint64_t rows[kRooms];
  uint32_t* cols[kRooms][VG_MAX_COLS];
  __host__ __device__ uint32_t of(uint64_t total) const {   // (total <= rows[0])
    uint32_t k = 0;
    while (k + 1 < n && total <= rows[k + 1]) ++k;
    return k;
  }
};

// ---------------------------------------------------------------------------
// Adjacent-unique compaction (thrust::unique over zipped columns): one kernel
// finds the rows to drop, a second one moves the others if there are any to
// drop (most results of a query have none).  Relations of one tile take one
// launch (100 rows: 34 us with two, 16.5 so).  Where repetitions are expected, up
// to kSoonRows, the second kernel is launched at once, and has nothing to do if
// none are dropped: 10,000 rows, half of them dropped, 31 -> 24 us, none dropped
// 16 -> 20.  Otherwise the first one is waited for in between.
// ---------------------------------------------------------------------------
struct UniqueArgs {
  const uint32_t* in[VG_MAX_COLS];
  uint32_t ncols;
  uint64_t n;
  uint32_t* keep;         // bit i of word w: row 32 w + i stays (whole tiles)
};
constexpr uint64_t kSoonRows = 1u << 19;
struct UniqueHost {    // page-locked
  uint64_t dropped;
  DeviceErrors err;    // what the work before left, so that no copy of its own is needed
};
struct UniqueTotal {   // zeroed before the first kernel, with the tiles' counts that follow it
  unsigned long long dropped;
  uint32_t done;       // finished blocks
  uint32_t pad;
};

// Which of the rows r0 .. r0 + 7 (of those below n) differ from the one before.
// Columns are compared from the last to the first, and only while some row
// still equals the one before it: in sorted rows and in join outputs the last
// columns change fastest, so most of the time one column is read (7.4e7 rows of
// 8 columns without repetitions: 0.13 ms, and 1.41 ms when all were read, and
// once more to be written elsewhere).  diff: the last column's.
__device__ __forceinline__ uint32_t unique_kept(const UniqueArgs& a, uint64_t r0, uint32_t diff, uint32_t& here) {
  static_assert(kRows == 8, "unique_diff_bits and compact_store take 8 rows per thread");
  here = r0 >= a.n ? 0u : a.n - r0 < kRows ? static_cast<uint32_t>(a.n - r0) : kRows;
  const uint32_t all = (1u << here) - 1u;
  if (r0 == 0) diff |= 1u;
#pragma unroll 1
  for (int c = static_cast<int>(a.ncols) - 2; c >= 0 && (diff & all) != all; --c)
    diff |= unique_diff_bits(a.in[c], a.n, r0);
  return diff & all;
}

// The flags, each tile's count of rows to drop, and (by the last block) every
// tile's first output row, so that the move waits for nothing.
__global__ void __launch_bounds__(kBlock, 6) unique_flags_kernel(const __grid_constant__ UniqueArgs a,
                                                                 UniqueTotal* tot, uint32_t* tile_drops,
                                                                 uint64_t* __restrict__ tile_first, uint32_t tiles,
                                                                 const DeviceErrors* err, UniqueHost* host) {
  __shared__ uint64_t s_scan[kBlock / 32 + 1];
  __shared__ uint64_t s_dropped;
  uint32_t drop = 0;
  const uint32_t* last = a.in[a.ncols - 1];
  constexpr int kIn = 2;   // tiles whose last columns are read together
  for (uint32_t t0 = blockIdx.x; t0 < tiles; t0 += kIn * gridDim.x) {
    uint32_t diff[kIn];
#pragma unroll
    for (int q = 0; q < kIn; ++q)
      diff[q] = unique_diff_bits(last, a.n, static_cast<uint64_t>(t0 + q * gridDim.x) * kTileRows + threadIdx.x * kRows);
#pragma unroll
    for (int q = 0; q < kIn; ++q) {
      const uint32_t tile = t0 + q * gridDim.x;
      if (tile >= tiles) break;
      const uint64_t r0 = static_cast<uint64_t>(tile) * kTileRows + threadIdx.x * kRows;
      uint32_t here;
      const uint32_t kept = unique_kept(a, r0, diff[q], here);
      reinterpret_cast<uint8_t*>(a.keep)[r0 / 8] = static_cast<uint8_t>(kept);
      const uint32_t d = here - __popc(kept);
      if (__any_sync(0xffffffffu, d)) {
        const uint32_t w = __reduce_add_sync(0xffffffffu, d);
        if (lane_id() == 0) atomicAdd(&tile_drops[tile], w);
        drop += w;
      }
    }
  }
  if (lane_id() == 0 && drop) atomicAdd(&tot->dropped, static_cast<unsigned long long>(drop));
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_dropped = 0;
    if (atomicAdd(&tot->done, 1u) == gridDim.x - 1) {
      __threadfence();
      s_dropped = ld_status_u64(reinterpret_cast<const uint64_t*>(&tot->dropped));
      host->dropped = s_dropped;
      host->err = *err;
    }
  }
  __syncthreads();
  if (s_dropped == 0) return;   // (or not the last block)
  constexpr uint32_t kEach = 4;
  uint64_t before = 0;
  for (uint32_t t0 = 0; t0 < tiles; t0 += kBlock * kEach) {
    uint32_t v[kEach];
    uint64_t mine = 0, all;
#pragma unroll
    for (uint32_t k = 0; k < kEach; ++k) {
      const uint32_t t = t0 + threadIdx.x * kEach + k;
      v[k] = t < tiles ? __ldcg(tile_drops + t) : 0u;
      mine += v[k];
    }
    uint64_t at = before + block_excl_scan64<kBlock>(mine, all, s_scan);
#pragma unroll
    for (uint32_t k = 0; k < kEach; ++k) {
      const uint32_t t = t0 + threadIdx.x * kEach + k;
      if (t < tiles) tile_first[t] = static_cast<uint64_t>(t) * kTileRows - at;
      at += v[k];
    }
    before += all;
  }
}

// A warp takes 256 rows of a tile, 32 consecutive ones at a time, whose bits
// tell each lane where its row goes: loads and stores coalesce, and nothing is
// staged or waited for.  A column is loaded, all of its rows, while the bits or
// the column before it are on their way: 20M rows of 3 columns, 1% of them
// repeated, take 76 us (6.3 TB/s), and 154 with each column's loads after its
// row numbers and stores.
__global__ void __launch_bounds__(kBlock, 5) unique_move_kernel(const __grid_constant__ UniqueArgs a,
                                                                const UniqueTotal* __restrict__ tot,
                                                                const uint64_t* __restrict__ tile_first,
                                                                const __grid_constant__ Rooms rooms) {
  constexpr uint32_t kWords = kTileRows / 32;
  static_assert(kWords == 64 && kRows == 8, "two words of the tile per lane, eight per warp");
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  const uint64_t tile = blockIdx.x, r0 = tile * kTileRows + warp * (32u * kRows) + lane;
  const uint64_t dropped = __ldcg(&tot->dropped);
  if (dropped == 0) return;
  const uint32_t w0 = __ldg(a.keep + tile * kWords + lane), w1 = __ldg(a.keep + tile * kWords + 32 + lane);
  const uint64_t to = __ldg(tile_first + tile);
  uint32_t v[kRows], next[kRows];
#pragma unroll
  for (int i = 0; i < kRows; ++i) v[i] = r0 + i * 32 < a.n ? __ldg(a.in[0] + r0 + i * 32) : 0u;
  const uint32_t i0 = warp_incl_scan(__popc(w0)), i1 = warp_incl_scan(__popc(w1));
  const uint32_t first_half = __shfl_sync(0xffffffffu, i0, 31);
  const bool lower = warp < 4;
  const uint32_t word = lower ? w0 : w1, before = lower ? i0 - __popc(w0) : first_half + i1 - __popc(w1);
  uint32_t at[kRows];       // the row's place in the tile's output (all ones: dropped)
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const uint32_t k = (warp * kRows + i) & 31u, m = __shfl_sync(0xffffffffu, word, k);
    at[i] = __shfl_sync(0xffffffffu, before, k) + __popc(m & lanemask_lt());
    if (!(m >> lane & 1u)) at[i] = 0xffffffffu;
  }
  uint32_t* const* cols = rooms.cols[rooms.of(a.n - dropped)];
  for (uint32_t c = 0; c < a.ncols; ++c) {
    if (c + 1 < a.ncols) {
#pragma unroll
      for (int i = 0; i < kRows; ++i) next[i] = at[i] != 0xffffffffu ? __ldg(a.in[c + 1] + r0 + i * 32) : 0u;
    }
    uint32_t* out = cols[c] + to;
#pragma unroll
    for (int i = 0; i < kRows; ++i)
      if (at[i] != 0xffffffffu) out[at[i]] = v[i];
#pragma unroll
    for (int i = 0; i < kRows; ++i) v[i] = next[i];
  }
}

// A relation of one tile, by one block.
__global__ void __launch_bounds__(kBlock) unique_tile_kernel(const __grid_constant__ UniqueArgs a,
                                                             const __grid_constant__ Rooms rooms,
                                                             const DeviceErrors* err, UniqueHost* host) {
  __shared__ uint32_t s_scan[kBlock / 32 + 1];
  __shared__ uint32_t s_keep[2 * kTileRows];
  const uint64_t r0 = static_cast<uint64_t>(threadIdx.x) * kRows;
  uint32_t here, kept;
  const uint32_t diff = unique_kept(a, r0, unique_diff_bits(a.in[a.ncols - 1], a.n, r0), here);
  const uint32_t e = block_excl_scan<kBlock>(__popc(diff), kept, s_scan);
  if (threadIdx.x == 0) {
    host->dropped = a.n - kept;
    host->err = *err;
  }
  if (kept < a.n)
    compact_store<kBlock>(a.in, rooms.cols[rooms.of(kept)], a.ncols, a.n, r0, diff, e, kept, 0, s_keep);
}

// ---------------------------------------------------------------------------
// Join of two relations.  Count and scan: lower bound, match count and output
// offset of every left key (vg_join_tile.cuh).  Write: every output row finds
// its left row by the offsets (load-balanced across heavy keys) and copies
// its columns.
// ---------------------------------------------------------------------------
template <bool TWO>
struct KeysOf {
  using K = OneKeys;
  static __host__ __device__ K of(const uint32_t* c0, const uint32_t*) { return K{c0}; }
};
template <>
struct KeysOf<true> {
  using K = PairKeys;
  static __host__ __device__ K of(const uint32_t* c0, const uint32_t* c1) { return K{c0, c1}; }
};

// Every tile's right-key window, one warp per tile (both ends at once).
template <bool TWO>
__global__ void __launch_bounds__(kJcBlock) join_window_kernel(typename KeysOf<TWO>::K L, uint64_t nl,
                                                               typename KeysOf<TWO>::K R, uint64_t nr,
                                                               uint64_t tiles, uint2* __restrict__ win) {
  const uint64_t nw = static_cast<uint64_t>(gridDim.x) * (kJcBlock / 32);
  for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * (kJcBlock / 32) + (threadIdx.x >> 5); t < tiles; t += nw) {
    const uint64_t i0 = t * kJcTile, i1 = (i0 + kJcTile < nl ? i0 + kJcTile : nl) - 1;
    uint64_t w0, w1;
    warp_bound_pair_of<false, true>(R, nr, L(i0), L(i1), w0, w1);
    if ((threadIdx.x & 31) == 0) win[t] = make_uint2(static_cast<uint32_t>(w0), static_cast<uint32_t>(w1));
  }
}

// One block per 2048 left keys.  The window comes from join_window_kernel where
// there are more tiles than the GPU runs at a time (a block's own search is
// five rounds of global loads before its copy can start), else warp 0 finds it.
template <bool TWO, typename Off>
__global__ void __launch_bounds__(kJcBlock, 4) join_count_kernel(
    typename KeysOf<TWO>::K L, uint64_t nl, typename KeysOf<TWO>::K R, uint64_t nr, const uint2* __restrict__ win,
    JoinCounts<Off> c, uint32_t* done, uint64_t* total, DeviceErrors* err) {
  __shared__ JoinCountSmem sm;
  __shared__ uint64_t s_scan[kJcBlock / 32 + 1];
  const uint32_t tile = blockIdx.x;
  const uint64_t i0 = static_cast<uint64_t>(tile) * kJcTile, i1 = i0 + kJcTile < nl ? i0 + kJcTile : nl;
  typename KeysOf<TWO>::K::T key[kJcKeys];
  jc_load_keys(L, i0 + static_cast<uint64_t>(threadIdx.x) * kJcKeys, i1, key);
  if (threadIdx.x < 32) {
    uint64_t w0, w1;
    if (win) {
      const uint2 w = win[tile];
      w0 = w.x;
      w1 = w.y;
    } else {
      warp_bound_pair_of<false, true>(R, nr, L(i0), L(i1 - 1), w0, w1);
    }
    if (threadIdx.x == 0) {
      if constexpr (TWO) jc_issue_pair_window(w0, w1, sm);
      else jc_issue_window(R.c0, w0, w1, sm);
    }
  }
  __syncthreads();
  uint32_t cnt[kJcKeys], lov[kJcKeys];
  if constexpr (TWO) jc_count_staged_pairs(key, nl, R, i0, lov, cnt, sm);
  else jc_count_staged(key, nl, R.c0, i0, lov, cnt, sm, err);
  jc_finish_tile(i0, lov, cnt, sm, s_scan, tile, gridDim.x, nl, c, done, total, err);
}

// What the host reads of a join (page-locked memory that the write kernel
// stores to).
constexpr uint32_t kTailKeys = 100;   // column 0 of smaller outputs is scanned for empty intervals
struct JoinTail {
  uint64_t total;
  DeviceErrors err;
  uint32_t first, last;        // of column 0, when rows were written
  uint32_t c0[kTailKeys];      // column 0, when fewer rows than that were written
};
static_assert(sizeof(JoinTail) <= Ctx::kSmallWords * sizeof(uint64_t), "the tail fits the small staging buffer");

// Groups [x, y) of left rows of every output tile, one warp per tile.
__global__ void __launch_bounds__(kJwBlock) join_ranges_kernel(JoinGroups<uint32_t> groups, uint64_t ng,
                                                               uint64_t total, uint64_t tiles, uint32_t tile_rows,
                                                               uint2* __restrict__ ranges) {
  const uint64_t nw = static_cast<uint64_t>(gridDim.x) * (kJwBlock / 32);
  for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * (kJwBlock / 32) + (threadIdx.x >> 5); t < tiles; t += nw) {
    const uint64_t kb = t * tile_rows, kend = kb + tile_rows < total ? kb + tile_rows : total;
    uint64_t a, b;
    warp_bound_pair_of<true, true>(groups, ng, static_cast<uint32_t>(kb), static_cast<uint32_t>(kend - 1), a, b);
    if ((threadIdx.x & 31) == 0) ranges[t] = make_uint2(static_cast<uint32_t>(a - 1), static_cast<uint32_t>(b));
  }
}

// The output rows, kJwBlock * ROWS per tile; a block loops over tiles.  The
// row count comes from o.total or, when total_dev is given, from the device:
// the rows then go to one of `rooms`, and nothing is written when there are
// more than the first holds.  Nothing is written either after a wait that gave
// up (the offsets are wrong).  Ranges come from join_ranges_kernel or are found
// by warp 0.
template <int ROWS, typename Off>
__global__ void __launch_bounds__(kJwBlock, 5) join_write_kernel(JoinOutOf<Off> o, const uint64_t* total_dev,
                                                                 const __grid_constant__ Rooms rooms,
                                                                 const uint2* __restrict__ ranges,
                                                                 const DeviceErrors* err, JoinTail* tail) {
  constexpr uint32_t kTile = kJwBlock * ROWS;
  __shared__ JoinOutOf<Off> s_o;
  __shared__ JwStage<ROWS> s_stage;
  __shared__ uint64_t s_range[2];
  const uint64_t total = total_dev ? *total_dev : o.total;
  const DeviceErrors e = *err;
  if (tail && blockIdx.x == 0 && threadIdx.x == 0) {
    tail->total = total;
    tail->err = e;
  }
  if (e.timeout || (total_dev && total > rooms.rows[0])) return;
  if (threadIdx.x == 0) {
    s_o = o;
    if (total_dev) {
      const uint32_t k = rooms.of(total);
      for (uint32_t c = 0; c < o.nlc + o.nrc; ++c) s_o.oc[c] = rooms.cols[k][c];
    }
  }
  const uint64_t tiles = (total + kTile - 1) / kTile;
#pragma unroll 1
  for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint64_t kb = tile * kTile, kend = kb + kTile < total ? kb + kTile : total;
    __syncthreads();   // s_o is set; the previous tile's readers of the shared arrays are done
    jw_clear(s_stage);
    if (threadIdx.x < 32) {
      uint64_t a, b;
      if (ranges) {
        const uint2 r = ranges[tile];
        a = r.x;
        b = r.y;
      } else {
        warp_bound_pair_of<true, true>(s_o.groups(), s_o.ngroups(), static_cast<Off>(kb), static_cast<Off>(kend - 1), a, b);
        --a;
      }
      if (threadIdx.x == 0) {
        s_range[0] = a;
        s_range[1] = b;
      }
    }
    __syncthreads();
    jw_write_tile<ROWS>(s_o, kb, kend, s_range[0], s_range[1], s_stage);
    if (tail) {   // each by the thread that wrote the row
      const uint32_t* c0 = s_o.oc[0];
      if (tile == 0 && threadIdx.x == 0) tail->first = c0[0];
      if (tile == tiles - 1 && threadIdx.x == (total - 1 - kb) % kJwBlock) tail->last = c0[total - 1];
      if (total < kTailKeys && threadIdx.x < total) tail->c0[threadIdx.x] = c0[threadIdx.x];
    }
  }
}

// Tiles from which the windows and ranges are found by kernels of their own.
// (blocks of one join that run at a time: 4 or 5 per SM)
bool many_tiles(int num_sms, uint64_t tiles) { return tiles > 4ull * static_cast<uint64_t>(num_sms); }

template <bool TWO, typename Off>
void launch_count(cudaStream_t stream, const Rel& l, const Rel& r, const uint2* win,
                  const JoinCounts<Off>& c, uint32_t* done, uint64_t* total, DeviceErrors* err) {
  const unsigned tiles = static_cast<unsigned>(div_up(l.nrows, kJcTile));
  join_count_kernel<TWO, Off><<<tiles, kJcBlock, 0, stream>>>(
      KeysOf<TWO>::of(l.cols[0], TWO ? l.cols[1] : nullptr), l.nrows,
      KeysOf<TWO>::of(r.cols[0], TWO ? r.cols[1] : nullptr), r.nrows, win, c, done, total, err);
  VG_CUDA(cudaGetLastError());
}

template <typename Off>
JoinOutOf<Off> join_out(const Rel& l, const Rel& r, uint32_t nk, const JoinCounts<Off>& c, uint64_t total,
                        uint32_t* const* oc) {
  JoinOutOf<Off> o{};
  o.cnt = c;
  o.nl = l.nrows;
  o.total = total;
  for (uint32_t c = 0; c < l.ncols; ++c) o.lc[c] = l.cols[c];
  for (uint32_t c = nk; c < r.ncols; ++c) o.rc[c - nk] = r.cols[c];
  o.nlc = l.ncols;
  o.nrc = r.ncols - nk;
  for (uint32_t c = 0; oc && c < o.nlc + o.nrc; ++c) o.oc[c] = oc[c];
  return o;
}

// ---------------------------------------------------------------------------
// Rows packed into one 64-bit key each (column 0 on top), for sorts over all
// columns.
// ---------------------------------------------------------------------------
struct PackCols {
  uint32_t* col[VG_MAX_COLS];
  uint32_t shift[VG_MAX_COLS];   // the column's lowest key bit
  uint64_t mask[VG_MAX_COLS];    // its values' bits (0: a column of zeros)
  uint32_t ncols;
};

// max[c] = the largest value of column c (blocks take columns in turn; one
// atomic per block and column: with one per warp, 9,700 on each word, three
// columns of 5M rows took 31 us, now 15).
__global__ void __launch_bounds__(kBlock) column_maxima_kernel(PackCols a, uint64_t n, uint32_t* max_out) {
  __shared__ uint32_t s_max[kBlock / 32];
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * kBlock;
  for (uint32_t c = 0; c < a.ncols; ++c) {
    uint32_t m = 0;
    const uint64_t t = static_cast<uint64_t>(blockIdx.x) * kBlock + threadIdx.x;
    uint64_t nv = 0;
    if ((reinterpret_cast<uintptr_t>(a.col[c]) & 15u) == 0) {
      nv = n / 4;
      const uint4* v = reinterpret_cast<const uint4*>(a.col[c]);
#pragma unroll 4
      for (uint64_t i = t; i < nv; i += stride) {
        const uint4 x = __ldg(v + i);
        m = max(m, max(max(x.x, x.y), max(x.z, x.w)));
      }
    }
    for (uint64_t i = nv * 4 + t; i < n; i += stride) m = max(m, __ldg(a.col[c] + i));
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane_id() == 0) s_max[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
      m = __reduce_max_sync(0xffffffffu, threadIdx.x < kBlock / 32 ? s_max[threadIdx.x] : 0u);
      if (threadIdx.x == 0 && m) atomicMax(&max_out[c], m);
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kBlock) pack_rows_kernel(PackCols a, uint64_t n, uint64_t* __restrict__ keys,
                                                           DigitList dl, unsigned long long* __restrict__ hist,
                                                           uint64_t* __restrict__ bases, uint32_t* done) {
  extern __shared__ uint32_t sh[];   // [dl.n][kRadixValues]
  digit_counts_init<kBlock>(dl, sh);
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * kBlock;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * kBlock + threadIdx.x; i < n; i += stride) {
    uint64_t k = 0;
#pragma unroll
    for (int c = 0; c < VG_MAX_COLS; ++c)
      if (c < static_cast<int>(a.ncols) && a.mask[c]) k |= static_cast<uint64_t>(__ldg(a.col[c] + i)) << a.shift[c];
    keys[i] = k;
    digit_counts_add(dl, sh, k);
  }
  digit_counts_finish<kBlock>(dl, sh, hist, bases, done);
}

__global__ void __launch_bounds__(kBlock) unpack_rows_kernel(PackCols a, uint64_t n, const uint64_t* __restrict__ keys) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * kBlock;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * kBlock + threadIdx.x; i < n; i += stride) {
    const uint64_t k = keys[i];
#pragma unroll
    for (int c = 0; c < VG_MAX_COLS; ++c)
      if (c < static_cast<int>(a.ncols)) a.col[c][i] = static_cast<uint32_t>((k >> a.shift[c]) & a.mask[c]);
  }
}

// What the host reads of a row sort (page-locked).
struct RowsHost {
  uint32_t big;        // a group of more than kRowGroup rows was left as it was
  uint32_t pad;
  DeviceErrors err;
};
struct RowsDone {      // zeroed before the launch
  uint32_t big;
  uint32_t done;
};
constexpr uint32_t kRowGroup = 64;

// Keys in order of their top bits (equal under `top`) to rows in full order:
// the rows of a group of equal top bits are ranked by whole keys, as the index
// build ranks the objects of a subject and predicate.  The tile's keys, 64 on
// either side and the group heads lie in shared memory; a row's place is the
// number of rows of its group that go before it.
__global__ void __launch_bounds__(kBlock) unpack_groups_kernel(PackCols a, uint64_t n, const uint64_t* __restrict__ keys,
                                                               uint64_t top, RowsDone* st, const DeviceErrors* err,
                                                               RowsHost* host) {
  constexpr uint32_t kHalo = kRowGroup;
  __shared__ uint64_t s_key[kTileRows + 2 * kHalo];
  __shared__ uint32_t s_head[(kTileRows + 2 * kHalo) / 32];
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  const uint64_t t0 = static_cast<uint64_t>(blockIdx.x) * kTileRows;
  // every 32 rows of the tile and its halos: keys and heads (rows outside the
  // relation count as heads)
  for (uint32_t g = warp; g < (kTileRows + 2 * kHalo) / 32; g += kBlock / 32) {
    const uint32_t x = g * 32 + lane;
    const bool in = t0 + x >= kHalo && t0 + x - kHalo < n;
    const uint64_t r = t0 + x - kHalo;
    const uint64_t k = in ? keys[r] : 0ull;
    uint64_t pv = __shfl_up_sync(0xffffffffu, k, 1);
    if (lane == 0) pv = in && r > 0 ? keys[r - 1] : 0ull;
    s_key[x] = k;
    const uint32_t h = __ballot_sync(0xffffffffu, !in || r == 0 || ((k ^ pv) & top));
    if (lane == 0) s_head[g] = h;
  }
  __syncthreads();
  bool big = false;
#pragma unroll 1
  for (int i = 0; i < kRows; ++i) {
    const uint32_t x = kHalo + warp * (32u * kRows) + i * 32u + lane, w = x >> 5;
    const uint64_t r = t0 + x - kHalo;
    if (r >= n) break;
    const uint32_t upto = 0xffffffffu >> (31u - lane);   // bits 0..lane (x & 31 == lane)
    // [b, e): the group, as far as it lies within 64 rows of this one
    uint32_t b = 0, e = 0xffffffffu;
    if (s_head[w] & upto) b = w * 32 + 31 - __clz(s_head[w] & upto);
    else if (s_head[w - 1]) b = w * 32 - 1 - __clz(s_head[w - 1]);
    else if (s_head[w - 2]) b = w * 32 - 33 - __clz(s_head[w - 2]);
    if (s_head[w] & ~upto) e = w * 32 + __ffs(s_head[w] & ~upto) - 1;
    else if (s_head[w + 1]) e = w * 32 + 31 + __ffs(s_head[w + 1]);
    else if (s_head[w + 2]) e = w * 32 + 63 + __ffs(s_head[w + 2]);
    const uint64_t mine = s_key[x];
    uint32_t at = x;
    // (b == 0 is not a found head: see the index build's kernel)
    if (b != 0 && e != 0xffffffffu && e - b <= kRowGroup) {
      at = b;
      for (uint32_t j = b; j < e; ++j) {
        const uint64_t v = s_key[j];
        at += (v < mine || (v == mine && j < x)) ? 1u : 0u;
      }
    } else {
      big = true;
    }
    const uint64_t to = t0 + at - kHalo;
#pragma unroll
    for (int c = 0; c < VG_MAX_COLS; ++c)
      if (c < static_cast<int>(a.ncols)) a.col[c][to] = static_cast<uint32_t>((mine >> a.shift[c]) & a.mask[c]);
  }
  if (__syncthreads_or(big) && threadIdx.x == 0) atomicExch(&st->big, 1u);
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&st->done, 1u) == gridDim.x - 1) {
      __threadfence();
      host->big = atomicAdd(&st->big, 0u);
      host->err = *err;
    }
  }
}

struct GatherCols {
  const uint32_t* in[VG_MAX_COLS];
  uint32_t* out[VG_MAX_COLS];
  uint32_t ncols;
};

// Four rows per thread at a time, kBlock apart: their row numbers, then each
// column's four reads are in flight together.
__global__ void __launch_bounds__(kBlock) gather_kernel(const uint32_t* __restrict__ perm, uint64_t n,
                                                        GatherCols g) {
  constexpr int kIn = 4;
  const uint64_t step = static_cast<uint64_t>(gridDim.x) * kBlock * kIn;
  for (uint64_t r = static_cast<uint64_t>(blockIdx.x) * kBlock * kIn + threadIdx.x; r < n; r += step) {
    uint32_t p[kIn], v[kIn];
#pragma unroll
    for (int q = 0; q < kIn; ++q) p[q] = r + q * kBlock < n ? perm[r + q * kBlock] : 0u;
    for (uint32_t c = 0; c < g.ncols; ++c) {
#pragma unroll
      for (int q = 0; q < kIn; ++q) v[q] = __ldg(g.in[c] + p[q]);
#pragma unroll
      for (int q = 0; q < kIn; ++q)
        if (r + q * kBlock < n) g.out[c][r + q * kBlock] = v[q];
    }
  }
}
}  // namespace

Rel rel_alloc(Ctx& ctx, uint32_t ncols, uint64_t nrows) {
  if (ncols > VG_MAX_COLS) fail(VG_ERR_UNSUPPORTED, "more than 9 columns");
  Rel r;
  r.nrows = nrows;
  try {
    for (; r.ncols < ncols; ++r.ncols) r.cols[r.ncols] = ctx.alloc<uint32_t>(nrows);
  } catch (...) {
    rel_free(ctx, r);
    throw;
  }
  return r;
}

void rel_free(Ctx& ctx, Rel& r) {
  for (uint32_t c = 0; c < r.ncols; ++c) {
    if (!(r.borrowed >> c & 1u)) ctx.free(r.cols[c]);
    r.cols[c] = nullptr;
  }
  r.ncols = 0;
  r.nrows = 0;
  r.borrowed = 0;
}

void rel_drop_col(Ctx& ctx, Rel& r, uint32_t c) {
  if (!(r.borrowed >> c & 1u)) ctx.free(r.cols[c]);
  r.borrowed &= ~(1u << c);
}

void rel_own(Ctx& ctx, Rel& r) {
  for (uint32_t c = 0; c < r.ncols; ++c) {
    if (!(r.borrowed >> c & 1u)) continue;
    uint32_t* o = ctx.alloc<uint32_t>(r.nrows);
    if (r.nrows)
      VG_CUDA(cudaMemcpyAsync(o, r.cols[c], r.nrows * sizeof(uint32_t), cudaMemcpyDeviceToDevice, ctx.stream));
    r.cols[c] = o;
    r.borrowed &= ~(1u << c);
  }
}

void multi_copy(Ctx& ctx, const CopyPiece* pieces, int np) {
  if (np > 16) fail(VG_ERR_INVALID, "multi_copy: too many pieces");
  CopyArgs a{};
  a.np = 0;
  a.start[0] = 0;
  for (int k = 0; k < np; ++k) {
    if (pieces[k].len == 0) continue;
    const uint64_t head = (4 - ((reinterpret_cast<uintptr_t>(pieces[k].dst) >> 2) & 3)) & 3;
    const uint64_t h = head < pieces[k].len ? head : pieces[k].len;
    const uint64_t chunks = (pieces[k].len - h) / 4;
    a.p[a.np] = pieces[k];
    a.start[a.np + 1] = a.start[a.np] + (chunks ? chunks : 1);
    ++a.np;
  }
  if (a.np == 0) return;
  double bytes = 0;
  for (int k = 0; k < a.np; ++k) bytes += 8.0 * a.p[k].len;
  ctx.launch("select_copy", bytes,
             [&] { multi_copy_kernel<<<grid_for(ctx, a.start[a.np], 2), kBlock, 0, ctx.stream>>>(a); });
  VG_CUDA(cudaGetLastError());
}

// Rooms of `asked` rows (0: none) and more, as their blocks allow, in falling
// order; none (false) where they would take more than a quarter of the largest
// free block (blocks of a size class are carved from it for good), or large
// ones would not leave as much again.
static bool take_rooms(Ctx& ctx, uint32_t ncols, std::initializer_list<uint64_t> asked, Rooms& rooms) {
  uint64_t free_bytes = 0;   // asked of the largest free block
  rooms = Rooms{};
  for (uint64_t rows : asked) {
    const uint64_t bytes = Arena::block_bytes(rows * sizeof(uint32_t)), room = bytes / sizeof(uint32_t);
    if (rows == 0 || (rooms.n && room >= rooms.rows[rooms.n - 1])) continue;
    rooms.rows[rooms.n++] = room;
    free_bytes += (bytes > Arena::kSmallMax ? 2 : 4) * ncols * bytes;
  }
  bool fits = free_bytes <= ctx.arena.largest_free();
  for (uint32_t k = 0; k < rooms.n && fits; ++k)
    for (uint32_t c = 0; c < ncols && fits; ++c) {
      rooms.cols[k][c] = static_cast<uint32_t*>(ctx.arena.try_alloc(rooms.rows[k] * sizeof(uint32_t)));
      fits = rooms.cols[k][c] != nullptr;
    }
  return fits;
}

// Gives the rooms back, but the one numbered `but`.
static void free_rooms(Ctx& ctx, uint32_t ncols, const Rooms& rooms, uint32_t but = kRooms) {
  for (uint32_t k = 0; k < rooms.n; ++k)
    for (uint32_t c = 0; c < ncols && k != but; ++c) ctx.free(rooms.cols[k][c]);
}

// Gives columns that lie in blocks of `bytes` the blocks that their rows ask
// for: a large block's tail goes back to the arena, and rows that belong in a
// size class (another one) are moved there, unless there is no block to be had.
// True when they are: the copy is then on the stream.
static bool fit_columns(Ctx& ctx, Rel& r, size_t bytes) {
  const size_t own = std::max<uint64_t>(r.nrows, 1) * sizeof(uint32_t), block = Arena::block_bytes(own);
  if (block == bytes || block > Arena::kSmallMax) {
    for (uint32_t c = 0; c < r.ncols; ++c) ctx.arena.shrink(r.cols[c], own);
    return false;
  }
  Rel to;
  to.nrows = r.nrows;
  CopyPiece pieces[VG_MAX_COLS];
  for (; to.ncols < r.ncols; ++to.ncols) {
    auto* p = static_cast<uint32_t*>(ctx.arena.try_alloc(own));
    if (!p) {
      rel_free(ctx, to);
      return false;
    }
    to.cols[to.ncols] = p;
    pieces[to.ncols] = {r.cols[to.ncols], p, r.nrows};
  }
  multi_copy(ctx, pieces, static_cast<int>(r.ncols));
  rel_free(ctx, r);
  r = to;
  return r.nrows > 0;
}

// The relation of `rows` rows that a kernel wrote to its room; the others go
// back.  True when a copy to blocks of its size is on the stream.
static bool keep_room(Ctx& ctx, uint32_t ncols, const Rooms& rooms, uint64_t rows, Rel& out) {
  const uint32_t k = rooms.of(rows);
  free_rooms(ctx, ncols, rooms, k);
  out = Rel();
  out.ncols = ncols;
  out.nrows = rows;
  std::copy(rooms.cols[k], rooms.cols[k] + ncols, out.cols);
  return fit_columns(ctx, out, rooms.rows[k] * sizeof(uint32_t));
}

bool join(Ctx& ctx, const Rel& l, const Rel& r, bool two_keys, Rel& out, JoinEnds* ends) {
  const uint32_t nk = two_keys ? 2 : 1;
  if (l.ncols < nk || r.ncols < nk) fail(VG_ERR_INVALID, "join: missing key columns");
  const uint32_t ncols = l.ncols + r.ncols - nk;
  if (ncols > VG_MAX_COLS) fail(VG_ERR_UNSUPPORTED, "join output has more than 9 columns");
  if (l.nrows > 0xFFFFFFFFull || r.nrows > 0xFFFFFFFFull)
    fail(VG_ERR_OVERFLOW, "join inputs are limited to 2^32 rows");
  if (ends) *ends = JoinEnds();
  if (l.nrows == 0 || r.nrows == 0) {
    out = rel_alloc(ctx, ncols, 0);
    return false;
  }
  const uint64_t tiles = div_up(l.nrows, kJcTile);
  if (tiles > 0x7FFFFFFFull) fail(VG_ERR_OVERFLOW, "join: too many tiles");
  const uint64_t ngroups = div_up(l.nrows, kJcKeys);
  Scratch<uint32_t> lo(ctx, ngroups * kJcKeys), offs(ctx, ngroups * kJcKeys), start(ctx, ngroups);
  Scratch<uint8_t> match(ctx, ngroups);
  Scratch<uint64_t> z(ctx, tiles + 2);   // first output row of every tile, total, tiles done
  uint64_t* total = z.get() + tiles;
  const JoinCounts<uint32_t> cnt{lo.get(), offs.get(), start.get(), match.get(), z.get()};
  VG_CUDA(cudaMemsetAsync(total, 0, 2 * sizeof(uint64_t), ctx.stream));
  std::optional<Scratch<uint2>> win;
  if (many_tiles(ctx.num_sms, tiles)) {
    win.emplace(ctx, tiles);
    const unsigned wblocks =
        static_cast<unsigned>(std::min<uint64_t>(div_up(tiles, kJcBlock / 32), static_cast<uint64_t>(ctx.num_sms) * 8));
    ctx.launch("join_windows", 8.0 * tiles, [&] {
      if (two_keys)
        join_window_kernel<true><<<wblocks, kJcBlock, 0, ctx.stream>>>({l.cols[0], l.cols[1]}, l.nrows,
                                                                       {r.cols[0], r.cols[1]}, r.nrows, tiles,
                                                                       win->get());
      else
        join_window_kernel<false><<<wblocks, kJcBlock, 0, ctx.stream>>>({l.cols[0]}, l.nrows, {r.cols[0]}, r.nrows,
                                                                        tiles, win->get());
    });
    VG_CUDA(cudaGetLastError());
  }
  ctx.launch("join_count", 4.0 * nk * (l.nrows + r.nrows) + 8.0 * l.nrows, [&] {
    const uint2* w = win ? win->get() : nullptr;
    auto* done = reinterpret_cast<uint32_t*>(total + 1);
    if (two_keys) launch_count<true>(ctx.stream, l, r, w, cnt, done, total, ctx.d_err);
    else launch_count<false>(ctx.stream, l, r, w, cnt, done, total, ctx.d_err);
  });
  auto* tail = reinterpret_cast<JoinTail*>(ctx.h_small);
  auto finish = [&](uint64_t t) {
    if (ends && t > 0) {
      ends->first = tail->first;
      ends->last = tail->last;
      if (t < kTailKeys) ends->c0.assign(tail->c0, tail->c0 + t);
    }
  };
  // A small left side: room for its output is taken at once and the write
  // follows the count without the host in between (a round trip, copies and an
  // allocation, took 25 of 120 us at 3,000 rows); larger outputs are written
  // below.  There are several rooms, for twice the left rows, as many and half
  // of them, each a size class of the arena, of which the output fills the one
  // that it would have been given: a result holds no more than its rows ask for.
  // From kWideGuess rows on, where the columns are large blocks of the arena,
  // whose unused tails go back to it, there is also a room for eight times the
  // rows, and the write takes tiles of 2048 rows for its 512: 1M left rows with
  // 3.3M output rows 126 -> 91 us.  Where there is no room for the rooms, the
  // size is waited for.  kGuessRows bounds the memory (eight times 2^20 rows are
  // 32 MiB a column); the gain goes on above it: with 2^22, 1.1M left rows with as
  // many output rows take 40 us for 51 and 3M 71 for 93.
  if (l.nrows <= kGuessRows) {
    const bool wide = l.nrows >= kWideGuess;
    Rooms rooms;
    const bool fits = take_rooms(ctx, ncols, {wide ? 8 * l.nrows : 0, std::max<uint64_t>(1024, 2 * l.nrows), l.nrows,
                                              (l.nrows + 1) / 2}, rooms);
    if (fits) {
      constexpr int kRowsSmall = 2;
      const JoinOut o = join_out(l, r, nk, cnt, 0, nullptr);
      auto kernel = wide ? join_write_kernel<kRows, uint32_t> : join_write_kernel<kRowsSmall, uint32_t>;
      const uint64_t rows = static_cast<uint64_t>(kJwBlock) * (wide ? kRows : kRowsSmall);
      const unsigned grid =
          static_cast<unsigned>(std::min<uint64_t>(div_up(rooms.rows[0], rows), static_cast<uint64_t>(ctx.num_sms) * 5));
      ctx.launch("join_write", 0.0, [&] {
        kernel<<<grid, kJwBlock, 0, ctx.stream>>>(o, total, rooms, nullptr, ctx.d_err, tail);
      });
      VG_CUDA(cudaGetLastError());
      ctx.sync();
      const uint64_t t = tail->total;
      if (!tail->err.timeout && !tail->err.overflow && t <= rooms.rows[0]) {
        finish(t);
        ctx.add_bytes("join_write", 4.0 * t * (2.0 * ncols - 1));
        return keep_room(ctx, ncols, rooms, t, out);
      }
      free_rooms(ctx, ncols, rooms);
      ctx.raise_device_errors(tail->err);
    } else {
      free_rooms(ctx, ncols, rooms);
    }
  }
  // the total and the error record come back together: after a wait that gave
  // up the write must not run
  VG_CUDA(cudaMemcpyAsync(&tail->total, total, sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx.stream));
  VG_CUDA(cudaMemcpyAsync(&tail->err, ctx.d_err, sizeof(DeviceErrors), cudaMemcpyDeviceToHost, ctx.stream));
  ctx.sync();
  const uint64_t t = tail->total;
  ctx.raise_device_errors(tail->err);
  if (t > kMaxJoinRows) fail(VG_ERR_OVERFLOW, "join output exceeds 2^32 rows");
  const uint64_t otiles = div_up(t, static_cast<uint64_t>(kTileRows));
  std::optional<Scratch<uint2>> ranges;
  if (many_tiles(ctx.num_sms, otiles)) ranges.emplace(ctx, otiles);
  out = rel_alloc(ctx, ncols, t);   // (the last block that is asked for: nothing is lost where one is not to be had)
  if (t == 0) return false;
  const JoinOut o = join_out(l, r, nk, cnt, t, out.cols);
  if (ranges) {
    const unsigned rblocks = static_cast<unsigned>(
        std::min<uint64_t>(div_up(otiles, kJwBlock / 32), static_cast<uint64_t>(ctx.num_sms) * 8));
    ctx.launch("join_write_ranges", 8.0 * otiles, [&] {
      join_ranges_kernel<<<rblocks, kJwBlock, 0, ctx.stream>>>(o.groups(), ngroups, t, otiles, kTileRows,
                                                               ranges->get());
    });
    VG_CUDA(cudaGetLastError());
  }
  ctx.launch("join_write", 4.0 * t * (2.0 * ncols - 1), [&] {
    join_write_kernel<kRows, uint32_t><<<static_cast<unsigned>(otiles), kJwBlock, 0, ctx.stream>>>(
        o, nullptr, Rooms{}, ranges ? ranges->get() : nullptr, ctx.d_err, tail);
  });
  VG_CUDA(cudaGetLastError());
  ctx.sync();
  finish(t);
  return false;
}

uint64_t join_into(cudaStream_t stream, const Rel& l, const Rel& r, uint32_t* const* out_cols, uint64_t capacity,
                   const JoinCounts<uint64_t>& c, uint32_t* done, uint64_t* total, DeviceErrors* err) {
  if (l.nrows == 0 || r.nrows == 0) return 0;
  launch_count<false>(stream, l, r, nullptr, c, done, total, err);
  uint64_t t = 0;
  DeviceErrors he{};
  VG_CUDA(cudaMemcpyAsync(&t, total, sizeof(uint64_t), cudaMemcpyDeviceToHost, stream));
  VG_CUDA(cudaMemcpyAsync(&he, err, sizeof(he), cudaMemcpyDeviceToHost, stream));
  VG_CUDA(cudaStreamSynchronize(stream));
  // no write after a wait that gave up
  if (he.timeout) fail(VG_ERR_TIMEOUT, "join_into: a bounded device wait expired");
  if (t == 0 || t > capacity) return t;
  const JoinOutOf<uint64_t> o = join_out(l, r, 1, c, t, out_cols);
  join_write_kernel<kRows, uint64_t><<<static_cast<unsigned>(std::min<uint64_t>(div_up(t, kTileRows), 0x7FFFFFFFull)), kJwBlock,
                             0, stream>>>(o, nullptr, Rooms{}, nullptr, err, nullptr);
  VG_CUDA(cudaGetLastError());
  return t;
}

void gather_cols(Ctx& ctx, const uint32_t* const* in, uint32_t* const* out, uint32_t ncols,
                 const uint32_t* perm, uint64_t n) {
  if (n == 0 || ncols == 0) return;
  GatherCols g{};
  for (uint32_t c = 0; c < ncols; ++c) {
    g.in[c] = in[c];
    g.out[c] = out[c];
  }
  g.ncols = ncols;
  ctx.launch("gather", static_cast<double>(n) * (4.0 + 8.0 * ncols),
             [&] { gather_kernel<<<grid_for(ctx, n, 4), kBlock, 0, ctx.stream>>>(perm, n, g); });
  VG_CUDA(cudaGetLastError());
}

// Columns [first, r.ncols) of r in the order of perm.  Up to kTogether cells
// go in one launch (as far as the new columns fit the arena); larger columns
// go one by one, so that each one's random reads have the L2 cache to
// themselves (three columns of 8M rows: 0.145 ms one by one, 0.181 together).
static void permute_columns(Ctx& ctx, Rel& r, uint32_t first, const uint32_t* perm) {
  constexpr uint64_t kTogether = 4u << 20;
  const bool together = r.nrows * (r.ncols - first) <= kTogether;
  for (uint32_t c = first; c < r.ncols;) {
    const uint32_t *in[VG_MAX_COLS] = {r.cols[c]};
    uint32_t* out[VG_MAX_COLS] = {ctx.alloc<uint32_t>(r.nrows)};
    uint32_t k = 1;
    for (; together && c + k < r.ncols; ++k) {
      out[k] = static_cast<uint32_t*>(ctx.arena.try_alloc(r.nrows * sizeof(uint32_t)));
      if (!out[k]) break;
      in[k] = r.cols[c + k];
    }
    gather_cols(ctx, in, out, k, perm, r.nrows);
    for (uint32_t q = 0; q < k; ++q) {
      rel_drop_col(ctx, r, c + q);
      r.cols[c + q] = out[q];
    }
    c += k;
  }
}

// An owned copy of column c where it is a view.
static void own_column(Ctx& ctx, Rel& r, uint32_t c) {
  if (!(r.borrowed >> c & 1u)) return;
  Rel one;
  one.ncols = 1;
  one.nrows = r.nrows;
  one.cols[0] = r.cols[c];
  one.borrowed = 1;
  rel_own(ctx, one);
  r.cols[c] = one.cols[0];
  r.borrowed &= ~(1u << c);
}

void sort_by_first(Ctx& ctx, Rel& r) {
  const uint64_t n = r.nrows;
  if (n <= 1 || r.ncols == 0) return;
  if (n > 0xFFFFFFFFull) fail(VG_ERR_OVERFLOW, "relation sorts are limited to 2^32 rows");
  own_column(ctx, r, 0);   // the sort uses column 0 as its key buffer
  if (r.ncols == 2) own_column(ctx, r, 1);
  std::optional<Scratch<uint32_t>> keys_alt(std::in_place, ctx, n);
  if (r.ncols == 1) {
    if (radix_sort_u32(ctx, r.cols[0], keys_alt->get(), nullptr, nullptr, n, 32, false)) std::swap(r.cols[0], keys_alt->p);
    return;
  }
  std::optional<Scratch<uint32_t>> vals_alt(std::in_place, ctx, n);
  if (r.ncols == 2) {
    // a second column travels with the keys as their values: no row numbers,
    // no gather
    if (radix_sort_u32(ctx, r.cols[0], keys_alt->get(), r.cols[1], vals_alt->get(), n, 32, false)) {
      std::swap(r.cols[0], keys_alt->p);
      std::swap(r.cols[1], vals_alt->p);
    }
    return;
  }
  Scratch<uint32_t> vals(ctx, n);
  const bool alt = radix_sort_u32(ctx, r.cols[0], keys_alt->get(), vals.get(), vals_alt->get(), n, 32, true);
  if (alt) {
    std::swap(r.cols[0], keys_alt->p);
    std::swap(vals.p, vals_alt->p);
  }
  keys_alt.reset();   // room for the new columns
  vals_alt.reset();
  permute_columns(ctx, r, 1, vals.get());
}

// Rows of at most 64 bits (each column as wide as its largest value): a sort
// of packed keys, which hold the whole rows.  Where the row count lets fewer
// bits tell most rows apart (its own bits and 4 more), only that many top bits
// are sorted by and the groups of rows that agree in them, a few each, are
// ranked while the columns are unpacked; if some group has more than kRowGroup
// rows, the keys are sorted by all bits after all.  5M rows of three 19-bit
// columns: 4 passes over 8-byte keys instead of 9 over keys and row numbers
// and six gathers.  Waits for the result and raises device errors.
static bool sort_packed_rows(Ctx& ctx, Rel& r) {
  const uint64_t n = r.nrows;
  PackCols a{};
  a.ncols = r.ncols;
  for (uint32_t c = 0; c < r.ncols; ++c) a.col[c] = r.cols[c];
  Scratch<uint32_t> mx(ctx, VG_MAX_COLS);
  VG_CUDA(cudaMemsetAsync(mx.get(), 0, VG_MAX_COLS * sizeof(uint32_t), ctx.stream));
  ctx.launch("column_max", 4.0 * n * r.ncols,
             [&] { column_maxima_kernel<<<grid_for(ctx, n, 8, 8), kBlock, 0, ctx.stream>>>(a, n, mx.get()); });
  VG_CUDA(cudaGetLastError());
  VG_CUDA(cudaMemcpyAsync(ctx.h_small, mx.get(), VG_MAX_COLS * sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx.stream));
  ctx.sync();
  const uint32_t* hm = reinterpret_cast<const uint32_t*>(ctx.h_small);
  uint32_t total = 0;
  for (int c = static_cast<int>(r.ncols) - 1; c >= 0; --c) {
    const uint32_t bits = hm[c] ? 32 - static_cast<uint32_t>(__builtin_clz(hm[c])) : 0;
    a.shift[c] = bits ? total : 0;
    a.mask[c] = (1ull << bits) - 1;
    total += bits;
  }
  if (total > 64) return false;
  if (total == 0) {   // equal rows throughout
    ctx.check_device_errors();
    return true;
  }
  // the top bits fill whole passes of seven bits
  const uint32_t want = (64 - static_cast<uint32_t>(__builtin_clzll(n)) + 4 + 6) / 7 * 7;
  const uint32_t low = want + 7 <= total ? total - want : 0;   // at least one pass saved
  std::vector<RadixDigit> digits;
  radix_plan(digits, static_cast<int>(low), static_cast<int>(total));
  DigitList dl{};
  dl.n = static_cast<uint32_t>(digits.size());
  for (uint32_t d = 0; d < dl.n; ++d) dl.d[d] = digits[d];
  const RadixCounts counts(ctx, dl);
  Scratch<uint64_t> keys(ctx, n), alt(ctx, n);
  ctx.launch("sort_pack", (8.0 + 4.0 * r.ncols) * n, [&] {
    pack_rows_kernel<<<grid_for(ctx, n, 8, 8), kBlock, dl.n * kRadixValues * sizeof(uint32_t), ctx.stream>>>(
        a, n, keys.get(), dl, counts.hist(), counts.bases(), counts.done());
  });
  VG_CUDA(cudaGetLastError());
  std::vector<const uint64_t*> bases;
  for (uint32_t d = 0; d < dl.n; ++d) bases.push_back(counts.bases(d));
  if (radix_sort_u64_counted(ctx, keys.get(), alt.get(), nullptr, nullptr, n, digits, bases)) std::swap(keys.p, alt.p);
  std::vector<Scratch<uint32_t>> own;   // for the columns that are views, which are not written
  for (uint32_t c = 0; c < r.ncols; ++c)
    if (r.borrowed >> c & 1u) own.emplace_back(ctx, n);
  Scratch<RowsDone> st(ctx, 1);
  for (uint32_t c = 0, k = 0; c < r.ncols; ++c) {
    if (r.borrowed >> c & 1u) r.cols[c] = std::exchange(own[k++].p, nullptr);
    a.col[c] = r.cols[c];
  }
  r.borrowed = 0;
  const double bytes = (8.0 + 4.0 * r.ncols) * n;
  if (low) {
    VG_CUDA(cudaMemsetAsync(st.get(), 0, sizeof(RowsDone), ctx.stream));
    auto* host = reinterpret_cast<RowsHost*>(ctx.h_small);
    ctx.launch("sort_unpack", bytes, [&] {
      unpack_groups_kernel<<<static_cast<unsigned>(div_up(n, kTileRows)), kBlock, 0, ctx.stream>>>(
          a, n, keys.get(), ~0ull << low, st.get(), ctx.d_err, host);
    });
    VG_CUDA(cudaGetLastError());
    ctx.sync();
    ctx.raise_device_errors(host->err);
    if (!host->big) return true;
    if (radix_sort_u64(ctx, keys.get(), alt.get(), n, static_cast<int>(total)))
      std::swap(keys.p, alt.p);
  }
  ctx.launch("sort_unpack", bytes,
             [&] { unpack_rows_kernel<<<grid_for(ctx, n, 8), kBlock, 0, ctx.stream>>>(a, n, keys.get()); });
  VG_CUDA(cudaGetLastError());
  ctx.check_device_errors();
  return true;
}

void sort_rows(Ctx& ctx, Rel& r) {
  const uint64_t n = r.nrows;
  if (n <= 1 || r.ncols <= 1) return;  // one column: a no-op in the reference
  if (n > 0xFFFFFFFFull) fail(VG_ERR_OVERFLOW, "relation sorts are limited to 2^32 rows");
  if (sort_packed_rows(ctx, r)) return;
  Scratch<uint32_t> perm(ctx, n), perm_alt(ctx, n), keys(ctx, n), keys_alt(ctx, n);
  fill_iota(ctx, perm.get(), n);
  // LSD over columns: stable sorts from the last column to the first.
  for (int c = static_cast<int>(r.ncols) - 1; c >= 0; --c) {
    const uint32_t* in[1] = {r.cols[c]};
    uint32_t* out[1] = {keys.get()};
    gather_cols(ctx, in, out, 1, perm.get(), n);
    if (radix_sort_u32(ctx, keys.get(), keys_alt.get(), perm.get(), perm_alt.get(), n, 32, false))
      std::swap(perm.p, perm_alt.p);
  }
  permute_columns(ctx, r, 0, perm.get());
  ctx.check_device_errors();
}

void unique_in_place(Ctx& ctx, Rel& r, bool repeats) {
  if (r.nrows <= 1 || r.ncols == 0) {
    ctx.check_device_errors();
    return;
  }
  const uint64_t n = r.nrows;
  UniqueArgs a{};
  for (uint32_t c = 0; c < r.ncols; ++c) a.in[c] = r.cols[c];
  a.ncols = r.ncols;
  a.n = n;
  auto* host = reinterpret_cast<UniqueHost*>(ctx.h_small);
  Rooms rooms{};
  if (n <= kTileRows) {
    if (take_rooms(ctx, r.ncols, {n, (n + 1) / 2, (n + 3) / 4}, rooms)) {
      ctx.launch("unique_flags", 4.0 * n,
                 [&] { unique_tile_kernel<<<1, kBlock, 0, ctx.stream>>>(a, rooms, ctx.d_err, host); });
      VG_CUDA(cudaGetLastError());
      ctx.sync();
      const uint64_t dropped = host->dropped;
      if (host->err.timeout || host->err.overflow || dropped == 0) {
        free_rooms(ctx, r.ncols, rooms);
        ctx.raise_device_errors(host->err);
        return;
      }
      Rel out;
      const bool copied = keep_room(ctx, r.ncols, rooms, n - dropped, out);
      rel_free(ctx, r);
      r = out;
      if (copied) ctx.sync();
      return;
    }
    free_rooms(ctx, r.ncols, rooms);
  }
  const uint64_t tiles = div_up(n, kTileRows);
  if (tiles > 0x7FFFFFFFull) fail(VG_ERR_OVERFLOW, "unique: too many tiles");
  Scratch<uint32_t> keep(ctx, tiles * (kTileRows / 32));
  const size_t zeroed = sizeof(UniqueTotal) + tiles * sizeof(uint32_t);
  Scratch<char> z(ctx, zeroed);
  Scratch<uint64_t> first(ctx, tiles);
  const bool soon = repeats && n <= kSoonRows && take_rooms(ctx, r.ncols, {n, (n + 1) / 2, (n + 3) / 4}, rooms);
  if (!soon) {
    free_rooms(ctx, r.ncols, rooms);
    rooms = Rooms{};
  }
  a.keep = keep.get();
  auto* tot = reinterpret_cast<UniqueTotal*>(z.get());
  VG_CUDA(cudaMemsetAsync(tot, 0, zeroed, ctx.stream));
  const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(tiles, static_cast<uint64_t>(ctx.num_sms) * 6));
  auto move = [&](double bytes) {
    ctx.launch("unique_compact", bytes, [&] {
      unique_move_kernel<<<static_cast<unsigned>(tiles), kBlock, 0, ctx.stream>>>(a, tot, first.get(), rooms);
    });
    VG_CUDA(cudaGetLastError());
  };
  // (what must be read: a column at least)
  ctx.launch("unique_flags", 4.0 * n, [&] {
    unique_flags_kernel<<<grid, kBlock, 0, ctx.stream>>>(a, tot, reinterpret_cast<uint32_t*>(tot + 1), first.get(),
                                                         static_cast<uint32_t>(tiles), ctx.d_err, host);
  });
  VG_CUDA(cudaGetLastError());
  if (soon) move(0.0);
  ctx.sync();
  const uint64_t dropped = host->dropped, kept = n - dropped;
  if (host->err.timeout || host->err.overflow || dropped == 0) {
    free_rooms(ctx, r.ncols, rooms);
    ctx.raise_device_errors(host->err);
    return;
  }
  const double bytes = 4.0 * (n + kept) * r.ncols;
  Rel out;
  bool busy = true;
  if (soon) {
    ctx.add_bytes("unique_compact", bytes);
    busy = keep_room(ctx, r.ncols, rooms, kept, out);
  } else {
    out = rel_alloc(ctx, r.ncols, kept);
    rooms.n = 1;
    rooms.rows[0] = kept;
    std::copy(out.cols, out.cols + r.ncols, rooms.cols[0]);
    move(bytes);
  }
  rel_free(ctx, r);
  r = out;
  if (busy) ctx.sync();
}

void download(Ctx& ctx, const uint32_t* dev, uint64_t n, uint32_t* host) {
  if (n) VG_CUDA(cudaMemcpyAsync(host, dev, n * sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx.stream));
  ctx.sync();
}

}  // namespace vg
