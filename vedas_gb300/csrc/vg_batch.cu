// Batched relation kernels.  Work from many queries is laid out as segments;
// a kernel maps its tile or chunk to its segments through a table made on the
// host (the tile's first segment), and a row to its segment by a search
// between the tile's first and last segments only.
#include "vg_batch.h"

#include <algorithm>
#include <cstring>
#include <functional>
#include <optional>

#include "vg_join_tile.cuh"
#include "vg_pool.h"
#include "vg_prims.cuh"
#include "vg_radix.cuh"
#include "vg_sort.h"

namespace vg {
namespace {

constexpr int kBlock = 256;
constexpr int kRows = 8;
constexpr int kTileRows = kBlock * kRows;

// The tables of one call (and words that start at zero) sent to the device in
// one copy: a copy of its own for each of the half dozen tables of a call, and
// a memset for each counter, cost the engines' threads more than the kernels
// took (a stage of a 64-query batch spent 110 to 490 us on about 30 runtime
// calls).  The device block is released, in stream order, with the object.
class Tables {
 public:
  explicit Tables(Ctx& ctx) : ctx_(ctx) {}
  Tables(const Tables&) = delete;
  Tables& operator=(const Tables&) = delete;
  ~Tables() {
    ctx_.free(dev_);
    for (char* z : zero_) ctx_.free(z);
  }
  template <typename T>
  size_t add(const std::vector<T>& v) {
    const size_t at = room(v.size() * sizeof(T));
    if (!v.empty()) std::memcpy(blob_.data() + at, v.data(), v.size() * sizeof(T));
    return at;
  }
  // Zeroed words; many of them (kInline bytes and more) get a block and a
  // memset of their own.
  template <typename T>
  size_t zeros(size_t count) {
    const size_t bytes = count * sizeof(T);
    if (bytes < kInline) return room(bytes);
    char* z = ctx_.alloc<char>(bytes);
    zero_.push_back(z);
    VG_CUDA(cudaMemsetAsync(z, 0, bytes, ctx_.stream));
    return SIZE_MAX - (zero_.size() - 1);
  }
  void send() {
    if (blob_.empty()) return;
    dev_ = ctx_.alloc<char>(blob_.size());
    ctx_.upload_bytes(dev_, blob_.data(), blob_.size());
  }
  template <typename T>
  T* at(size_t off) const {
    return reinterpret_cast<T*>(off > blob_.size() ? zero_[SIZE_MAX - off] : dev_ + off);
  }

 private:
  static constexpr size_t kInline = 32 << 10;
  size_t room(size_t bytes) {
    const size_t at = (blob_.size() + 15) / 16 * 16;
    blob_.resize(at + (bytes ? bytes : 1), 0);
    return at;
  }
  Ctx& ctx_;
  std::vector<char> blob_;
  char* dev_ = nullptr;
  std::vector<char*> zero_;
};

unsigned grid_cap(const Ctx& ctx, uint64_t units, int per_thread) {
  uint64_t g = div_up(units, static_cast<uint64_t>(kBlock) * per_thread);
  const uint64_t gmax = static_cast<uint64_t>(ctx.num_sms) * 16;
  if (g > gmax) g = gmax;
  return static_cast<unsigned>(g < 1 ? 1 : g);
}

// ---------------------------------------------------------------------------
constexpr int kCopyPer = 4;                                   // 16-byte chunks per thread per tile
constexpr uint64_t kCopyTile = static_cast<uint64_t>(kBlock) * kCopyPer;

// Copies every piece; destination chunks are 16-byte aligned (head and tail
// elements are copied by the piece's first chunk).  Blocks take tiles of
// kCopyTile consecutive chunks; a tile's first piece comes from a table made
// on the host and the next tile's bounds its last, so a thread's piece lookup
// is a search over those few pieces only (no global search, no barrier).
__global__ void __launch_bounds__(kBlock) bcopy_kernel(const CopyPiece* __restrict__ p,
                                                       const uint64_t* __restrict__ cstart, uint32_t P,
                                                       const uint32_t* __restrict__ tile_piece, uint64_t ntiles) {
  const uint64_t total = cstart[P];
  for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const uint64_t q0 = t * kCopyTile;
    const uint64_t q1 = (q0 + kCopyTile < total) ? q0 + kCopyTile : total;
    const uint32_t k0 = tile_piece[t], k1 = t + 1 < ntiles ? tile_piece[t + 1] : P - 1;
#pragma unroll
    for (int i = 0; i < kCopyPer; ++i) {
      const uint64_t q = q0 + static_cast<uint64_t>(i) * kBlock + threadIdx.x;
      if (q >= q1) break;
      uint32_t k = k0;
      if (k1 > k0) {
        uint32_t lo = k0, hi = k1;   // last k in [k0, k1] with cstart[k] <= q
        while (lo < hi) {
          const uint32_t mid = (lo + hi + 1) >> 1;
          if (cstart[mid] <= q) lo = mid;
          else hi = mid - 1;
        }
        k = lo;
      }
      const CopyPiece pc = p[k];
      const uint64_t c = q - cstart[k];
      const uint64_t head = (4 - ((reinterpret_cast<uintptr_t>(pc.dst) >> 2) & 3)) & 3;
      const uint64_t h = head < pc.len ? head : pc.len;
      if (c == 0) {
        for (uint64_t e = 0; e < h; ++e) pc.dst[e] = pc.src[e];
        const uint64_t body = (pc.len - h) / 4 * 4;
        for (uint64_t e = h + body; e < pc.len; ++e) pc.dst[e] = pc.src[e];
      }
      const uint64_t e0 = h + c * 4;
      if (e0 + 4 > pc.len) continue;
      const uint32_t* s = pc.src + e0;
      uint4 v;
      // vectors [s - sh, s - sh + 8) stay inside the piece for every chunk
      // but the first and the last
      if (c > 0 && e0 + 8 <= pc.len) {
        v = load4_realigned(s);
      } else {
        v.x = s[0];
        v.y = s[1];
        v.z = s[2];
        v.w = s[3];
      }
      *reinterpret_cast<uint4*>(pc.dst + e0) = v;
    }
  }
}

// ---------------------------------------------------------------------------
// Adjacent-unique compaction of every segment.  Segments of at most
// kSmallSeg rows (most final results) take one warp each in the first
// small_blocks blocks: each lane flags its kRows consecutive rows, a warp
// scan places the kept ones.  Larger segments take tiles of kTileRows rows
// in ticket order (the tile's segment from a per-tile table), with a block
// scan and a segmented look-back over the segment's earlier tiles.
constexpr uint32_t kSmallSeg = 32 * kRows;

// Bits of the rows r0 .. r0 + 7 that stay.  Columns are compared from the last
// to the first (the last change fastest in join outputs), only while some row
// still equals the one before it.
__device__ __forceinline__ uint32_t kept_rows(const SegRows& g, uint64_t r0) {
  if (r0 >= g.n) return 0;
  const uint32_t all = g.n - r0 < kRows ? (1u << (g.n - r0)) - 1u : (1u << kRows) - 1u;
  uint32_t diff = r0 == 0 ? 1u : 0u;
  for (int c = static_cast<int>(g.ncols) - 1; c >= 0 && (diff & all) != all; --c)
    diff |= unique_diff_bits(g.in[c], g.n, r0);
  return diff & all;
}

__device__ __forceinline__ void unique_small_segment(const SegRows& g, uint64_t* count) {
  const uint32_t lane = lane_id();
  const uint64_t n = g.n, r0 = static_cast<uint64_t>(lane) * kRows;
  const uint32_t diff = kept_rows(g, r0);
  const uint32_t cnt = __popc(diff);
  const uint32_t incl = warp_incl_scan(cnt);
  uint64_t o = incl - cnt;
  for (int i = 0; i < kRows; ++i) {
    if (!(diff >> i & 1u)) continue;
    copy_row(g.out, g.in, g.ncols, r0 + i, o);
    ++o;
  }
  if (lane == 31) *count = incl;
}

__global__ void __launch_bounds__(kBlock) bunique_kernel(const SegRows* __restrict__ segs,
                                                         const uint64_t* __restrict__ tstart,
                                                         const uint32_t* __restrict__ tile_seg,
                                                         const uint32_t* __restrict__ small, uint32_t nsmall,
                                                         uint32_t small_blocks, uint64_t* status, uint32_t* ticket,
                                                         uint64_t* counts, DeviceErrors* err) {
  if (blockIdx.x < small_blocks) {   // block-uniform: this block only compacts small segments
    const uint64_t w = static_cast<uint64_t>(blockIdx.x) * (kBlock / 32) + (threadIdx.x >> 5);
    if (w < nsmall) unique_small_segment(segs[small[w]], &counts[small[w]]);
    return;
  }
  __shared__ uint32_t s_scan[kBlock / 32 + 1];
  __shared__ uint64_t s_b;
  __shared__ uint32_t s_tile;
  __shared__ SegRows s_seg;
  __shared__ uint32_t s_s;
  __shared__ uint32_t s_keep[2 * kTileRows];   // compact_store: two columns at a time
  if (threadIdx.x == 0) {
    s_tile = atomicAdd(ticket, 1u);
    s_s = tile_seg[s_tile];
    s_seg = segs[s_s];
  }
  __syncthreads();
  const uint64_t tile = s_tile;
  const uint32_t s = s_s;
  const uint64_t n = s_seg.n;
  const uint32_t ncols = s_seg.ncols;
  const uint64_t r0 = (tile - tstart[s]) * kTileRows + threadIdx.x * kRows;
  const uint32_t diff = kept_rows(s_seg, r0);
  uint32_t tot;
  const uint32_t e = block_excl_scan<kBlock>(__popc(diff), tot, s_scan);
  if (threadIdx.x < 32) {
    const uint64_t p = warp_lookback_seg(status, tile, tstart[s], tot, err);
    if (threadIdx.x == 0) s_b = p;
  }
  __syncthreads();
  const uint64_t g = s_b;
  if (tile == tstart[s + 1] - 1 && threadIdx.x == 0) counts[s] = g + tot;
  compact_store<kBlock>(s_seg.in, s_seg.out, ncols, n, r0, diff, e, tot, g, s_keep);
}

// ---------------------------------------------------------------------------
// Rows [r0, r0 + kBlock) of a grid-stride loop over segmented rows: the
// block finds the segments of its first and last row once (two searches of
// the segment starts), then each row searches only between those, which is
// usually one or two segments.
__device__ __forceinline__ uint32_t seg_of_row(const uint64_t* __restrict__ rstart, uint32_t k0, uint32_t k1,
                                               uint64_t r) {
  uint32_t lo = k0, hi = k1;   // last k in [k0, k1] with rstart[k] <= r
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (rstart[mid] <= r) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Segmented row loops: blocks take chunks of kChunkRows consecutive rows
// (each thread kRows of them, kBlock apart, so loads and stores coalesce);
// a chunk's first segment comes from a table made on the host and the next
// chunk's bounds its last, so each row searches only between those two
// (usually one segment).
constexpr uint32_t kChunkRows = kBlock * kRows;

__device__ __forceinline__ void chunk_segments(const uint32_t* __restrict__ chunk_seg, uint64_t nchunks,
                                               uint32_t S, uint64_t c, uint32_t& k0, uint32_t& k1) {
  k0 = chunk_seg[c];
  k1 = c + 1 < nchunks ? chunk_seg[c + 1] : S - 1;
}

// (segment, key) composite sort keys: the segment sits above the key's
// key_bits bits, so one sort orders rows by segment and, within it, by key;
// and the digit counts of that sort.
__global__ void __launch_bounds__(kBlock) composite_keys_kernel(
    const uint32_t* const* __restrict__ col0, const uint64_t* __restrict__ rstart, uint32_t S,
    const uint32_t* __restrict__ chunk_seg, uint64_t nchunks, uint32_t key_bits, uint64_t* __restrict__ keys,
    DigitList dl, unsigned long long* __restrict__ hist, uint64_t* __restrict__ bases, uint32_t* done) {
  extern __shared__ uint32_t sh[];   // [dl.n][kRadixValues]
  digit_counts_init<kBlock>(dl, sh);
  const uint64_t total = rstart[S];
  for (uint64_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
    uint32_t k0, k1;
    chunk_segments(chunk_seg, nchunks, S, c, k0, k1);
#pragma unroll
    for (int it = 0; it < kRows; ++it) {
      const uint64_t r = c * kChunkRows + static_cast<uint64_t>(it) * kBlock + threadIdx.x;
      if (r < total) {
        const uint32_t s = seg_of_row(rstart, k0, k1, r);
        const uint64_t k = (static_cast<uint64_t>(s) << key_bits) | __ldg(col0[s] + (r - rstart[s]));
        keys[r] = k;
        digit_counts_add(dl, sh, k);
      }
    }
  }
  digit_counts_finish<kBlock>(dl, sh, hist, bases, done);
}

// Stable sorts of small relations by column 0, each in one step: a row's place
// is the number of rows that go before it.  Up to 32 rows take one warp (the
// first warp_blocks blocks), up to kSortSmall one block.  Most re-sorts of a
// wave have a few rows, and a composite sort of all of them took some 20
// runtime calls and ten kernels.
constexpr uint32_t kSortWarp = 32, kSortSmall = 1024;

__global__ void __launch_bounds__(kBlock) sort_small_kernel(const SegRows* __restrict__ segs,
                                                            const uint32_t* __restrict__ by_warp, uint32_t nwarp,
                                                            const uint32_t* __restrict__ by_block,
                                                            uint32_t warp_blocks) {
  if (blockIdx.x < warp_blocks) {
    const uint32_t w = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5), lane = lane_id();
    if (w >= nwarp) return;
    const SegRows& g = segs[by_warp[w]];
    const uint32_t n = static_cast<uint32_t>(g.n);
    const uint32_t k = lane < n ? g.in[0][lane] : 0u;
    uint32_t at = 0;
    for (uint32_t j = 0; j < n; ++j) {
      const uint32_t x = __shfl_sync(0xffffffffu, k, j);
      at += (x < k || (x == k && j < lane)) ? 1u : 0u;
    }
    if (lane < n)
      for (uint32_t c = 0; c < g.ncols; ++c) g.out[c][at] = g.in[c][lane];
    return;
  }
  constexpr int kEach = kSortSmall / kBlock;
  __shared__ __align__(16) uint32_t s_key[kSortSmall];
  const SegRows& g = segs[by_block[blockIdx.x - warp_blocks]];
  const uint32_t n = static_cast<uint32_t>(g.n), tid = threadIdx.x;
  const uint32_t* col0 = g.in[0];
  uint32_t k[kEach], at[kEach];
#pragma unroll
  for (int q = 0; q < kEach; ++q) {
    const uint32_t r = q * kBlock + tid;
    k[q] = r < n ? col0[r] : 0u;
    s_key[r] = k[q];
    at[q] = 0;
  }
  __syncthreads();
  for (uint32_t j = 0; j < n; ++j) {
    const uint32_t x = s_key[j];
#pragma unroll
    for (int q = 0; q < kEach; ++q) at[q] += (x < k[q] || (x == k[q] && j < q * kBlock + tid)) ? 1u : 0u;
  }
  for (uint32_t c = 0; c < g.ncols; ++c) {
    const uint32_t* in = g.in[c];
    uint32_t* out = g.out[c];
#pragma unroll
    for (int q = 0; q < kEach; ++q)
      if (q * kBlock + tid < n) out[at[q]] = in[q * kBlock + tid];
  }
}

__global__ void __launch_bounds__(kBlock) seg_gather_kernel(const SegRows* __restrict__ segs,
                                                            const uint64_t* __restrict__ rstart, uint32_t S,
                                                            const uint32_t* __restrict__ chunk_seg,
                                                            uint64_t nchunks, const uint32_t* __restrict__ perm) {
  const uint64_t total = rstart[S];
  for (uint64_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
    uint32_t k0, k1;
    chunk_segments(chunk_seg, nchunks, S, c, k0, k1);
#pragma unroll 2
    for (int it = 0; it < kRows; ++it) {
      const uint64_t r = c * kChunkRows + static_cast<uint64_t>(it) * kBlock + threadIdx.x;
      if (r < total) {
        const uint32_t s = seg_of_row(rstart, k0, k1, r);
        const uint64_t base = rstart[s];
        const SegRows& g = segs[s];
        copy_row(g.out, g.in, g.ncols, perm[r] - base, r - base);
      }
    }
  }
}

// ---------------------------------------------------------------------------
struct JoinSeg {
  const uint32_t* lk;
  const uint32_t* rk;
  uint64_t nl, nr;
  uint64_t row0;   // offset of this join's left rows in the count's arrays (whole groups)
};

// A join's part of the wave's count arrays.
__host__ __device__ __forceinline__ JoinCounts<uint32_t> join_counts(const JoinCounts<uint32_t>& all, uint64_t row0,
                                                                     uint64_t tile0) {
  return {all.lo + row0, all.offs + row0, all.start + row0 / kJcKeys, all.match + row0 / kJcKeys, all.base + tile0};
}

// One block per tile of kJcTile left keys of one join (the tile's join from a
// per-tile table, one load instead of a search of the join starts).  The
// right-key window, found beforehand by jc_window_kernel where there are more
// tiles than run at a time, is staged by a bulk copy when it fits; the tile's
// match counts stay in registers, their block scan gives every left key its
// output offset from the tile's first row, and the join's last tile to arrive
// scans its tiles' totals (jc_finish_tile).
//
// Joins with at most kSmallJoin left rows (most joins of a wave have a few)
// take one warp each instead: the first small_blocks blocks hold
// kJcBlock / 32 such joins, one per warp.  The warp finds the join's window
// of right keys with two 32-ary searches, each lane counts the matches of
// its kJcKeys keys with lockstep searches in that window, and a warp scan
// gives the offsets and the total (no shared memory).
constexpr uint32_t kSmallJoin = 32 * kJcKeys;

__device__ __forceinline__ void count_small_join(const JoinSeg& g, const JoinCounts<uint32_t>& c, uint64_t* total) {
  const uint32_t lane = lane_id();
  const uint64_t nl = g.nl;
  const uint64_t w0 = warp_bound<false, uint32_t>(g.rk, 0, g.nr, g.lk[0]);
  const uint64_t w1 = warp_bound<true, uint32_t>(g.rk, w0, g.nr, g.lk[nl - 1]);
  const uint64_t first = static_cast<uint64_t>(lane) * kJcKeys;
  uint32_t key[kJcKeys];
  uint32_t lb[kJcKeys], ub[kJcKeys];
#pragma unroll
  for (int q = 0; q < kJcKeys; ++q) key[q] = g.lk[first + q < nl ? first + q : nl - 1];
  lockstep_bounds32<kJcKeys>(g.rk, static_cast<uint32_t>(w0), static_cast<uint32_t>(w1), key, lb, ub);
  uint64_t sum = 0;
#pragma unroll
  for (int q = 0; q < kJcKeys; ++q)
    if (first + q < nl) sum += ub[q] - lb[q];
  const uint64_t incl = warp_incl_scan64(sum);
  if (first < nl) {
    uint32_t run = static_cast<uint32_t>(incl - sum), match = 0;
    c.start[lane] = run;
#pragma unroll
    for (int q = 0; q < kJcKeys; ++q)
      if (first + q < nl) {
        c.lo[first + q] = lb[q];
        c.offs[first + q] = run;
        run += ub[q] - lb[q];
        match |= (ub[q] != lb[q] ? 1u : 0u) << q;
      }
    c.match[lane] = static_cast<uint8_t>(match);
  }
  if (lane == 31) {
    *c.base = 0;
    *total = incl;
  }
}

// Every tile's right-key window [win.x, win.y) (one warp per tile, both ends
// at once), so that the counting blocks start their bulk copies at once
// instead of each searching the right keys first.
__global__ void __launch_bounds__(kJcBlock) jc_window_kernel(const JoinSeg* __restrict__ js,
                                                             const uint64_t* __restrict__ bstart,
                                                             const uint32_t* __restrict__ tile_join, uint64_t T,
                                                             uint2* __restrict__ win) {
  const uint64_t nw = static_cast<uint64_t>(gridDim.x) * (kJcBlock / 32);
  for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * (kJcBlock / 32) + (threadIdx.x >> 5); t < T; t += nw) {
    const uint32_t j = tile_join[t];
    const uint64_t nl = js[j].nl;
    const uint32_t* lk = js[j].lk;
    const uint64_t i0 = (t - bstart[j]) * static_cast<uint64_t>(kJcTile);
    const uint64_t i1 = (i0 + kJcTile < nl ? i0 + kJcTile : nl) - 1;
    uint64_t w0, w1;
    warp_window(js[j].rk, js[j].nr, lk[i0], lk[i1], w0, w1);
    if ((threadIdx.x & 31) == 0) win[t] = make_uint2(static_cast<uint32_t>(w0), static_cast<uint32_t>(w1));
  }
}

__global__ void __launch_bounds__(kJcBlock, 4) bjoin_count_kernel(
    const JoinSeg* __restrict__ js, const uint64_t* __restrict__ bstart, const uint32_t* __restrict__ tile_join,
    const uint2* __restrict__ win, const uint32_t* __restrict__ small, uint32_t nsmall, uint32_t small_blocks,
    JoinCounts<uint32_t> all, uint32_t* done, uint64_t* __restrict__ totals, DeviceErrors* err) {
  if (blockIdx.x < small_blocks) {   // block-uniform: this block only counts small joins
    const uint64_t sj = static_cast<uint64_t>(blockIdx.x) * (kJcBlock / 32) + (threadIdx.x >> 5);
    if (sj < nsmall) {
      const uint32_t j = small[sj];
      count_small_join(js[j], join_counts(all, js[j].row0, gridDim.x - small_blocks + sj), &totals[j]);
    }
    return;
  }
  __shared__ JoinCountSmem sm;
  __shared__ uint64_t s_scan[kJcBlock / 32 + 1];
  const uint32_t tile = blockIdx.x - small_blocks, j = tile_join[tile];
  const JoinSeg g = js[j];
  const uint32_t tile0 = static_cast<uint32_t>(bstart[j]), tiles = static_cast<uint32_t>(bstart[j + 1]) - tile0;
  const uint64_t i0 = static_cast<uint64_t>(tile - tile0) * kJcTile, i1 = i0 + kJcTile < g.nl ? i0 + kJcTile : g.nl;
  uint32_t key[kJcKeys];
  jc_load_keys(g.lk, i0 + static_cast<uint64_t>(threadIdx.x) * kJcKeys, i1, key);
  if (threadIdx.x < 32) {
    uint64_t w0, w1;
    if (win) {
      const uint2 w = win[tile];
      w0 = w.x;
      w1 = w.y;
    } else {   // few tiles: found here
      warp_window(g.rk, g.nr, g.lk[i0], g.lk[i1 - 1], w0, w1);
    }
    if (threadIdx.x == 0) jc_issue_window(g.rk, w0, w1, sm);
  }
  __syncthreads();
  uint32_t cnt[kJcKeys], lov[kJcKeys];
  jc_count_staged(key, g.nl, g.rk, i0, lov, cnt, sm, err);
  jc_finish_tile(i0, lov, cnt, sm, s_scan, tile - tile0, tiles, g.nl, join_counts(all, g.row0, tile0), &done[j],
                 &totals[j], err);
}

// Output rows [kb, kb + kTileRows) of one join per tile (the tile's join
// from a per-tile table).  Blocks loop over tiles [blockIdx.x, T) with
// stride gridDim.x; T is read from the device when ostart_end is given (a
// device-side placement wrote it there), each written by jw_write_tile.
//
// Small outputs (at most Ctx::tune.write_small_rows rows of a join with at most kSmallJoin
// left rows; most outputs of a wave) are written one join per warp first,
// before the tiles: the warp stages the join's offsets and lower bounds in
// its own slice of the shared arrays and each lane writes every 32nd row.
// Their list (small, nsmall of them; nsmall_dev when on the device) holds no
// tiles.

// What the host reads of a wave's written joins (page-locked memory): column
// 0's first and last value of join j at fl[2j], fl[2j + 1], and the whole
// column 0 of an output with 2 < rows < kSmallC0Words at stage + slot[j] *
// kSmallC0Words where slot[j] >= 0.  Each word is stored by the thread that
// wrote the row.
struct JoinEdges {
  uint32_t* fl;
  const int32_t* slot;   // nullable
  uint32_t* stage;
};

__device__ __forceinline__ uint32_t* edge_stage(const JoinEdges& ed, uint32_t j, uint64_t total) {
  if (!ed.slot || total <= 2 || total >= kSmallC0Words) return nullptr;
  const int32_t s = ed.slot[j];
  return s < 0 ? nullptr : ed.stage + static_cast<uint64_t>(s) * kSmallC0Words;
}

__device__ __forceinline__ void write_small_join(const JoinOut* __restrict__ src, JoinOut* jp, uint32_t* s_off,
                                                 uint32_t* s_lo, uint32_t j, const JoinEdges& ed) {
  const uint32_t lane = lane_id();
  // the join's description in the warp's shared slot: the row loop reads its
  // column pointers from shared memory
  {
    const uint32_t* a = reinterpret_cast<const uint32_t*>(src);
    uint32_t* b = reinterpret_cast<uint32_t*>(jp);
    for (uint32_t w = lane; w < sizeof(JoinOut) / 4; w += 32) b[w] = a[w];
    __syncwarp();
  }
  const uint64_t total = jp->total, nl = jp->nl;
  // one tile (its base is 0), a group per lane; a row without matches gets the
  // offset of the next one with
  static_assert(kSmallJoin <= 32 * kJcKeys, "a group per lane");
  const JoinCounts<uint32_t>& c = jp->cnt;
  const uint32_t first = lane * kJcKeys;
  uint32_t next = static_cast<uint32_t>(total);
  const bool own = first < nl;
  const uint32_t s = own ? c.start[lane] : static_cast<uint32_t>(total), match = own ? c.match[lane] : 0u;
  const uint32_t after = __shfl_down_sync(0xffffffffu, s, 1);
  if (lane < 31) next = after;
#pragma unroll
  for (int q = kJcKeys - 1; q >= 0; --q) {
    if (match >> q & 1u) {
      next = c.offs[first + q];
      s_lo[first + q] = c.lo[first + q];
    }
    s_off[first + q] = next;
  }
  __syncwarp();
  const uint32_t nlc = jp->nlc, nrc = jp->nrc;
  uint32_t* stage = edge_stage(ed, j, total);
  for (uint64_t k = lane; k < total; k += 32) {
    uint32_t a = 0, b = static_cast<uint32_t>(nl);   // last p with s_off[p] <= k
    while (b - a > 1) {
      const uint32_t mid = (a + b) >> 1;
      if (s_off[mid] <= k) a = mid;
      else b = mid;
    }
    const uint64_t jj = s_lo[a] + (k - s_off[a]);
    copy_join_row(jp->oc, jp->lc, nlc, jp->rc, nrc, a, jj, k);
    const uint32_t key = jp->oc[0][k];
    if (k == 0) ed.fl[2 * j] = key;
    if (k == total - 1) ed.fl[2 * j + 1] = key;
    if (stage) stage[k] = key;
  }
  __syncwarp();   // the slice is free for the warp's next join
}

// The join of an output tile: the last one whose tiles start at or before it
// (every lane of the warp calls it).
__device__ __forceinline__ uint32_t tile_join_of(const uint64_t* __restrict__ ostart, uint32_t J, uint64_t tile) {
  return static_cast<uint32_t>(warp_bound<true, uint64_t>(ostart, 0, static_cast<uint64_t>(J) + 1, tile) - 1);
}

// Every output tile's groups [x, y) of left rows and join z: x the last group
// whose output starts at or before the tile's first row, y the first one whose
// output starts after its last (one warp per tile, both searches at once), so that
// the writing blocks start staging at once.  T as for bjoin_write_kernel.
__global__ void __launch_bounds__(kBlock) jw_range_kernel(const JoinOut* __restrict__ jo,
                                                          const uint64_t* __restrict__ ostart, uint32_t J,
                                                          uint64_t T_host, const uint64_t* ostart_end,
                                                          uint4* __restrict__ ranges) {
  const uint64_t T = ostart_end ? *ostart_end : T_host;
  const uint64_t nw = static_cast<uint64_t>(gridDim.x) * (kBlock / 32);
  for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * (kBlock / 32) + (threadIdx.x >> 5); t < T; t += nw) {
    const uint32_t jn = tile_join_of(ostart, J, t);
    const uint64_t total = jo[jn].total, ng = jo[jn].ngroups();
    const uint64_t kb = (t - ostart[jn]) * static_cast<uint64_t>(kTileRows);
    const uint64_t kend = (kb + kTileRows < total) ? kb + kTileRows : total;
    uint64_t a, b;
    warp_bound_pair_of<true, true>(jo[jn].groups(), ng, static_cast<uint32_t>(kb), static_cast<uint32_t>(kend - 1), a, b);
    if ((threadIdx.x & 31) == 0)
      ranges[t] = make_uint4(static_cast<uint32_t>(a - 1), static_cast<uint32_t>(b), jn, 0u);
  }
}

// Ranges come from jw_range_kernel, or (null: few tiles are expected) warp 0
// finds each tile's join and left rows.
__global__ void __launch_bounds__(kBlock, 5) bjoin_write_kernel(const JoinOut* __restrict__ jo,
                                                             const uint64_t* __restrict__ ostart, uint32_t J,
                                                             const uint4* __restrict__ ranges,
                                                             uint64_t T_host, const uint64_t* ostart_end,
                                                             const uint32_t* __restrict__ small, uint32_t nsmall_host,
                                                             const uint32_t* nsmall_dev, JoinEdges ed) {
  static_assert(kBlock == kJwBlock, "jw_write_tile's block");
  static_assert(JwStage<kRows>::kTile >= (kBlock / 32) * kSmallJoin, "a warp's slice holds a small join's left rows");
  __shared__ JoinOut s_o;
  __shared__ JoinOut s_w[kBlock / 32];
  __shared__ JwStage<kRows> s_stage;
  __shared__ uint32_t s_j;
  __shared__ uint64_t s_range[2];
  {
    const uint32_t nsm = nsmall_dev ? *nsmall_dev : nsmall_host;
    const uint32_t warp = threadIdx.x >> 5, nwarps = kBlock / 32;
    for (uint64_t w = static_cast<uint64_t>(blockIdx.x) * nwarps + warp; w < nsm;
         w += static_cast<uint64_t>(gridDim.x) * nwarps)
      write_small_join(&jo[small[w]], &s_w[warp], s_stage.left + warp * kSmallJoin, s_stage.right + warp * kSmallJoin,
                       small[w], ed);
  }
  const uint64_t T = ostart_end ? *ostart_end : T_host;
#pragma unroll 1
  for (uint64_t tile = blockIdx.x; tile < T; tile += gridDim.x) {
    __syncthreads();   // the previous tile's readers of the shared arrays are done
    jw_clear(s_stage);
    if (threadIdx.x < 32) {
      uint32_t j;
      uint64_t a, b;
      if (ranges) {
        const uint4 rg = ranges[tile];
        j = rg.z;
        a = rg.x;
        b = rg.y;
      } else {
        j = tile_join_of(ostart, J, tile);
        const uint64_t kb = (tile - ostart[j]) * static_cast<uint64_t>(kTileRows), tot = jo[j].total;
        const uint64_t kend = kb + kTileRows < tot ? kb + kTileRows : tot;
        warp_bound_pair_of<true, true>(jo[j].groups(), jo[j].ngroups(), static_cast<uint32_t>(kb),
                                       static_cast<uint32_t>(kend - 1), a, b);
        --a;
      }
      if (threadIdx.x == 0) {
        s_j = j;
        s_range[0] = a;
        s_range[1] = b;
      }
    }
    __syncthreads();
    const uint32_t jn = s_j;
    {
      const uint32_t* src = reinterpret_cast<const uint32_t*>(&jo[jn]);
      uint32_t* dst = reinterpret_cast<uint32_t*>(&s_o);
      for (uint32_t w = threadIdx.x; w < sizeof(JoinOut) / 4; w += kBlock) dst[w] = src[w];
    }
    __syncthreads();
    const uint64_t total = s_o.total;
    const uint64_t kb = (tile - ostart[jn]) * static_cast<uint64_t>(kTileRows);
    const uint64_t kend = (kb + kTileRows < total) ? kb + kTileRows : total;
    jw_write_tile<kRows>(s_o, kb, kend, s_range[0], s_range[1], s_stage);
    const uint32_t* c0 = s_o.oc[0];
    if (kb == 0 && threadIdx.x == 0) ed.fl[2 * jn] = c0[0];
    if (kend == total && threadIdx.x == (total - 1 - kb) % kBlock) ed.fl[2 * jn + 1] = c0[total - 1];
    uint32_t* stage = edge_stage(ed, jn, total);
    if (stage && threadIdx.x < total) stage[threadIdx.x] = c0[threadIdx.x];
  }
}

// ---------------------------------------------------------------------------
// Device-side placement of a wave's join outputs in a region (no host round
// trip between the count and the write).  One block: every join's output
// size comes from its count, each column is rounded up to 256 bytes, and the
// outputs are laid out back to back after the bytes the region handed out in
// earlier waves (*bump).  A join whose output does not fit is left unplaced
// (total 0, no columns; the host writes it itself); the offsets only grow,
// so every later join with rows is unplaced too.  The same arithmetic on the
// host (place_outputs_on_host) reproduces every placement from the totals.
constexpr int kPlaceBlock = 1024;

__host__ __device__ inline uint64_t place_stride(uint64_t rows) { return (rows * 4 + 255) / 256 * 256; }

// Bytes of an output in a region of `cap` bytes.  More rows than a join may
// write (its 32-bit offsets would wrap, and the write read outside the columns;
// the host refuses the join) count as more than any region holds.
__host__ __device__ inline uint64_t place_bytes(uint64_t rows, uint32_t ncols, uint64_t cap) {
  return rows > kMaxJoinRows ? cap + 1 : rows ? ncols * place_stride(rows) : 0;
}

struct JoinPlace {
  char* base;            // the region
  uint64_t cap;          // its bytes
  uint64_t* bump;        // bytes handed out before this wave (updated)
  uint64_t* ostart;      // J + 1 output-tile starts (written; small outputs have no tiles)
  uint32_t* small;       // joins whose outputs are written one per warp (written)
  uint32_t* nsmall;      // their number (written)
  uint32_t small_rows;   // outputs of at most this many rows are small
  uint64_t* totals_host; // page-locked: every join's rows,
  uint64_t* bump_host;   // the bump after the wave
  DeviceErrors* err_host;   // and the error record after the count
  const DeviceErrors* err;
};

__global__ void __launch_bounds__(kPlaceBlock) join_place_kernel(JoinOut* __restrict__ jo,
                                                                 const uint64_t* __restrict__ totals, uint32_t J,
                                                                 JoinPlace pl) {
  __shared__ uint64_t s_scan[kPlaceBlock / 32 + 1];
  __shared__ unsigned long long s_fit;   // end of the placed outputs, after the bump
  const uint64_t bump0 = *pl.bump;
  // after a wait that gave up nothing is written, and the host raises the error
  const DeviceErrors e = *pl.err;
  if (threadIdx.x == 0) s_fit = 0;
  uint64_t carry_b = 0, carry_t = 0, carry_s = 0;
  for (uint32_t c0 = 0; c0 < J; c0 += kPlaceBlock) {
    const uint32_t j = c0 + threadIdx.x;
    const uint64_t t = j < J && !e.timeout ? totals[j] : 0;
    const uint32_t ncols = j < J ? jo[j].nlc + jo[j].nrc : 0;
    const uint64_t stride = place_stride(t);
    const uint64_t bytes = place_bytes(t, ncols, pl.cap);
    uint64_t tot_b, tot_ts;
    const uint64_t eb = block_excl_scan64<kPlaceBlock>(bytes, tot_b, s_scan);
    const uint64_t off = bump0 + carry_b + eb;
    const bool fits = off + bytes <= pl.cap;
    const bool is_small = fits && t > 0 && t <= pl.small_rows && j < J && jo[j].nl <= kSmallJoin;
    const uint64_t tiles = (fits && t && !is_small) ? div_up(t, kTileRows) : 0;
    // tiles above bit 11, small outputs (at most kPlaceBlock < 2^11) below
    static_assert(kPlaceBlock < (1 << 11), "a chunk's small outputs fit 11 bits");
    const uint64_t ets = block_excl_scan64<kPlaceBlock>((tiles << 11) | (is_small ? 1 : 0), tot_ts, s_scan);
    if (j < J) {
      JoinOut& o = jo[j];
      pl.totals_host[j] = t;
      o.total = fits ? t : 0;
      for (uint32_t c = 0; c < VG_MAX_COLS; ++c)
        o.oc[c] = (fits && t && c < ncols) ? reinterpret_cast<uint32_t*>(pl.base + off + c * stride) : nullptr;
      pl.ostart[j] = carry_t + (ets >> 11);
      if (is_small) pl.small[carry_s + (ets & 2047)] = j;
      // what fits is a prefix of the joins with rows: its end is their sum
      if (fits) atomicMax(&s_fit, static_cast<unsigned long long>(carry_b + eb + bytes));
    }
    carry_b += tot_b;
    carry_t += tot_ts >> 11;
    carry_s += tot_ts & 2047;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    pl.ostart[J] = carry_t;
    *pl.nsmall = static_cast<uint32_t>(carry_s);
    *pl.bump = bump0 + s_fit;
    *pl.bump_host = bump0 + s_fit;
    *pl.err_host = e;
  }
}

struct Col0Req {
  const uint32_t* src;
  uint64_t n;
  uint64_t dst;
};

__global__ void col0_kernel(const Col0Req* __restrict__ rq, uint32_t R, uint32_t* __restrict__ out) {
  for (uint32_t q = blockIdx.x; q < R; q += gridDim.x)
    for (uint64_t i = threadIdx.x; i < rq[q].n; i += blockDim.x) out[rq[q].dst + i] = rq[q].src[i];
}

int bits_for_segments(uint32_t S) {
  int b = 0;
  while ((1ull << b) < S) ++b;
  return b;
}

}  // namespace

struct BatchStage::Impl {
  Tables tb;
  std::vector<std::function<void()>> launches;
  explicit Impl(Ctx& ctx) : tb(ctx) {}
};

BatchStage::BatchStage(Ctx& ctx) : impl_(new Impl(ctx)) {}
BatchStage::~BatchStage() = default;

namespace {

// Adds a call's tables to the stage's and leaves the launch that `add` returns
// to BatchStage::run; without a stage, runs it.
template <typename Add>
void in_stage(Ctx& ctx, BatchStage* stage, Add add) {
  if (stage) {
    stage->impl().launches.push_back(add(stage->impl().tb));
    return;
  }
  Tables tb(ctx);
  const std::function<void()> launch = add(tb);
  tb.send();
  launch();
}

}  // namespace

void BatchStage::run() {
  impl_->tb.send();
  for (auto& f : impl_->launches) f();
  impl_->launches.clear();
}

void batched_copy(Ctx& ctx, const std::vector<CopyPiece>& pieces, BatchStage* stage) {
  std::vector<CopyPiece> p;
  std::vector<uint64_t> cstart(1, 0);
  double bytes = 0;
  for (const CopyPiece& pc : pieces) {
    if (pc.len == 0) continue;
    const uint64_t head = (4 - ((reinterpret_cast<uintptr_t>(pc.dst) >> 2) & 3)) & 3;
    const uint64_t h = head < pc.len ? head : pc.len;
    const uint64_t chunks = (pc.len - h) / 4;
    p.push_back(pc);
    cstart.push_back(cstart.back() + (chunks ? chunks : 1));
    bytes += 8.0 * pc.len;
  }
  if (p.empty()) return;
  const uint32_t P = static_cast<uint32_t>(p.size());
  // each tile's first piece
  const uint64_t ntiles = div_up(cstart.back(), kCopyTile);
  std::vector<uint32_t> tile_piece(ntiles);
  {
    uint32_t k = 0;
    for (uint64_t t = 0; t < ntiles; ++t) {
      const uint64_t q = t * kCopyTile;
      while (cstart[k + 1] <= q) ++k;
      tile_piece[t] = k;
    }
  }
  const unsigned grid = grid_cap(ctx, cstart.back(), kCopyPer);
  in_stage(ctx, stage, [&](Tables& tb) -> std::function<void()> {
    const size_t op = tb.add(p), oc = tb.add(cstart), ot = tb.add(tile_piece);
    return [=, &ctx, &tb] {
      ctx.launch("select_copy", bytes, [&] {
        bcopy_kernel<<<grid, kBlock, 0, ctx.stream>>>(tb.at<CopyPiece>(op), tb.at<uint64_t>(oc), P,
                                                      tb.at<uint32_t>(ot), ntiles);
      });
      VG_CUDA(cudaGetLastError());
    };
  });
}

void batched_unique_enqueue(Ctx& ctx, const std::vector<SegRows>& segs, uint64_t* counts_host, BatchStage* stage) {
  const uint32_t S = static_cast<uint32_t>(segs.size());
  if (S == 0) return;
  std::vector<uint64_t> tstart(S + 1, 0);
  std::vector<uint32_t> small;
  double bytes = 0;
  for (uint32_t s = 0; s < S; ++s) {
    const bool is_small = segs[s].n > 0 && segs[s].n <= std::min<uint32_t>(kSmallSeg, ctx.tune.unique_small_rows);
    if (is_small) small.push_back(s);
    tstart[s + 1] = tstart[s] + (is_small ? 0 : div_up(segs[s].n, kTileRows));
    bytes += 4.0 * segs[s].n * segs[s].ncols;
    counts_host[s] = 0;   // the kernel stores the others' counts
  }
  const uint64_t tiles = tstart[S];
  const uint32_t nsmall = static_cast<uint32_t>(small.size());
  const uint32_t small_blocks = static_cast<uint32_t>(div_up(nsmall, kBlock / 32));
  if (tiles == 0 && nsmall == 0) return;
  std::vector<uint32_t> tile_seg(tiles);
  for (uint32_t s = 0; s < S; ++s)
    for (uint64_t t = tstart[s]; t < tstart[s + 1]; ++t) tile_seg[t] = s;
  in_stage(ctx, stage, [&](Tables& tb) -> std::function<void()> {
    const size_t og = tb.add(segs), ot = tb.add(tstart), os = tb.add(tile_seg), om = tb.add(small);
    const size_t oz = tb.zeros<uint64_t>(tiles + 1);   // look-back words, then the ticket
    return [=, &ctx, &tb] {
      uint64_t* status = tb.at<uint64_t>(oz);
      ctx.launch("unique_compact", bytes, [&] {
        bunique_kernel<<<static_cast<unsigned>(small_blocks + tiles), kBlock, 0, ctx.stream>>>(
            tb.at<SegRows>(og), tb.at<uint64_t>(ot), tb.at<uint32_t>(os), tb.at<uint32_t>(om), nsmall, small_blocks,
            status, reinterpret_cast<uint32_t*>(status + tiles), counts_host, ctx.d_err);
      });
      VG_CUDA(cudaGetLastError());
    };
  });
}

void note_unique_writes(Ctx& ctx, const std::vector<SegRows>& segs, const uint64_t* counts) {
  double wb = 0;
  for (size_t s = 0; s < segs.size(); ++s) wb += 4.0 * counts[s] * segs[s].ncols;
  ctx.add_bytes("unique_compact", wb);
}

namespace {

// The relations' rows with newly allocated output columns.
std::vector<SegRows> sort_segments(Ctx& ctx, const std::vector<Rel*>& rels) {
  std::vector<SegRows> segs(rels.size());
  parallel_for(rels.size(), [&](size_t s) {
    segs[s].ncols = rels[s]->ncols;
    segs[s].n = rels[s]->nrows;
    for (uint32_t c = 0; c < rels[s]->ncols; ++c) {
      segs[s].in[c] = rels[s]->cols[c];
      segs[s].out[c] = ctx.alloc<uint32_t>(rels[s]->nrows);
    }
  });
  return segs;
}

void take_sorted(Ctx& ctx, const std::vector<Rel*>& rels, const std::vector<SegRows>& segs) {
  parallel_for(rels.size(), [&](size_t s) {
    for (uint32_t c = 0; c < rels[s]->ncols; ++c) {
      rel_drop_col(ctx, *rels[s], c);
      rels[s]->cols[c] = segs[s].out[c];
    }
  });
}

// Relations of at most kSortSmall rows: one launch.
void sort_small(Ctx& ctx, const std::vector<Rel*>& rels) {
  const uint32_t S = static_cast<uint32_t>(rels.size());
  if (S == 0) return;
  const std::vector<SegRows> segs = sort_segments(ctx, rels);
  std::vector<uint32_t> by_warp, by_block;
  double bytes = 0;
  for (uint32_t s = 0; s < S; ++s) {
    (segs[s].n <= kSortWarp ? by_warp : by_block).push_back(s);
    bytes += 8.0 * segs[s].n * segs[s].ncols;
  }
  Tables tb(ctx);
  const size_t og = tb.add(segs), ow = tb.add(by_warp), ob = tb.add(by_block);
  tb.send();
  const uint32_t warp_blocks = static_cast<uint32_t>(div_up(by_warp.size(), kBlock / 32));
  ctx.launch("sort_small", bytes, [&] {
    sort_small_kernel<<<warp_blocks + static_cast<unsigned>(by_block.size()), kBlock, 0, ctx.stream>>>(
        tb.at<SegRows>(og), tb.at<uint32_t>(ow), static_cast<uint32_t>(by_warp.size()), tb.at<uint32_t>(ob),
        warp_blocks);
  });
  VG_CUDA(cudaGetLastError());
  take_sorted(ctx, rels, segs);
}

}  // namespace

void batched_sort_by_first(Ctx& ctx, const std::vector<Rel*>& rels_in, int key_bits) {
  std::vector<Rel*> rels, small;
  for (Rel* r : rels_in)
    if (r->nrows > 1 && r->ncols > 0) (r->nrows <= kSortSmall ? small : rels).push_back(r);
  sort_small(ctx, small);
  const uint32_t S = static_cast<uint32_t>(rels.size());
  if (S == 0) return;
  std::vector<uint64_t> rstart(S + 1, 0);
  for (uint32_t s = 0; s < S; ++s) rstart[s + 1] = rstart[s] + rels[s]->nrows;
  const uint64_t N = rstart[S];
  if (N > 0xFFFFFFFFull) fail(VG_ERR_OVERFLOW, "batched sort is limited to 2^32 rows");
  const int kb = key_bits > 0 && key_bits <= 32 ? key_bits : 32;
  // each chunk's first segment
  const uint64_t nchunks = div_up(N, static_cast<uint64_t>(kChunkRows));
  std::vector<uint32_t> chunk_seg(nchunks);
  {
    uint32_t sg = 0;
    for (uint64_t c = 0; c < nchunks; ++c) {
      const uint64_t r = c * kChunkRows;
      while (rstart[sg + 1] <= r) ++sg;
      chunk_seg[c] = sg;
    }
  }
  const unsigned cgrid = static_cast<unsigned>(std::min<uint64_t>(nchunks, static_cast<uint64_t>(ctx.num_sms) * 8));
  Scratch<uint32_t> vals(ctx, N), vals_alt(ctx, N);
  std::vector<RadixDigit> digits;
  radix_plan(digits, 0, kb + bits_for_segments(S));
  DigitList dl{};
  dl.n = static_cast<uint32_t>(digits.size());
  for (uint32_t d = 0; d < dl.n; ++d) dl.d[d] = digits[d];
  std::vector<const uint32_t*> col0(S);
  for (uint32_t s = 0; s < S; ++s) col0[s] = rels[s]->cols[0];
  Tables tb(ctx);
  const size_t okey = tb.add(col0), orow = tb.add(rstart), oc = tb.add(chunk_seg);
  tb.send();
  bool alt;
  {
    Scratch<uint64_t> keys(ctx, N), keys_alt(ctx, N);
    const RadixCounts counts(ctx, dl);
    ctx.launch("sort_keys", 12.0 * N, [&] {
      composite_keys_kernel<<<cgrid, kBlock, dl.n * kRadixValues * sizeof(uint32_t), ctx.stream>>>(
          tb.at<const uint32_t*>(okey), tb.at<uint64_t>(orow), S, tb.at<uint32_t>(oc), nchunks,
          static_cast<uint32_t>(kb), keys.get(), dl, counts.hist(), counts.bases(), counts.done());
    });
    VG_CUDA(cudaGetLastError());
    // the passes are fixed by the key width and nothing waits on the device
    std::vector<const uint64_t*> bases;
    for (uint32_t d = 0; d < dl.n; ++d) bases.push_back(counts.bases(d));
    alt = radix_sort_u64_counted(ctx, keys.get(), keys_alt.get(), vals.get(), vals_alt.get(), N, digits, bases, true);
  }
  const uint32_t* perm = alt ? vals_alt.get() : vals.get();
  const std::vector<SegRows> segs = sort_segments(ctx, rels);
  double bytes = 4.0 * N;
  for (uint32_t s = 0; s < S; ++s) bytes += 8.0 * rels[s]->nrows * rels[s]->ncols;
  Tables tg(ctx);
  const size_t og = tg.add(segs);
  tg.send();
  ctx.launch("gather", bytes, [&] {
    seg_gather_kernel<<<cgrid, kBlock, 0, ctx.stream>>>(tg.at<SegRows>(og), tb.at<uint64_t>(orow), S,
                                                        tb.at<uint32_t>(oc), nchunks, perm);
  });
  VG_CUDA(cudaGetLastError());
  take_sorted(ctx, rels, segs);
}

namespace {

// Tiles of all joins of a wave above which the windows (and, by the left
// rows, the output tiles' ranges) get kernels of their own: below, the blocks
// all run at once and find their own in about the time of a launch.
uint64_t window_tiles(const Ctx& ctx) { return 2ull * static_cast<uint64_t>(ctx.num_sms); }

// The tables of a wave's join count (and what follows it in the same stage).
struct CountTables {
  size_t js, bstart, tile_join, small, done;   // done: tiles counted, per join
  uint32_t nsmall = 0, small_blocks = 0;
  uint64_t T = 0, rows = 0;
  double bytes = 0;
};

CountTables count_tables(Ctx& ctx, Tables& tb, const std::vector<const Rel*>& l, const std::vector<const Rel*>& r,
                         JoinBatch& jb) {
  CountTables ct;
  const uint32_t J = static_cast<uint32_t>(l.size());
  jb = JoinBatch();
  jb.J = J;
  jb.l = l;
  jb.r = r;
  std::vector<JoinSeg> js(J);
  std::vector<uint64_t> bstart(J + 1, 0);
  jb.row0.resize(J);
  jb.base_at.resize(J);
  std::vector<uint32_t> small;   // joins counted by one warp each
  for (uint32_t j = 0; j < J; ++j) {
    if (l[j]->nrows == 0 || r[j]->nrows == 0) fail(VG_ERR_INVALID, "batched join of an empty relation");
    if (l[j]->nrows > 0xFFFFFFFFull || r[j]->nrows > 0xFFFFFFFFull)
      fail(VG_ERR_OVERFLOW, "join inputs are limited to 2^32 rows");
    if (l[j]->ncols + r[j]->ncols - 1 > VG_MAX_COLS) fail(VG_ERR_UNSUPPORTED, "join output has more than 9 columns");
    js[j] = {l[j]->cols[0], r[j]->cols[0], l[j]->nrows, r[j]->nrows, ct.rows};
    jb.row0[j] = ct.rows;
    ct.rows += div_up(l[j]->nrows, kJcKeys) * kJcKeys;
    const bool is_small = l[j]->nrows <= std::min<uint32_t>(kSmallJoin, ctx.tune.join_small_rows);
    if (is_small) small.push_back(j);
    bstart[j + 1] = bstart[j] + (is_small ? 0 : div_up(l[j]->nrows, kJcTile));
    ct.bytes += 4.0 * (l[j]->nrows + r[j]->nrows);
  }
  ct.T = bstart[J];
  if (ct.T > 0x7FFFFFFFull) fail(VG_ERR_OVERFLOW, "batched join count: too many tiles");
  ct.nsmall = static_cast<uint32_t>(small.size());
  ct.small_blocks = static_cast<uint32_t>(div_up(ct.nsmall, kJcBlock / 32));
  for (uint32_t j = 0; j < J; ++j) jb.base_at[j] = bstart[j];
  for (uint32_t s = 0; s < ct.nsmall; ++s) jb.base_at[small[s]] = ct.T + s;   // after the tiles'
  std::vector<uint32_t> tile_join(ct.T);
  for (uint32_t j = 0; j < J; ++j)
    for (uint64_t t = bstart[j]; t < bstart[j + 1]; ++t) tile_join[t] = j;
  ct.js = tb.add(js);
  ct.bstart = tb.add(bstart);
  ct.tile_join = tb.add(tile_join);
  ct.small = tb.add(small);
  ct.done = tb.zeros<uint32_t>(J);
  return ct;
}

// Device arrays of a count: before the joins are described.
void alloc_count(Ctx& ctx, const CountTables& ct, JoinBatch& jb) {
  const uint64_t groups = ct.rows / kJcKeys;
  jb.cnt.lo = ctx.alloc<uint32_t>(ct.rows);
  jb.cnt.offs = ctx.alloc<uint32_t>(ct.rows);
  jb.cnt.start = ctx.alloc<uint32_t>(groups + div_up(groups, 4));   // and the match bits
  jb.cnt.match = reinterpret_cast<uint8_t*>(jb.cnt.start + groups);
  jb.d_totals = ctx.alloc<uint64_t>(jb.J + ct.T + ct.nsmall);
  jb.cnt.base = jb.d_totals + jb.J;
}

// Enqueues the count of the joins (tables sent): jb.cnt and jb.d_totals.
void launch_count(Ctx& ctx, const Tables& tb, const CountTables& ct, JoinBatch& jb) {
  std::optional<Scratch<uint2>> win;
  if (ct.T > window_tiles(ctx)) {
    win.emplace(ctx, ct.T);
    const uint64_t wblocks = std::min<uint64_t>(div_up(ct.T, kJcBlock / 32), static_cast<uint64_t>(ctx.num_sms) * 8);
    ctx.launch("join_windows", 8.0 * ct.T, [&] {
      jc_window_kernel<<<static_cast<unsigned>(wblocks), kJcBlock, 0, ctx.stream>>>(
          tb.at<JoinSeg>(ct.js), tb.at<uint64_t>(ct.bstart), tb.at<uint32_t>(ct.tile_join), ct.T, win->get());
    });
    VG_CUDA(cudaGetLastError());
  }
  ctx.launch("join_count", ct.bytes + 8.0 * ct.rows, [&] {
    bjoin_count_kernel<<<static_cast<unsigned>(ct.small_blocks + ct.T), kJcBlock, 0, ctx.stream>>>(
        tb.at<JoinSeg>(ct.js), tb.at<uint64_t>(ct.bstart), tb.at<uint32_t>(ct.tile_join), win ? win->get() : nullptr,
        tb.at<uint32_t>(ct.small), ct.nsmall, ct.small_blocks, jb.cnt, tb.at<uint32_t>(ct.done), jb.d_totals, ctx.d_err);
  });
  VG_CUDA(cudaGetLastError());
}

// Output descriptions without the output columns.
void describe_join(const JoinBatch& jb, size_t j, JoinOut& o) {
  const Rel* l = jb.l[j];
  const Rel* r = jb.r[j];
  std::memset(&o, 0, sizeof(o));
  o.cnt = join_counts(jb.cnt, jb.row0[j], jb.base_at[j]);
  o.nl = l->nrows;
  for (uint32_t c = 0; c < l->ncols; ++c) o.lc[c] = l->cols[c];
  for (uint32_t c = 1; c < r->ncols; ++c) o.rc[c - 1] = r->cols[c];
  o.nlc = l->ncols;
  o.nrc = r->ncols - 1;
}

}  // namespace

void batched_join_count(Ctx& ctx, const std::vector<const Rel*>& l, const std::vector<const Rel*>& r, JoinBatch& jb,
                        uint64_t* totals_host) {
  Tables tb(ctx);
  const CountTables ct = count_tables(ctx, tb, l, r, jb);
  if (jb.J == 0) return;
  tb.send();
  alloc_count(ctx, ct, jb);
  launch_count(ctx, tb, ct, jb);
  VG_CUDA(cudaMemcpyAsync(totals_host, jb.d_totals, jb.J * sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx.stream));
}

void batched_join_write(Ctx& ctx, JoinBatch& jb, const uint64_t* totals, std::vector<Rel>& out,
                        uint32_t* first_last_host, const uint8_t* skip) {
  const uint32_t J = jb.J;
  if (!skip) out.assign(J, Rel());
  if (J == 0) return;
  std::vector<JoinOut> jo(J);
  std::vector<uint64_t> ostart(J + 1, 0);
  double wbytes = 0;
  auto rows = [&](uint32_t j) -> uint64_t { return (skip && skip[j]) ? 0 : totals[j]; };
  std::vector<uint32_t> small;   // outputs written one join per warp
  for (uint32_t j = 0; j < J; ++j) {
    if (rows(j) > kMaxJoinRows) fail(VG_ERR_OVERFLOW, "join output exceeds 2^32 rows");
    const bool is_small = rows(j) > 0 && rows(j) <= ctx.tune.write_small_rows && jb.l[j]->nrows <= kSmallJoin;
    if (is_small) small.push_back(j);
    ostart[j + 1] = ostart[j] + (is_small ? 0 : div_up(rows(j), kTileRows));
    wbytes += 4.0 * rows(j) * (2.0 * (jb.l[j]->ncols + jb.r[j]->ncols - 1) - 1);
    first_last_host[2 * j] = first_last_host[2 * j + 1] = 0;   // the kernel stores the others'
  }
  const uint32_t nsmall = static_cast<uint32_t>(small.size());
  const uint64_t T = ostart[J], small_blocks = div_up(nsmall, kBlock / 32);
  // the outputs of a wave's joins are allocated and described on the host pool
  parallel_for(J, [&](size_t j) {
    std::memset(&jo[j], 0, sizeof(jo[j]));
    if (skip && skip[j]) return;                // written already: out[j] stays as it is
    const uint32_t ncols = jb.l[j]->ncols + jb.r[j]->ncols - 1;
    out[j] = rel_alloc(ctx, ncols, totals[j]);
    describe_join(jb, j, jo[j]);
    jo[j].total = totals[j];
    for (uint32_t c = 0; c < ncols; ++c) jo[j].oc[c] = out[j].cols[c];
  });
  if (T > 0 || nsmall > 0) {
    if (T > 0x7FFFFFFFull) fail(VG_ERR_OVERFLOW, "batched join write: too many tiles");
    Tables tb(ctx);
    const size_t oj = tb.add(jo), os = tb.add(ostart), om = tb.add(small);
    tb.send();
    std::optional<Scratch<uint4>> ranges;
    if (T > window_tiles(ctx)) {
      ranges.emplace(ctx, T);
      const uint64_t rblocks = std::min<uint64_t>(div_up(T, kBlock / 32), static_cast<uint64_t>(ctx.num_sms) * 8);
      ctx.launch("join_write_ranges", 8.0 * T, [&] {
        jw_range_kernel<<<static_cast<unsigned>(rblocks), kBlock, 0, ctx.stream>>>(
            tb.at<JoinOut>(oj), tb.at<uint64_t>(os), J, T, nullptr, ranges->get());
      });
      VG_CUDA(cudaGetLastError());
    }
    const unsigned grid = static_cast<unsigned>(std::max<uint64_t>(T, small_blocks));
    ctx.launch("join_write", wbytes, [&] {
      bjoin_write_kernel<<<grid, kBlock, 0, ctx.stream>>>(
          tb.at<JoinOut>(oj), tb.at<uint64_t>(os), J, ranges ? ranges->get() : nullptr, T, nullptr,
          tb.at<uint32_t>(om), nsmall, nullptr, JoinEdges{first_last_host, nullptr, nullptr});
    });
    VG_CUDA(cudaGetLastError());
  }
  jb.release(ctx);
}

uint64_t place_outputs_on_host(const JoinBatch& jb, const uint64_t* totals, const Arena::Region* region,
                               uint64_t bump, std::vector<Rel>& out, std::vector<uint8_t>& placed,
                               int64_t& blocks) {
  const uint32_t J = jb.J;
  out.assign(J, Rel());
  placed.assign(J, 0);
  blocks = 0;
  uint64_t off = bump, fit = 0;
  for (uint32_t j = 0; j < J; ++j) {
    const uint64_t t = totals[j];
    const uint32_t ncols = jb.l[j]->ncols + jb.r[j]->ncols - 1;
    const uint64_t stride = place_stride(t);
    const uint64_t bytes = place_bytes(t, ncols, region->bytes);
    const bool fits = off + bytes <= region->bytes;
    if (fits && t) {
      Rel& r = out[j];
      r.ncols = ncols;
      r.nrows = t;
      for (uint32_t c = 0; c < ncols; ++c) r.cols[c] = reinterpret_cast<uint32_t*>(region->begin + off + c * stride);
      placed[j] = 1;
      blocks += ncols;
    }
    if (fits) fit += bytes;
    off += bytes;
  }
  return bump + fit;
}

namespace {

// The count, the placement and the write (tables sent).
void launch_placed(Ctx& ctx, const Tables& tb, const CountTables& ct, JoinBatch& jb, JoinOut* djo,
                   const Arena::Region* region, uint64_t* d_bump, const int32_t* c0_slot, const PlacedHost& host) {
  const uint32_t J = jb.J;
  launch_count(ctx, tb, ct, jb);
  Scratch<uint64_t> ostart(ctx, J + 1);
  Scratch<uint32_t> small(ctx, J + 1);   // small list, then its length
  const JoinPlace pl{region->begin, region->bytes, d_bump,        ostart.get(),   small.get(), small.get() + J,
                     ctx.tune.write_small_rows,    host.totals, host.bump, host.err, ctx.d_err};
  ctx.launch("join_place", 16.0 * J, [&] {
    join_place_kernel<<<1, kPlaceBlock, 0, ctx.stream>>>(djo, jb.d_totals, J, pl);
  });
  VG_CUDA(cudaGetLastError());
  // the tile count is on the device: fixed grids loop over the tiles (the
  // algorithmic bytes are added when the host reads the totals)
  std::optional<Scratch<uint4>> ranges;
  if (ct.rows > kTileRows * window_tiles(ctx)) {
    // every placed output tile covers kTileRows rows of at least one 4-byte column
    ranges.emplace(ctx, region->bytes / (4ull * kTileRows) + J + 1);
    ctx.launch("join_write_ranges", 0.0, [&] {
      jw_range_kernel<<<static_cast<unsigned>(ctx.num_sms) * 8, kBlock, 0, ctx.stream>>>(
          djo, ostart.get(), J, 0, ostart.get() + J, ranges->get());
    });
    VG_CUDA(cudaGetLastError());
  }
  ctx.launch("join_write", 0.0, [&] {
    bjoin_write_kernel<<<static_cast<unsigned>(ctx.num_sms) * ctx.tune.write_blocks_per_sm, kBlock, 0, ctx.stream>>>(
        djo, ostart.get(), J, ranges ? ranges->get() : nullptr, 0, ostart.get() + J, small.get(), 0, small.get() + J,
        JoinEdges{host.first_last, c0_slot, host.c0});
  });
  VG_CUDA(cudaGetLastError());
}

}  // namespace

void batched_join_placed(Ctx& ctx, const std::vector<const Rel*>& l, const std::vector<const Rel*>& r, JoinBatch& jb,
                         const Arena::Region* region, uint64_t* d_bump, const std::vector<int32_t>& c0_slot,
                         uint32_t nslots, const PlacedHost& host, BatchStage* stage) {
  if (l.empty()) {
    jb = JoinBatch();
    return;
  }
  in_stage(ctx, stage, [&](Tables& tb) -> std::function<void()> {
    const CountTables ct = count_tables(ctx, tb, l, r, jb);
    alloc_count(ctx, ct, jb);
    std::vector<JoinOut> jo(jb.J);
    parallel_for(jb.J, [&](size_t j) { describe_join(jb, j, jo[j]); });
    const size_t oj = tb.add(jo), oslot = tb.add(c0_slot);
    return [=, &ctx, &tb, &jb] {
      launch_placed(ctx, tb, ct, jb, tb.at<JoinOut>(oj), region, d_bump, nslots ? tb.at<int32_t>(oslot) : nullptr, host);
    };
  });
}

void JoinBatch::release(Ctx& ctx) {
  ctx.free(cnt.lo);
  ctx.free(cnt.offs);
  ctx.free(cnt.start);   // and match
  ctx.free(d_totals);    // and base
  cnt = {};
  d_totals = nullptr;
}

uint64_t col0_words(const std::vector<const Rel*>& rels) {
  uint64_t t = 0;
  for (const Rel* r : rels) t += r->nrows;
  return t;
}

void batched_col0_enqueue(Ctx& ctx, const std::vector<const Rel*>& rels, uint32_t* host, BatchStage* stage) {
  const uint32_t R = static_cast<uint32_t>(rels.size());
  if (R == 0) return;
  std::vector<Col0Req> rq(R);
  uint64_t total = 0;
  for (uint32_t q = 0; q < R; ++q) {
    rq[q] = {rels[q]->cols[0], rels[q]->nrows, total};
    total += rels[q]->nrows;
  }
  if (total == 0) return;
  in_stage(ctx, stage, [&](Tables& tb) -> std::function<void()> {
    const size_t orq = tb.add(rq);
    return [=, &ctx, &tb] {
      ctx.launch("col0_stage", 8.0 * total, [&] {
        col0_kernel<<<R < 1024 ? R : 1024, 128, 0, ctx.stream>>>(tb.at<Col0Req>(orq), R, host);
      });
      VG_CUDA(cudaGetLastError());
    };
  });
}

PinnedWords::~PinnedWords() { ctx_.give_pinned(p_, cap_); }

uint64_t* PinnedWords::reserve(size_t words) {
  const size_t bytes = std::max<size_t>(words, 1) * sizeof(uint64_t);
  if (p_ && bytes <= cap_) return p_;
  ctx_.give_pinned(p_, cap_);
  p_ = static_cast<uint64_t*>(ctx_.take_pinned(std::max<size_t>(bytes, size_t{1} << 16), &cap_));
  return p_;
}

}  // namespace vg
