// Permutation-index construction (hot path a).
//
// The three uint32 columns of the triples are packed into one 64-bit key,
// whose fields every sort takes as they lie: a permutation is the result of
// stable radix sorts by single fields, each starting from the last one's
// order.  (p, s) order comes first, from the digits of s and p only; the
// objects of each (p, s) group, usually a few, are put in order by the kernel
// that unpacks PSO.  From there
//   by o: (o, p, s) = OPS,  by p: (p, o, s) = POS,  by s: (s, p, o) = SPO,
//   by o: (o, s, p) = OSP,  by s: (s, o, p) = SOP.
// Sorting each permutation by its whole key took 12 passes over 100M triples
// (7 for PSO, 5 for POS from PSO) where this takes 8, and 40 where it takes
// 14 for the full index of 3M triples.
//
// One fused pass per permutation unpacks the sorted keys into the data
// columns and run-length encodes the level-1 and level-2 boundaries into
// (value, first row) arrays -- the reduce_by_key + exclusive scan pair of the
// reference -- with a decoupled look-back for the output positions.
#include "vg_index.h"

#include <algorithm>
#include <cstring>
#include <optional>

#include "vg_prims.cuh"
#include "vg_radix.cuh"
#include "vg_sort.h"

namespace vg {
namespace {

constexpr int kBlock = 256;
constexpr int kRows = 8;                 // rows per thread, 32 apart
constexpr int kTileRows = kBlock * kRows;
constexpr uint32_t kGroupMax = 64;       // groups of more rows are sorted apart (big_* below)

// Ids from this one on are literals (src/vedas.h:31); between the largest
// entity id and them lies an unused range, which the packed keys leave out.
constexpr uint32_t kLiteralStart = 50000000u;

// out4: the maxima of a, b and c, and c's among the ids below the literals,
// plus one (0: none).  Columns are read in 16-byte pieces where they are
// aligned.
__global__ void max4_kernel(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b,
                            const uint32_t* __restrict__ c, uint64_t n, uint32_t* out4) {
  uint32_t ma = 0, mb = 0, mc = 0, ml = 0;
  auto low = [&](uint32_t v) {
    if (v < kLiteralStart) ml = max(ml, v + 1);
  };
  const uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  uint64_t nv = 0;
  if (((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15u) == 0) {
    nv = n / 4;
    for (uint64_t i = t; i < nv; i += stride) {
      const uint4 x = reinterpret_cast<const uint4*>(a)[i];
      const uint4 y = reinterpret_cast<const uint4*>(b)[i];
      const uint4 z = reinterpret_cast<const uint4*>(c)[i];
      ma = max(ma, max(max(x.x, x.y), max(x.z, x.w)));
      mb = max(mb, max(max(y.x, y.y), max(y.z, y.w)));
      mc = max(mc, max(max(z.x, z.y), max(z.z, z.w)));
      low(z.x), low(z.y), low(z.z), low(z.w);
    }
  }
  for (uint64_t i = nv * 4 + t; i < n; i += stride) {
    ma = max(ma, a[i]);
    mb = max(mb, b[i]);
    mc = max(mc, c[i]);
    low(c[i]);
  }
  for (int d = 16; d > 0; d >>= 1) {
    ma = max(ma, __shfl_xor_sync(0xffffffffu, ma, d));
    mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, d));
    mc = max(mc, __shfl_xor_sync(0xffffffffu, mc, d));
    ml = max(ml, __shfl_xor_sync(0xffffffffu, ml, d));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&out4[0], ma);
    atomicMax(&out4[1], mb);
    atomicMax(&out4[2], mc);
    atomicMax(&out4[3], ml);
  }
}

// A field of the packed key: (key >> shift) & mask is the column's value,
// less `add` from `thr` on (the objects' unused range left out).
struct Field {
  uint32_t shift, mask, thr, add;
  __host__ __device__ uint64_t bits_of() const { return static_cast<uint64_t>(mask) << shift; }
  __device__ __forceinline__ uint32_t get(uint64_t key) const {
    const uint32_t v = static_cast<uint32_t>(key >> shift) & mask;
    return v >= thr ? v + add : v;
  }
  __device__ __forceinline__ uint64_t put(uint32_t v) const {
    return static_cast<uint64_t>(add && v >= kLiteralStart ? v - add : v) << shift;
  }
};

// Packed keys and the digit counts of every sort that follows (counts do not
// depend on the order of the keys): one read of the columns instead of a
// second one of the keys.
__global__ void __launch_bounds__(kBlock) pack_count_kernel(const uint32_t* __restrict__ s,
                                                            const uint32_t* __restrict__ p,
                                                            const uint32_t* __restrict__ o, uint64_t n, Field fs,
                                                            Field fp, Field fo, uint64_t* __restrict__ keys,
                                                            DigitList dl, unsigned long long* __restrict__ hist,
                                                            uint64_t* __restrict__ bases, uint32_t* done) {
  extern __shared__ uint32_t sh[];   // [dl.n][kRadixValues]
  digit_counts_init<kBlock>(dl, sh);
  auto pack = [&](uint32_t vs, uint32_t vp, uint32_t vo) { return fs.put(vs) | fp.put(vp) | fo.put(vo); };
  const uint64_t t = static_cast<uint64_t>(blockIdx.x) * kBlock + threadIdx.x;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * kBlock;
  uint64_t nv = 0;
  if (((reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(o)) & 15u) == 0) {
    nv = n / 4;
    for (uint64_t i = t; i < nv; i += stride) {
      const uint4 x = reinterpret_cast<const uint4*>(s)[i];
      const uint4 y = reinterpret_cast<const uint4*>(p)[i];
      const uint4 z = reinterpret_cast<const uint4*>(o)[i];
      const uint64_t k0 = pack(x.x, y.x, z.x), k1 = pack(x.y, y.y, z.y);
      const uint64_t k2 = pack(x.z, y.z, z.z), k3 = pack(x.w, y.w, z.w);
      ulonglong2* out = reinterpret_cast<ulonglong2*>(keys + 4 * i);
      out[0] = make_ulonglong2(k0, k1);
      out[1] = make_ulonglong2(k2, k3);
      digit_counts_add(dl, sh, k0);
      digit_counts_add(dl, sh, k1);
      digit_counts_add(dl, sh, k2);
      digit_counts_add(dl, sh, k3);
    }
  }
  for (uint64_t i = nv * 4 + t; i < n; i += stride) {
    const uint64_t k = pack(s[i], p[i], o[i]);
    keys[i] = k;
    digit_counts_add(dl, sh, k);
  }
  digit_counts_finish<kBlock>(dl, sh, hist, bases, done);
}

struct UnpackArgs {
  const uint64_t* keys;
  uint64_t n;
  Field f0, f1, f2;
  uint64_t m1, m2;         // key bits of (k0) and of (k0, k1): equal within a level-1 / level-2 run
  uint32_t* col1;          // k1 per row (nullable)
  uint32_t* col2;          // k2 per row (nullable)
  uint32_t* l1_vals;       // level-1 run values (k0) (nullable)
  uint32_t* l1_offs;
  uint32_t* l2_vals;       // level-2 run values (k1) (nullable)
  uint32_t* l2_offs;
  uint64_t* status1;
  uint64_t* status2;
  uint32_t* ticket;
  uint64_t* counts;        // [0] level-1 runs, [1] level-2 runs, [2] not 0: a group of more than kGroupMax rows
  uint64_t tiles;
  DeviceErrors* err;
};

// A tile is 2048 rows; a warp takes 256 consecutive ones, 32 at a time, so
// loads, column stores and (as nearly every row starts a level-2 run) run
// stores are all coalesced, and while warp 0 looks back the other warps store
// their columns.  100M rows take 0.67 ms (2.4 TB/s of keys, columns and runs),
// and 1.22 ms with GROUPS.
//
// GROUPS: the rows of a level-2 group come in any order of k2 and col2 gets
// them in ascending order, for groups of at most kGroupMax rows: k2 and the
// run heads of the tile and of 64 rows on either side lie in shared memory,
// and a row's place is the number of rows of its group that go before it.
// Groups average a few rows (the objects of one subject and predicate); a
// longer one keeps its order and sets counts[2].  What bounds it is that loop
// (8 steps a row, 13 for the slowest lane of a warp; two thirds of the issue
// slots): it saves the three passes of a sort by k2, 0.5 ms each.
template <bool GROUPS>
__global__ void __launch_bounds__(kBlock) unpack_rle_kernel(UnpackArgs a) {
  constexpr uint32_t kHalo = kGroupMax, kWarps = kBlock / 32;
  __shared__ uint32_t s_cnt[kWarps];
  __shared__ uint64_t s_b[2];
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_k2[GROUPS ? kTileRows + 2 * kHalo : 1];
  __shared__ uint32_t s_head[GROUPS ? (kTileRows + 2 * kHalo) / 32 : 1];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_tile = atomicAdd(a.ticket, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint64_t t0 = static_cast<uint64_t>(tile) * kTileRows;
  const uint64_t r0 = t0 + warp * (32u * kRows) + lane;

  uint64_t key[kRows];
#pragma unroll
  for (int i = 0; i < kRows; ++i) key[i] = r0 + i * 32u < a.n ? a.keys[r0 + i * 32u] : 0ull;
  uint64_t before = (lane == 0 && r0 > 0 && r0 <= a.n) ? a.keys[r0 - 1] : 0ull;
  uint32_t h1[kRows], h2[kRows];   // the warp's run heads, bit = lane
  uint32_t c1 = 0, c2 = 0;
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const uint64_t r = r0 + i * 32u;
    uint64_t pv = __shfl_up_sync(0xffffffffu, key[i], 1);
    if (lane == 0) pv = before;
    before = __shfl_sync(0xffffffffu, key[i], 31);
    const uint64_t x = key[i] ^ pv;
    h1[i] = __ballot_sync(0xffffffffu, r < a.n && (r == 0 || (x & a.m1)));
    h2[i] = __ballot_sync(0xffffffffu, r < a.n && (r == 0 || (x & a.m2)));
    c1 += __popc(h1[i]);
    c2 += __popc(h2[i]);
  }
  static_assert(kTileRows < (1 << 16), "a tile's run counts fit 16 bits each");
  if (lane == 0) s_cnt[warp] = (c1 << 16) | c2;
  if (GROUPS) {
    // rows past the end count as heads (they end the last group)
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const uint32_t x = kHalo + warp * (32u * kRows) + i * 32u;
      s_k2[x + lane] = static_cast<uint32_t>(key[i] >> a.f2.shift) & a.f2.mask;
      const uint32_t past = __ballot_sync(0xffffffffu, r0 + i * 32u >= a.n);
      if (lane == 0) s_head[x / 32] = h2[i] | past;
    }
    if (warp < 4) {
      // two warps for the 64 rows before the tile, two for those after it
      const uint32_t x = warp < 2 ? warp * 32u : kHalo + kTileRows + (warp - 2) * 32u;
      const bool in = t0 + x + lane >= kHalo && t0 + x + lane - kHalo < a.n;
      const uint64_t r = t0 + x + lane - kHalo;
      const uint64_t k = in ? a.keys[r] : 0ull;
      const uint64_t pv = in && r > 0 ? a.keys[r - 1] : 0ull;
      s_k2[x + lane] = static_cast<uint32_t>(k >> a.f2.shift) & a.f2.mask;
      const uint32_t h = __ballot_sync(0xffffffffu, !in || r == 0 || ((k ^ pv) & a.m2));
      if (lane == 0) s_head[x / 32] = h;
    }
  }
  __syncthreads();
  uint32_t pre = 0, all = 0;
#pragma unroll
  for (uint32_t w = 0; w < kWarps; ++w) {
    if (w < warp) pre += s_cnt[w];
    all += s_cnt[w];
  }
  const uint32_t t1 = all >> 16, t2 = all & 0xFFFFu;
  if (warp == 0) {
    // one look-back over both levels where the row count allows it (level 1
    // above bit 31, level 2 below)
    uint64_t g1 = 0, g2 = 0;
    if (a.l1_vals && a.l2_vals && a.n < (1ull << 31)) {
      const uint64_t g = warp_lookback(a.status1, tile, (static_cast<uint64_t>(t1) << 31) | t2, a.err);
      g1 = g >> 31;
      g2 = g & ((1ull << 31) - 1);
    } else {
      if (a.l1_vals) g1 = warp_lookback(a.status1, tile, t1, a.err);
      if (a.l2_vals) g2 = warp_lookback(a.status2, tile, t2, a.err);
    }
    if (lane == 0) {
      s_b[0] = g1;
      s_b[1] = g2;
      if (tile == a.tiles - 1) {
        a.counts[0] = g1 + t1;
        a.counts[1] = g2 + t2;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const uint64_t r = r0 + i * 32u;
    if (r < a.n && a.col1) a.col1[r] = a.f1.get(key[i]);
    if (!GROUPS && r < a.n && a.col2) a.col2[r] = a.f2.get(key[i]);
  }
  if (GROUPS) {
    // the last head before and the first after every 32 rows (the same for the
    // whole warp): a row's group is then two bit scans of its own 32 heads,
    // where a search of the words from each row's own took 45 of the kernel's
    // some 200 instructions a row, on diverging paths
    const uint32_t wb = kHalo / 32 + warp * kRows;
    uint32_t heads[kRows], next[kRows];
#pragma unroll
    for (int i = 0; i < kRows; ++i) heads[i] = s_head[wb + i];
    uint32_t prev = 0;   // 0: none found (a group that starts there is too long for the rows it is asked for)
    if (s_head[wb - 1]) prev = wb * 32 - 1 - __clz(s_head[wb - 1]);
    else if (s_head[wb - 2]) prev = wb * 32 - 33 - __clz(s_head[wb - 2]);
    uint32_t nx = 0xffffffffu;
    if (s_head[wb + kRows]) nx = (wb + kRows) * 32 - 1 + __ffs(s_head[wb + kRows]);
    else if (s_head[wb + kRows + 1]) nx = (wb + kRows) * 32 + 31 + __ffs(s_head[wb + kRows + 1]);
#pragma unroll
    for (int i = kRows - 1; i >= 0; --i) {
      next[i] = nx;
      if (heads[i]) nx = (wb + i) * 32 - 1 + __ffs(heads[i]);
    }
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const uint32_t w0 = (wb + i) * 32, x = w0 + lane;
      const uint32_t upto = 0xffffffffu >> (31u - lane);   // bits 0..lane
      const uint32_t hb = heads[i] & upto, he = heads[i] & ~upto;
      const uint32_t b = hb ? w0 + 31 - __clz(hb) : prev;   // [b, e): the group
      const uint32_t e = he ? w0 - 1 + __ffs(he) : next[i];
      if (heads[i]) prev = w0 + 31 - __clz(heads[i]);
      const uint32_t mine = s_k2[x];
      if (t0 + x - kHalo < a.n) {
        uint32_t at = x;
        if (b != 0 && e != 0xffffffffu && e - b <= kGroupMax) {
          at = b;
#pragma unroll 4
          for (uint32_t j = b; j < e; ++j) {
            const uint32_t v = s_k2[j];
            at += (v < mine || (v == mine && j < x)) ? 1u : 0u;
          }
        } else {
          a.counts[2] = 1;
        }
        if (a.col2) a.col2[t0 + at - kHalo] = mine >= a.f2.thr ? mine + a.f2.add : mine;
      }
    }
  }
  __syncthreads();
  uint64_t o1 = s_b[0] + (pre >> 16), o2 = s_b[1] + (pre & 0xFFFFu);
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const uint64_t r = r0 + i * 32u;
    if (a.l1_vals && (h1[i] >> lane & 1u)) {
      const uint64_t q = o1 + __popc(h1[i] & lanemask_lt());
      a.l1_vals[q] = a.f0.get(key[i]);
      a.l1_offs[q] = static_cast<uint32_t>(r);
    }
    if (a.l2_vals && (h2[i] >> lane & 1u)) {
      const uint64_t q = o2 + __popc(h2[i] & lanemask_lt());
      a.l2_vals[q] = a.f1.get(key[i]);
      a.l2_offs[q] = static_cast<uint32_t>(r);
    }
    o1 += __popc(h1[i]);
    o2 += __popc(h2[i]);
  }
}

// Groups of more than kGroupMax rows: listed (start row, first row among the
// rows of all such groups), their values sorted by (list position, value) and
// put back.  The packed counter (groups above bit 36, rows below) makes list
// order and row order agree.
struct BigGroups {
  unsigned long long* packed;
  uint32_t* start;
  uint64_t* at;
};

__global__ void big_list_kernel(const uint32_t* __restrict__ offs, uint64_t runs, uint64_t n, BigGroups g) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t r = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < runs; r += stride) {
    const uint64_t b = offs[r], e = r + 1 < runs ? offs[r + 1] : n;
    if (e - b <= kGroupMax) continue;
    const unsigned long long old = atomicAdd(g.packed, (1ull << 36) | (e - b));
    g.start[old >> 36] = static_cast<uint32_t>(b);
    g.at[old >> 36] = old & ((1ull << 36) - 1);
  }
}

// SCATTER: the sorted values back to the column; else the keys from it.
template <bool SCATTER>
__global__ void big_move_kernel(const uint32_t* __restrict__ start, const uint64_t* __restrict__ at, uint64_t groups,
                                uint64_t rows, uint32_t bits, uint32_t* __restrict__ col,
                                uint64_t* __restrict__ keys) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < rows; i += stride) {
    const uint64_t g = upper_bound_dev(at, 0, groups, i) - 1;
    uint32_t* c = col + start[g] + (i - at[g]);
    if (SCATTER) *c = static_cast<uint32_t>(keys[i] & ((1ull << bits) - 1));
    else keys[i] = (g << bits) | *c;
  }
}

int bits_for(uint64_t maxv) { return maxv == 0 ? 1 : 64 - __builtin_clzll(maxv); }
int passes_for(int bits) { return (bits + 7) / 8; }

unsigned grid_for(const Ctx& ctx, uint64_t n, int per_thread, int per_sm = 16) {
  uint64_t g = div_up(n, static_cast<uint64_t>(kBlock) * per_thread);
  const uint64_t gmax = static_cast<uint64_t>(ctx.num_sms) * per_sm;
  if (g > gmax) g = gmax;
  return static_cast<unsigned>(g < 1 ? 1 : g);
}

void column_max4(Ctx& ctx, const uint32_t* a, const uint32_t* b, const uint32_t* c, uint64_t n, uint32_t out[4]) {
  Scratch<uint32_t> d(ctx, 4);
  VG_CUDA(cudaMemsetAsync(d.get(), 0, 4 * sizeof(uint32_t), ctx.stream));
  if (n) {
    ctx.launch("column_max", 12.0 * n,
               [&] { max4_kernel<<<grid_for(ctx, n, 16, 8), kBlock, 0, ctx.stream>>>(a, b, c, n, d.get()); });
    VG_CUDA(cudaGetLastError());
  }
  VG_CUDA(cudaMemcpyAsync(ctx.h_small, d.get(), 4 * sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx.stream));
  ctx.sync();
  for (int i = 0; i < 4; ++i) out[i] = reinterpret_cast<const uint32_t*>(ctx.h_small)[i];
}

// Builds of at most kLateRows rows wait for the host once, when the largest
// free block holds kLateBytes per row (the full index's outputs at full size
// and two key buffers take 108, up to twice that in the arena's size classes):
// 1.25 -> 1.18 ms for the full index of 3M triples.  With more rows a wait is a
// small part.
constexpr uint64_t kLateRows = 16u << 20, kLateBytes = 256;

// The packed keys of one build and the sorts and unpackings over them.
class Permuter {
 public:
  enum Col { S, P, O };

  Permuter(Ctx& ctx, const uint32_t* s, const uint32_t* p, const uint32_t* o, uint64_t n, const uint32_t mx[4],
           bool full)
      : ctx_(ctx), n_(n), max_o_(mx[2]), late_(n <= kLateRows && ctx.arena.largest_free() >= kLateBytes * n) {
    // objects without the unused range below the literals
    const bool lits = mx[2] >= kLiteralStart;
    const uint32_t cut = lits ? kLiteralStart - mx[3] : 0;
    const int bs = bits_for(mx[0]), bp = bits_for(mx[1]), bo = bits_for(mx[2] - cut);
    // p on top; whichever of s and o lies below it shares its digits with p
    // where that saves a pass of a two-column sort
    const int apart = passes_for(bp);
    const int with_s = passes_for(bs + bp) + passes_for(bo) + apart, with_o = passes_for(bs) + apart + passes_for(bo + bp);
    const bool s_next = full || with_s <= with_o;
    const int at_s = s_next ? bo : 0, at_o = s_next ? 0 : bs, at_p = bs + bo;
    auto mask = [](int bits) { return static_cast<uint32_t>((1ull << bits) - 1); };
    f_[S] = {static_cast<uint32_t>(at_s), mask(bs), 0xffffffffu, 0};
    f_[P] = {static_cast<uint32_t>(at_p), mask(bp), 0xffffffffu, 0};
    f_[O] = {static_cast<uint32_t>(at_o), mask(bo), lits ? mx[3] : 0xffffffffu, cut};
    plan({S}, at_s, at_s + bs);
    plan({P}, at_p, at_p + bp);
    plan({O}, at_o, at_o + bo);
    const Col low = s_next ? S : O;
    const int at_low = s_next ? at_s : at_o, b_low = s_next ? bs : bo;
    if (passes_for(b_low + bp) < passes_for(b_low) + apart) plan({low, P}, at_low, at_p + bp);

    DigitList dl{};
    for (const Sort& q : sorts_)
      for (const RadixDigit& d : q.digits) dl.d[dl.n++] = d;
    counts_.emplace(ctx, dl);
    uint32_t at = 0;
    for (Sort& q : sorts_)
      for (size_t d = 0; d < q.digits.size(); ++d) q.bases.push_back(counts_->bases(at++));
    keys_.emplace(ctx, n);
    ctx.launch("index_pack", 20.0 * n, [&] {
      pack_count_kernel<<<grid_for(ctx, n, 16, 8), kBlock, dl.n * kRadixValues * sizeof(uint32_t), ctx.stream>>>(
          s, p, o, n, f_[S], f_[P], f_[O], keys_->get(), dl, counts_->hist(), counts_->bases(), counts_->done());
    });
    VG_CUDA(cudaGetLastError());
  }
  Permuter(const Permuter&) = delete;
  Permuter& operator=(const Permuter&) = delete;

  // Stable sort of the keys by the columns, the last named counting most.
  void sort_by(const std::vector<Col>& cols) {
    std::vector<RadixDigit> digits;
    std::vector<const uint64_t*> bases;
    auto take = [&](const std::vector<Col>& c) {
      for (const Sort& q : sorts_)
        if (q.cols == c) {
          digits.insert(digits.end(), q.digits.begin(), q.digits.end());
          bases.insert(bases.end(), q.bases.begin(), q.bases.end());
          return true;
        }
      return false;
    };
    if (!take(cols))
      for (Col c : cols) take({c});
    Scratch<uint64_t> alt(ctx_, n_);
    if (radix_sort_u64_counted(ctx_, keys_->get(), alt.get(), nullptr, nullptr, n_, digits, bases)) std::swap(keys_->p, alt.p);
  }

  // The requested outputs of the keys as (c0, c1, c2); groups: the keys are
  // in (c0, c1) order only.
  void unpack(Col c0, Col c1, Col c2, PermOutputs& out, bool groups = false) {
    Ctx& ctx = ctx_;
    const uint64_t n = n_;
    UnpackArgs a{};
    a.keys = keys_->get();
    a.n = n;
    a.f0 = f_[c0];
    a.f1 = f_[c1];
    a.f2 = f_[c2];
    a.m1 = a.f0.bits_of();
    a.m2 = a.m1 | a.f1.bits_of();
    auto room = [&](bool want, DevArray& d) {   // (the outputs': freed with them if the build fails)
      if (want) d = DevArray(ctx.alloc<uint32_t>(n), n);
      return d.ptr;
    };
    a.col1 = room(out.want_col1, out.col1);
    a.col2 = room(out.want_col2, out.col2);
    a.l1_vals = room(out.want_l1, out.l1_vals);
    a.l1_offs = room(out.want_l1, out.l1_offs);
    a.l2_vals = room(out.want_l2, out.l2_vals);
    a.l2_offs = room(out.want_l2, out.l2_offs);
    a.tiles = div_up(n, kTileRows);
    // counts, ticket and both levels' look-back words, zeroed together
    Scratch<uint64_t> z(ctx, 4 + 2 * a.tiles);
    VG_CUDA(cudaMemsetAsync(z.get(), 0, (4 + 2 * a.tiles) * sizeof(uint64_t), ctx.stream));
    a.counts = z.get();
    a.ticket = reinterpret_cast<uint32_t*>(z.get() + 3);
    a.status1 = z.get() + 4;
    a.status2 = z.get() + 4 + a.tiles;
    a.err = ctx.d_err;
    const double ub = 8.0 * n + 4.0 * n * ((a.col1 ? 1 : 0) + (a.col2 ? 1 : 0));
    ctx.launch("index_unpack_rle", ub, [&] {
      if (groups) unpack_rle_kernel<true><<<static_cast<unsigned>(a.tiles), kBlock, 0, ctx.stream>>>(a);
      else unpack_rle_kernel<false><<<static_cast<unsigned>(a.tiles), kBlock, 0, ctx.stream>>>(a);
    });
    VG_CUDA(cudaGetLastError());
    // counts and error record, read when the stream has got here
    const size_t slot = pending_.size();
    uint64_t* h = ctx.h_small + slot * kSlotWords;
    VG_CUDA(cudaMemcpyAsync(h, z.get(), 3 * sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx.stream));
    VG_CUDA(cudaMemcpyAsync(h + 3, ctx.d_err, sizeof(DeviceErrors), cudaMemcpyDeviceToHost, ctx.stream));
    pending_.push_back({&out, a, groups});
    if (!late_) finish();
  }

  // Waits for the unpackings enqueued so far and gives their outputs their
  // sizes.
  void finish() {
    Ctx& ctx = ctx_;
    const std::vector<Pending> all = std::move(pending_);
    pending_.clear();
    if (all.empty()) return;
    ctx.sync();
    uint64_t hc[kSlots][3];
    for (size_t k = 0; k < all.size(); ++k) {
      const uint64_t* h = ctx.h_small + k * kSlotWords;
      std::copy(h, h + 3, hc[k]);
      DeviceErrors he;
      std::memcpy(&he, h + 3, sizeof(he));
      ctx.raise_device_errors(he);
    }
    for (size_t k = 0; k < all.size(); ++k) {
      PermOutputs& out = *all[k].out;
      const UnpackArgs& a = all[k].a;
      if (a.l1_vals) {
        ctx.arena.shrink(a.l1_vals, hc[k][0] * 4);
        ctx.arena.shrink(a.l1_offs, hc[k][0] * 4);
        out.l1_vals.len = out.l1_offs.len = hc[k][0];
      }
      if (a.l2_vals) {
        ctx.arena.shrink(a.l2_vals, hc[k][1] * 4);
        ctx.arena.shrink(a.l2_offs, hc[k][1] * 4);
        out.l2_vals.len = out.l2_offs.len = hc[k][1];
      }
      if (all[k].groups && hc[k][2]) sort_big_groups(out);
    }
  }

 private:
  struct Sort {
    std::vector<Col> cols;
    std::vector<RadixDigit> digits;
    std::vector<const uint64_t*> bases;
  };
  struct Pending {
    PermOutputs* out;
    UnpackArgs a;
    bool groups;
  };
  static constexpr size_t kSlots = 6, kSlotWords = 4;   // unpackings, and the words the host reads of each
  static_assert(sizeof(DeviceErrors) <= sizeof(uint64_t) && kSlots * kSlotWords <= Ctx::kSmallWords,
                "the counts and error records fit the small staging buffer");
  Ctx& ctx_;
  uint64_t n_;
  uint32_t max_o_;
  // Whether the host waits for all unpackings at the end only, so that no sort
  // waits for it: the boundary arrays, made for as many runs as rows, then
  // keep that size until the end.
  bool late_;
  std::vector<Pending> pending_;
  Field f_[3];
  std::vector<Sort> sorts_;
  std::optional<RadixCounts> counts_;       // digit counts and bases of every sort
  std::optional<Scratch<uint64_t>> keys_;   // the packed keys in their present order

  void plan(const std::vector<Col>& cols, int begin, int end) {
    Sort q;
    q.cols = cols;
    radix_plan(q.digits, begin, end);
    sorts_.push_back(std::move(q));
  }

  // Orders col2 (objects) within the level-2 runs of more than kGroupMax rows.
  void sort_big_groups(PermOutputs& out) {
    Ctx& ctx = ctx_;
    const uint64_t runs = out.l2_offs.len;
    const uint64_t most = n_ / (kGroupMax + 1) + 1;
    Scratch<uint32_t> start(ctx, most);
    Scratch<uint64_t> at(ctx, most);
    Scratch<unsigned long long> packed(ctx, 1);
    VG_CUDA(cudaMemsetAsync(packed.get(), 0, sizeof(unsigned long long), ctx.stream));
    ctx.launch("index_big_groups", 4.0 * runs, [&] {
      big_list_kernel<<<grid_for(ctx, runs, 4), kBlock, 0, ctx.stream>>>(out.l2_offs.ptr, runs, n_,
                                                                        {packed.get(), start.get(), at.get()});
    });
    VG_CUDA(cudaGetLastError());
    VG_CUDA(cudaMemcpyAsync(ctx.h_small, packed.get(), sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    const uint64_t groups = ctx.h_small[0] >> 36, rows = ctx.h_small[0] & ((1ull << 36) - 1);
    if (groups == 0) return;
    const int bo = bits_for(max_o_);
    Scratch<uint64_t> kb(ctx, rows), ab(ctx, rows);
    uint64_t *keys = kb.get(), *alt = ab.get();
    ctx.launch("index_big_groups", 12.0 * rows, [&] {
      big_move_kernel<false><<<grid_for(ctx, rows, 4), kBlock, 0, ctx.stream>>>(
          start.get(), at.get(), groups, rows, static_cast<uint32_t>(bo), out.col2.ptr, keys);
    });
    VG_CUDA(cudaGetLastError());
    if (radix_sort_u64(ctx, keys, alt, rows, bo + (groups > 1 ? bits_for(groups - 1) : 0)))
      std::swap(keys, alt);
    ctx.launch("index_big_groups", 12.0 * rows, [&] {
      big_move_kernel<true><<<grid_for(ctx, rows, 4), kBlock, 0, ctx.stream>>>(
          start.get(), at.get(), groups, rows, static_cast<uint32_t>(bo), out.col2.ptr, keys);
    });
    VG_CUDA(cudaGetLastError());
  }
};

}  // namespace

void column_max3(Ctx& ctx, const uint32_t* a, const uint32_t* b, const uint32_t* c, uint64_t n,
                 uint32_t out[3]) {
  uint32_t m[4];
  column_max4(ctx, a, b, c, n, m);
  std::copy(m, m + 3, out);
}

uint32_t build_permutations(Ctx& ctx, const uint32_t* s, const uint32_t* p, const uint32_t* o, uint64_t n,
                            Permutations& out, bool full) {
  uint32_t mx[4];
  column_max4(ctx, s, p, o, n, mx);
  if (bits_for(mx[0]) + bits_for(mx[1]) + bits_for(mx[2]) > 64)
    fail(VG_ERR_UNSUPPORTED, "triple ids need more than 64 key bits for the packed index sort");
  if (n == 0) return 0;
  try {
    using C = Permuter;
    Permuter keys(ctx, s, p, o, n, mx, full);
    keys.sort_by({C::S, C::P});
    keys.unpack(C::P, C::S, C::O, out.pso, true);
    if (!full) {
      keys.sort_by({C::O, C::P});
      keys.unpack(C::P, C::O, C::S, out.pos);
    } else {
      keys.sort_by({C::O});
      keys.unpack(C::O, C::P, C::S, out.ops);
      keys.sort_by({C::P});
      keys.unpack(C::P, C::O, C::S, out.pos);
      keys.sort_by({C::S});
      keys.unpack(C::S, C::P, C::O, out.spo);
      keys.sort_by({C::O});
      keys.unpack(C::O, C::S, C::P, out.osp);
      keys.sort_by({C::S});
      keys.unpack(C::S, C::O, C::P, out.sop);
    }
    keys.finish();
  } catch (...) {
    for (PermOutputs* q : {&out.pso, &out.pos, &out.spo, &out.sop, &out.osp, &out.ops})
      for (DevArray* d : {&q->col1, &q->col2, &q->l1_vals, &q->l1_offs, &q->l2_vals, &q->l2_offs}) {
        if (d->ptr) ctx.free(d->ptr);
        d->clear();
      }
    throw;
  }
  return std::max(mx[0], std::max(mx[1], mx[2]));
}

}  // namespace vg
