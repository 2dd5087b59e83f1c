// N-Triples ingest on the device.
//
// 1. the lines' number, which sizes everything else: newlines are counted, or
//    (long texts, parsed while they are copied) guessed from samples;
// 2. blocks take 16 KiB pieces of the text into shared memory, find their
//    lines, and one thread parses each line into its three terms and looks
//    them up in one open-addressing table of terms: a slot is claimed by the
//    place of a term's text, so terms are compared byte by byte and equal
//    hashes need no further care.  Every slot keeps the lowest line its term
//    occurs on;
// 3. a scan over the lines counts statements and, per dictionary, the terms
//    that occur first on each line: their ids, in order of first appearance;
// 4. ids go to the s, p, o columns, and the text of every id's term, in id
//    order, to the host.
//
// The table replaced a radix sort of 63-bit hashes per dictionary (31 passes),
// run heads, a byte-by-byte check and a second sort into id order: 2.5 ms of
// kernels for 1M statements (101 MB).
#include "vg_ingest.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <fstream>
#include <optional>
#include <sstream>
#include <string_view>

#include "vg_pool.h"
#include "vg_prims.cuh"

namespace vg {
namespace {

constexpr int kBlock = 256;
constexpr uint32_t kPiece = kBlock * 64;       // bytes of text per block
constexpr uint32_t kHalo = 1024;               // bytes after the piece, for the line that leaves it
constexpr uint32_t kLineList = 2048;           // lines of a piece listed at a time
constexpr int kRows = 8;
constexpr uint64_t kTileLines = kBlock * kRows;
constexpr uint32_t kProbeMax = 8192;           // a longer search gives up (the host then resolves the terms)

// A long text is copied and parsed in parts of a quarter of it, within these
// bounds (101 MB, us in all: one part 1157, parts of 52 MB 1159, 40 1023, 33
// 1066, 26 1040, 17 1078, 8 1137: a part's copy starts some 20 us late).  Around
// them the sizes matter little: 39 MB take 0.60 ms with parts of 16 MB at least,
// 0.62 with 8 and 0.64 with 32; 997 MB 7.12 ms with 64 MB at most, 7.42 with 32
// and 7.09 with 256.
constexpr uint64_t kUploadLeast = 16ull << 20, kUploadMost = 64ull << 20;

std::atomic<int> g_hash_bits{63};

// Where the terms of each line lie (only made for the host's exact path):
// lengths are 0 where the line holds no statement.
struct Spans {
  uint64_t* off[3];   // subject, predicate, object
  uint64_t* len[3];
  uint8_t* lit;
};

// A slot of the term table.  loc is the place of the term that claimed it:
// (offset << len_bits | length) << 2 | dictionary (0 subjects and objects, 1
// predicates, 2 literals), never 0.  first holds ~(lowest line), so that
// zeroed memory is an empty table; id is set once ids are known.
struct Slot {
  unsigned long long loc;
  uint32_t first;
  uint32_t id;
};
static_assert(sizeof(Slot) == 16, "one 16-byte slot");
constexpr uint32_t kNoSlot = 0xffffffffu;

struct Flags {                   // device flags of the parse
  unsigned long long bad_line;   // lowest malformed line, from 1 (~0: none)
  unsigned long long newlines;   // of the whole text
  uint32_t give_up;              // a term too long for loc, or a search past kProbeMax
  uint32_t far;                  // lines left to far_lines_kernel
};
struct FarLine {
  uint64_t line, start;
};

// ---------------------------------------------------------------------------
// 1. newlines
constexpr uint32_t kNewlines = 0x0a0a0a0au;

__global__ void newline_count_kernel(const uint8_t* __restrict__ text, uint64_t len,
                                     unsigned long long* __restrict__ count) {
  const uint64_t words = len / 16;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  uint32_t c = 0;
  for (uint64_t w = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; w < words; w += stride) {
    const uint4 v = reinterpret_cast<const uint4*>(text)[w];
    c += (__popc(__vcmpeq4(v.x, kNewlines)) + __popc(__vcmpeq4(v.y, kNewlines)) +
          __popc(__vcmpeq4(v.z, kNewlines)) + __popc(__vcmpeq4(v.w, kNewlines))) >> 3;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0)
    for (uint64_t b = words * 16; b < len; ++b) c += text[b] == '\n' ? 1u : 0u;
  c = static_cast<uint32_t>(warp_sum64(c));
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, static_cast<unsigned long long>(c));
}


// ---------------------------------------------------------------------------
// 2. lines, statements and terms
__device__ __forceinline__ bool is_ws(uint8_t c) { return c == ' ' || c == '\t' || c == '\r'; }

// nb (1..8) bytes at p + off as a little-endian word.  p is 8-byte aligned;
// only the aligned words that hold those bytes are read.
__device__ __forceinline__ uint64_t word_at(const uint8_t* p, uint64_t off, uint32_t nb) {
  const uint64_t* q = reinterpret_cast<const uint64_t*>(p + (off & ~7ull));
  const uint32_t in = static_cast<uint32_t>(off & 7);
  uint64_t w = q[0] >> (8 * in);
  if (in + nb > 8) w |= q[1] << (64 - 8 * in);
  return nb < 8 ? w & ((1ull << (8 * nb)) - 1) : w;
}

// Term at t[i]; returns its end (one past) or 0 on a malformed term.
// kind: 0 any, 1 IRI only (predicate), 2 IRI or blank node (subject).
template <typename I>
__device__ __forceinline__ I iri_end(const uint8_t* t, I i, I end) {
  for (I j = i + 1; j < end; ++j) {
    if (t[j] == '>') return j + 1;
    if (t[j] == ' ' || t[j] == '\t') return 0;
  }
  return 0;
}
template <typename I>
__device__ I term_end(const uint8_t* t, I i, I end, int kind, bool& literal) {
  literal = false;
  if (i >= end) return 0;
  const uint8_t c = t[i];
  if (c == '<') return iri_end<I>(t, i, end);
  if (kind == 1) return 0;
  if (c == '_') {
    if (i + 1 >= end || t[i + 1] != ':') return 0;
    I j = i + 2;
    while (j < end && !is_ws(t[j])) ++j;
    if (j == i + 2) return 0;
    // a label does not end with '.': "_:b1." before the statement's dot
    if (t[j - 1] == '.' && j - 1 > i + 2) --j;
    return j;
  }
  if (kind == 2 || c != '"') return 0;
  I j = i + 1;
  while (j < end) {
    if (t[j] == '\\') {
      j += 2;
      continue;
    }
    if (t[j] == '"') break;
    ++j;
  }
  if (j >= end) return 0;
  ++j;   // past the closing quote
  literal = true;
  if (j < end && t[j] == '@') {
    I k = j + 1;
    while (k < end && ((t[k] >= 'a' && t[k] <= 'z') || (t[k] >= 'A' && t[k] <= 'Z') ||
                       (t[k] >= '0' && t[k] <= '9') || t[k] == '-'))
      ++k;
    if (k == j + 1) return 0;
    return k;
  }
  if (j + 1 < end && t[j] == '^' && t[j + 1] == '^')
    return j + 2 < end && t[j + 2] == '<' ? iri_end<I>(t, j + 2, end) : 0;
  return j;
}

// The statement on t[b, e): 0 none (blank or comment), 1 well formed (its
// terms at off, len), 2 malformed.
template <typename I>
__device__ int parse_line(const uint8_t* t, I b, I e, I (&off)[3], I (&len)[3], bool& lit) {
  I i = b;
  while (i < e && is_ws(t[i])) ++i;
  if (i >= e || t[i] == '#') return 0;
#pragma unroll 1
  for (int k = 0; k < 3; ++k) {
    off[k] = i;
    const I end = term_end<I>(t, i, e, k == 0 ? 2 : (k == 1 ? 1 : 0), lit);
    if (end == 0) return 2;
    len[k] = end - i;
    i = end;
    const I ws = i;
    while (i < e && is_ws(t[i])) ++i;
    if (k < 2 && i == ws) return 2;
  }
  if (i >= e || t[i] != '.') return 2;
  ++i;
  while (i < e && is_ws(t[i])) ++i;
  return i >= e || t[i] == '#' ? 1 : 2;
}

// A 64-bit multiply-xorshift mix over 8-byte words: David Stafford's published
// "Mix01" constants for MurmurHash3's 64-bit finalizer ("Better Bit Mixing",
// 2011).  Any good mix works: terms are compared byte by byte.
__device__ __forceinline__ uint64_t mix64(uint64_t h) {
  h ^= h >> 31;
  h *= 0x7fb5d329728ea185ull;
  h ^= h >> 27;
  h *= 0x81dadef4bc2dd44dull;
  h ^= h >> 33;
  return h;
}

struct Table {
  Slot* slots;
  uint64_t cap;
  uint32_t len_bits;
  int hash_bits;
};

// The slot of the term at t + off (text offset at), claimed if it is new;
// kNoSlot (and give_up set) when there is none to be had.
__device__ uint32_t find_slot(const Table& tb, const uint8_t* text, const uint8_t* t, uint64_t off, uint64_t at,
                              uint64_t len, uint32_t dict, uint32_t line, Flags* fl) {
  if (len >> tb.len_bits) {
    fl->give_up = 1;
    return kNoSlot;
  }
  uint64_t h = 0x243f6a8885a308d3ull ^ (len << 2 | dict);
  for (uint64_t i = 0; i < len; i += 8)
    h = mix64(h ^ word_at(t, off + i, static_cast<uint32_t>(len - i < 8 ? len - i : 8)));
  if (tb.hash_bits < 63) h &= ~((1ull << (64 - tb.hash_bits)) - 1);
  const unsigned long long mine = ((at << tb.len_bits | len) << 2) | dict;
  uint64_t i = __umul64hi(h, tb.cap);
  for (uint32_t probe = 0; probe < kProbeMax; ++probe) {
    Slot* s = &tb.slots[i];
    unsigned long long loc = s->loc;
    if (loc == 0) loc = atomicCAS(&s->loc, 0ull, mine);
    bool same = loc == 0 || loc == mine;
    if (!same && (loc & 3) == dict && ((loc >> 2) & ((1ull << tb.len_bits) - 1)) == len) {
      const uint64_t other = loc >> (2 + tb.len_bits);
      same = true;
      for (uint64_t k = 0; same && k < len; k += 8) {
        const uint32_t nb = static_cast<uint32_t>(len - k < 8 ? len - k : 8);
        same = word_at(t, off + k, nb) == word_at(text, other + k, nb);
      }
    }
    if (same) {
      // most occurrences come after their term's first one: no atomic then
      if (s->first < ~line) atomicMax(&s->first, ~line);
      return static_cast<uint32_t>(i);
    }
    if (++i == tb.cap) i = 0;
    if ((probe & 63) == 63 && *reinterpret_cast<volatile uint32_t*>(&fl->give_up)) return kNoSlot;
  }
  fl->give_up = 1;
  return kNoSlot;
}

// Byte classes of a piece as bitmaps, one 64-bit word per 64 bytes: a parser
// that jumps from one byte of interest to the next reads a word or two where
// it read every byte (0.47 ms for 101 MB).
struct ByteMaps {
  static constexpr uint32_t kWords = (kPiece + kHalo) / 64;
  uint64_t iri_stop[kWords];   // '>', space, tab
  uint64_t space[kWords];      // space, tab, carriage return
  uint64_t quote[kWords];      // '"', backslash
};

// 0x80 in every byte of w that equals c.
__device__ __forceinline__ uint32_t bytes_equal(uint32_t w, uint8_t c) {
  const uint32_t x = w ^ (0x01010101u * c);
  return ~(((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x | 0x7f7f7f7fu);
}
// The four top bits of such a mask, lowest byte first.
__device__ __forceinline__ uint64_t byte_bits(uint32_t m) {
  return ((m >> 7) * 0x00204081u >> 21) & 15u;
}

// Classifies the 64 bytes at s_text + 64 * word (bytes from `have` on belong
// to no class); returns their newlines.
__device__ __forceinline__ uint64_t classify(const uint8_t* s_text, uint32_t word, uint32_t have, ByteMaps& bm) {
  uint64_t stop = 0, space = 0, quote = 0, nl = 0;
#pragma unroll 4
  for (int q = 0; q < 16; ++q) {
    const uint32_t w = reinterpret_cast<const uint32_t*>(s_text)[word * 16 + q];
    const uint32_t blank = bytes_equal(w, ' ') | bytes_equal(w, '\t');
    stop |= byte_bits(blank | bytes_equal(w, '>')) << (4 * q);
    space |= byte_bits(blank | bytes_equal(w, '\r')) << (4 * q);
    quote |= byte_bits(bytes_equal(w, '"') | bytes_equal(w, '\\')) << (4 * q);
    nl |= byte_bits(bytes_equal(w, '\n')) << (4 * q);
  }
  const uint32_t first = word * 64;
  const uint64_t in = first >= have ? 0 : have - first >= 64 ? ~0ull : (1ull << (have - first)) - 1;
  bm.iri_stop[word] = stop & in;
  bm.space[word] = space & in;
  bm.quote[word] = quote & in;
  return nl & in;
}

// First byte of [i, e) in the class (SET) or outside it; e when there is none.
template <bool SET>
__device__ __forceinline__ uint32_t next_byte(const uint64_t* map, uint32_t i, uint32_t e) {
  if (i >= e) return e;
  uint32_t w = i >> 6;
  uint64_t m = (SET ? map[w] : ~map[w]) >> (i & 63);
  uint32_t at = i;
  while (m == 0) {
    at = ++w * 64;
    if (at >= e) return e;
    m = SET ? map[w] : ~map[w];
  }
  at += __ffsll(static_cast<long long>(m)) - 1;
  return at < e ? at : e;
}

// term_end and parse_line for a line within the piece, over its byte maps.
__device__ __forceinline__ uint32_t mapped_term_end(const uint8_t* t, const ByteMaps& bm, uint32_t i, uint32_t end,
                                                    int kind, bool& literal) {
  literal = false;
  if (i >= end) return 0;
  const uint8_t c = t[i];
  if (c == '<') {
    const uint32_t j = next_byte<true>(bm.iri_stop, i + 1, end);
    return j < end && t[j] == '>' ? j + 1 : 0;
  }
  if (kind == 1) return 0;
  if (c == '_') {
    if (i + 1 >= end || t[i + 1] != ':') return 0;
    uint32_t j = next_byte<true>(bm.space, i + 2, end);
    if (j == i + 2) return 0;
    if (t[j - 1] == '.' && j - 1 > i + 2) --j;
    return j;
  }
  if (kind == 2 || c != '"') return 0;
  uint32_t j = i + 1;
  while (true) {
    j = next_byte<true>(bm.quote, j, end);
    if (j >= end) return 0;
    if (t[j] == '"') break;
    j += 2;   // a backslash and what it escapes
  }
  ++j;
  literal = true;
  if (j < end && t[j] == '@') {
    uint32_t k = j + 1;
    while (k < end && ((t[k] >= 'a' && t[k] <= 'z') || (t[k] >= 'A' && t[k] <= 'Z') ||
                       (t[k] >= '0' && t[k] <= '9') || t[k] == '-'))
      ++k;
    return k == j + 1 ? 0 : k;
  }
  if (j + 1 < end && t[j] == '^' && t[j + 1] == '^') {
    if (j + 2 >= end || t[j + 2] != '<') return 0;
    const uint32_t k = next_byte<true>(bm.iri_stop, j + 3, end);
    return k < end && t[k] == '>' ? k + 1 : 0;
  }
  return j;
}

__device__ __forceinline__ int mapped_parse_line(const uint8_t* t, const ByteMaps& bm, uint32_t b, uint32_t e,
                                                 uint32_t (&off)[3], uint32_t (&len)[3], bool& lit) {
  uint32_t i = next_byte<false>(bm.space, b, e);
  if (i >= e || t[i] == '#') return 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    off[k] = i;
    const uint32_t end = mapped_term_end(t, bm, i, e, k == 0 ? 2 : (k == 1 ? 1 : 0), lit);
    if (end == 0) return 2;
    len[k] = end - i;
    i = next_byte<false>(bm.space, end, e);
    if (k < 2 && i == end) return 2;
  }
  if (i >= e || t[i] != '.') return 2;
  i = next_byte<false>(bm.space, i + 1, e);
  return i >= e || t[i] == '#' ? 1 : 2;
}

// A line that leaves its piece by more than kHalo bytes, by one thread from
// global memory.
__device__ __noinline__ void parse_far_line(const uint8_t* __restrict__ text, uint64_t len, uint64_t start,
                                            uint64_t line, uint64_t rows, const Table& tb,
                                            uint32_t* __restrict__ slots, const Spans& sp, bool literal_dict,
                                            Flags* fl) {
  uint64_t e = start;
  while (e < len && text[e] != '\n') ++e;
  uint64_t off[3] = {0, 0, 0}, tl[3] = {0, 0, 0};
  bool lit = false;
  const int got = parse_line<uint64_t>(text, start, e, off, tl, lit);
  if (slots) {
    if (got == 1) {
      for (int q = 0; q < 3; ++q) {
        const uint32_t dict = q == 1 ? 1u : (q == 2 && lit && literal_dict ? 2u : 0u);
        slots[q * rows + line] = find_slot(tb, text, text, off[q], off[q], tl[q], dict, static_cast<uint32_t>(line), fl);
      }
    } else {
      slots[line] = kNoSlot;
    }
  }
  if (sp.lit) {
    for (int q = 0; q < 3; ++q) {
      sp.off[q][line] = off[q];
      sp.len[q][line] = got == 1 ? tl[q] : 0;
    }
    sp.lit[line] = lit ? 1 : 0;
  }
  if (got == 2) atomicMin(&fl->bad_line, static_cast<unsigned long long>(line + 1));
}

// The lines that parse_kernel put aside because their text had not all
// arrived (at most one a piece).
__global__ void __launch_bounds__(kBlock) far_lines_kernel(const uint8_t* __restrict__ text, uint64_t len, uint64_t rows,
                                                           Table tb, uint32_t* __restrict__ slots, bool literal_dict,
                                                           const FarLine* __restrict__ far, Flags* fl) {
  const uint32_t n = fl->far, stride = gridDim.x * kBlock;
  for (uint32_t i = blockIdx.x * kBlock + threadIdx.x; i < n; i += stride)
    parse_far_line(text, len, far[i].start, far[i].line, rows, tb, slots, Spans{}, literal_dict, fl);
}

// A block per piece of kPiece bytes, in ticket order; it owns the lines that
// start after the piece's newlines (and the text's first line).  The piece
// lies in shared memory (from global memory a byte at a time costs a cache
// access per byte and lane).  Its lines are taken kBlock at a time: one
// thread parses each, then the threads share their terms, three a line, out
// among them for the table searches.  A line that ends more than kHalo bytes
// after the piece is parsed and looked up by one thread from global memory, at
// once or (far given: the text has not all arrived) by far_lines_kernel.
// slots: [3][rows], kNoSlot in the subject's place where the line holds no
// statement; lines from `rows` on are only counted.  A text may take several
// launches, each over the pieces that have arrived with their halos: tickets
// and look-back words carry on.
__global__ void __launch_bounds__(kBlock, 4) parse_kernel(const uint8_t* __restrict__ text, uint64_t len,
                                                          uint64_t rows, Table tb, uint32_t* __restrict__ slots,
                                                          Spans sp, bool literal_dict, uint64_t* status,
                                                          uint32_t* ticket, FarLine* __restrict__ far, Flags* fl,
                                                          DeviceErrors* err) {
  __shared__ __align__(16) uint8_t s_text[kPiece + kHalo + 16];
  __shared__ ByteMaps s_map;
  __shared__ uint16_t s_start[kLineList + 1];   // first bytes of the listed lines (kPiece at most)
  __shared__ uint32_t s_term[3][kBlock];        // length << 16 | first byte (0: no term, or looked up already)
  __shared__ uint8_t s_lit[kBlock];
  __shared__ uint32_t s_scan[kBlock / 32 + 1];
  __shared__ uint64_t s_b;
  __shared__ uint32_t s_tile;
  static_assert(kPiece + kHalo < (1 << 16), "places and lengths in a piece fit 16 bits");
  static_assert(kLineList % kBlock == 0, "listed lines are taken kBlock at a time");
  const uint32_t tid = threadIdx.x;
  if (tid == 0) s_tile = atomicAdd(ticket, 1u);
  __syncthreads();
  const uint64_t base = static_cast<uint64_t>(s_tile) * kPiece;
  // the text is padded to whole 16-byte words
  const uint32_t have = static_cast<uint32_t>(len - base < kPiece + kHalo ? len - base : kPiece + kHalo);
  for (uint32_t w = tid; w < (have + 15) / 16; w += kBlock)
    reinterpret_cast<uint4*>(s_text)[w] = reinterpret_cast<const uint4*>(text + base)[w];
  __syncthreads();
  // newlines of the thread's 64 bytes, and of the bytes after the piece none
  const uint32_t mine0 = tid * 64;
  const uint64_t nl = classify(s_text, tid, have, s_map);
  if (tid < kHalo / 64) (void)classify(s_text, kBlock + tid, have, s_map);
  const uint32_t piece = have < kPiece ? have : kPiece;
  uint32_t total;
  const uint32_t ahead = block_excl_scan<kBlock>(static_cast<uint32_t>(__popcll(nl)), total, s_scan);
  if (tid < 32) {
    const uint64_t p = warp_lookback(status, s_tile, total, err);
    if (tid == 0) {
      s_b = p;
      if (base + kPiece >= len) fl->newlines = p + total;
    }
  }
  __syncthreads();
  // line k (from 0) of the piece starts after its newline k - 1; the text's
  // first line counts as one more of piece 0
  const uint32_t own0 = base == 0 ? 1u : 0u;
  const uint64_t line0 = s_b + (base == 0 ? 0 : 1);   // number of the piece's line 0
  const uint32_t n_lines = total + own0;
  for (uint32_t from = 0; from < n_lines; from += kLineList) {
    // list entries [from, from + kLineList] (one more: the end of the last)
    __syncthreads();
    if (own0 && from == 0 && tid == 0) s_start[0] = 0;
    {
      uint64_t m = nl;
      uint32_t k = ahead + own0;
      while (m) {
        const uint32_t q = __ffsll(static_cast<long long>(m)) - 1;
        if (k >= from && k <= from + kLineList) s_start[k - from] = static_cast<uint16_t>(mine0 + q + 1);
        m &= m - 1;
        ++k;
      }
    }
    for (uint32_t k0 = 0; k0 < kLineList && from + k0 < n_lines; k0 += kBlock) {
      __syncthreads();   // the list is complete; the last round's terms are looked up
      const uint32_t k = k0 + tid;
      const uint64_t line = line0 + from + k;
      const bool own = from + k < n_lines && base + s_start[k] < len && line < rows;
      uint32_t o4[3] = {0, 0, 0}, l4[3] = {0, 0, 0};
      bool lit = false;
      int got = 0;
      if (own) {   // (the text's last newline starts no line)
        const uint32_t b = s_start[k];
        uint32_t e;
        bool near = true;
        if (from + k + 1 < n_lines) {
          e = s_start[k + 1] - 1u;
        } else {
          e = piece > b ? piece : b;
          while (e < have && s_text[e] != '\n') ++e;
          near = e < have || base + have == len;   // the line ends within shared memory
        }
        if (near) {
          got = mapped_parse_line(s_text, s_map, b, e, o4, l4, lit);
          if (sp.lit) {
            for (int q = 0; q < 3; ++q) {
              sp.off[q][line] = base + o4[q];
              sp.len[q][line] = got == 1 ? l4[q] : 0;
            }
            sp.lit[line] = lit ? 1 : 0;
          }
          if (got == 2) atomicMin(&fl->bad_line, static_cast<unsigned long long>(line + 1));
          if (got != 1 && slots) slots[line] = kNoSlot;
        } else if (far) {
          far[atomicAdd(&fl->far, 1u)] = {line, base + b};
        } else {
          parse_far_line(text, len, base + b, line, rows, tb, slots, sp, literal_dict, fl);
        }
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) s_term[q][tid] = got == 1 ? (l4[q] << 16 | o4[q]) : 0u;
      s_lit[tid] = lit ? 1 : 0;
      __syncthreads();
      if (!slots) continue;
      const uint32_t here = n_lines - from - k0 < kBlock ? n_lines - from - k0 : kBlock;
      for (uint32_t x = tid; x < 3 * here; x += kBlock) {
        const uint32_t q = x / here, r = x - q * here, w = s_term[q][r];
        if (w == 0) continue;
        const uint64_t l = line0 + from + k0 + r;
        const uint32_t off = w & 0xffffu;
        const uint32_t dict = q == 1 ? 1u : (q == 2 && s_lit[r] && literal_dict ? 2u : 0u);
        slots[q * rows + l] =
            find_slot(tb, text, s_text, off, base + off, w >> 16, dict, static_cast<uint32_t>(l), fl);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// 3. ids: per line, whether it holds a statement and which of its terms occur
// on it first (a subject before an equal object), scanned over the lines.
struct Counts {
  uint64_t n[4];                 // statements, terms of dictionaries 0, 1, 2
  unsigned long long bytes[3];   // those terms' text, a NUL after each
};

struct LineFirsts {
  bool statement, s, p, o;
  uint32_t o_dict;
};
__device__ __forceinline__ LineFirsts line_firsts(const uint32_t* __restrict__ slots, const Slot* __restrict__ table,
                                                  uint64_t rows, uint64_t lines, uint64_t line, uint32_t (&sl)[3]) {
  LineFirsts f{false, false, false, false, 0};
  sl[0] = line < lines ? slots[line] : kNoSlot;
  if (sl[0] == kNoSlot) return f;
  sl[1] = slots[rows + line];
  sl[2] = slots[2 * rows + line];
  const uint32_t l = ~static_cast<uint32_t>(line);
  const Slot o = table[sl[2]];
  f.statement = true;
  f.s = table[sl[0]].first == l;
  f.p = table[sl[1]].first == l;
  f.o = o.first == l && sl[2] != sl[0];
  f.o_dict = static_cast<uint32_t>(o.loc & 3);
  return f;
}

// base3: the first id of each dictionary.
__global__ void __launch_bounds__(kBlock) ids_kernel(const uint32_t* __restrict__ slots, Slot* table, uint64_t rows,
                                                     uint64_t lines, uint64_t tiles, uint32_t len_bits, uint3 base3, uint64_t* status, uint32_t* ticket,
                                                     uint64_t* __restrict__ tile_first, Counts* counts,
                                                     DeviceErrors* err) {
  __shared__ uint32_t s_scan[kBlock / 32 + 1];
  __shared__ uint64_t s_b[4];
  __shared__ uint32_t s_tile;
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint64_t l0 = static_cast<uint64_t>(tile) * kTileLines + static_cast<uint64_t>(threadIdx.x) * kRows;
  LineFirsts f[kRows];
  uint32_t sl[kRows][3];
  uint32_t c[4] = {0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    f[i] = line_firsts(slots, table, rows, lines, l0 + i, sl[i]);
    c[0] += f[i].statement;
    c[1] += f[i].s + (f[i].o && f[i].o_dict == 0);
    c[2] += f[i].p;
    c[3] += f[i].o && f[i].o_dict == 2;
  }
  uint32_t e[4], tot[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) e[q] = block_excl_scan<kBlock>(c[q], tot[q], s_scan);
  const uint32_t warp = threadIdx.x >> 5;
  if (warp < 4) {
    const uint64_t p = warp_lookback(status + warp * tiles, tile, warp == 0 ? tot[0] : warp == 1 ? tot[1] : warp == 2 ? tot[2] : tot[3], err);
    if ((threadIdx.x & 31) == 0) s_b[warp] = p;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    tile_first[tile] = s_b[0];
    if (tile == tiles - 1)
      for (int q = 0; q < 4; ++q) counts->n[q] = s_b[q] + tot[q];
  }
  const uint64_t len_mask = (1ull << len_bits) - 1;
  uint64_t bytes[3] = {0, 0, 0};
  auto text_of = [&](uint32_t slot) { return (table[slot].loc >> 2 & len_mask) + 1; };
  uint32_t id[3] = {base3.x + static_cast<uint32_t>(s_b[1] + e[1]), base3.y + static_cast<uint32_t>(s_b[2] + e[2]),
                    base3.z + static_cast<uint32_t>(s_b[3] + e[3])};
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    if (f[i].s) {
      table[sl[i][0]].id = id[0]++;
      bytes[0] += text_of(sl[i][0]);
    }
    if (f[i].o) {
      const int k = f[i].o_dict == 0 ? 0 : 2;
      table[sl[i][2]].id = k == 0 ? id[0]++ : id[2]++;
      (k == 0 ? bytes[0] : bytes[2]) += text_of(sl[i][2]);
    }
    if (f[i].p) {
      table[sl[i][1]].id = id[1]++;
      bytes[1] += text_of(sl[i][1]);
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const uint64_t b = warp_sum64(bytes[k]);
    if (lane_id() == 0 && b) atomicAdd(&counts->bytes[k], static_cast<unsigned long long>(b));
  }
}

// 4. ids to the columns, and the places of the terms in id order.
struct TermList {
  uint64_t* loc[3];   // per dictionary: offset << len_bits | length, by id - base
};
__global__ void __launch_bounds__(kBlock) columns_kernel(const uint32_t* __restrict__ slots,
                                                         const Slot* __restrict__ table, uint64_t rows, uint64_t lines,
                                                         uint3 base3,
                                                         const uint64_t* __restrict__ tile_first,
                                                         uint32_t* __restrict__ s, uint32_t* __restrict__ p,
                                                         uint32_t* __restrict__ o, TermList terms) {
  __shared__ uint32_t s_scan[kBlock / 32 + 1];
  const uint64_t l0 = static_cast<uint64_t>(blockIdx.x) * kTileLines + static_cast<uint64_t>(threadIdx.x) * kRows;
  uint32_t c = 0;
#pragma unroll
  for (int i = 0; i < kRows; ++i) c += l0 + i < lines && slots[l0 + i] != kNoSlot;
  uint32_t tot;
  uint64_t t = tile_first[blockIdx.x] + block_excl_scan<kBlock>(c, tot, s_scan);
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    uint32_t sl[3];
    const LineFirsts f = line_firsts(slots, table, rows, lines, l0 + i, sl);
    if (!f.statement) continue;
    const Slot a = table[sl[0]], b = table[sl[1]], d = table[sl[2]];
    s[t] = a.id;
    p[t] = b.id;
    o[t] = d.id;
    ++t;
    if (f.s) terms.loc[0][a.id - base3.x] = a.loc >> 2;
    if (f.p) terms.loc[1][b.id - base3.y] = b.loc >> 2;
    if (f.o) {
      if (f.o_dict == 0) terms.loc[0][d.id - base3.x] = d.loc >> 2;
      else terms.loc[2][d.id - base3.z] = d.loc >> 2;
    }
  }
}

// The terms' places in one text of all of them (at[i]; at[terms] its length):
// a scan of their lengths, a NUL after each.
__global__ void __launch_bounds__(kBlock) term_places_kernel(const uint64_t* __restrict__ loc, uint64_t terms,
                                                             uint32_t len_bits, uint64_t* __restrict__ at,
                                                             uint64_t* status, uint32_t* ticket, DeviceErrors* err) {
  __shared__ uint64_t s_scan[kBlock / 32 + 1];
  __shared__ uint64_t s_b;
  __shared__ uint32_t s_tile;
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
  __syncthreads();
  const uint64_t r0 = static_cast<uint64_t>(s_tile) * kTileLines + static_cast<uint64_t>(threadIdx.x) * kRows;
  const uint64_t mask = (1ull << len_bits) - 1;
  uint64_t v[kRows], sum = 0;
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    v[i] = r0 + i < terms ? (loc[r0 + i] & mask) + 1 : 0;
    sum += v[i];
  }
  uint64_t tot;
  const uint64_t e = block_excl_scan64<kBlock>(sum, tot, s_scan);
  uint64_t run = block_lookback(status, s_tile, tot, err, &s_b) + e;
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    if (r0 + i <= terms) at[r0 + i] = run;
    run += v[i];
  }
}

// The text of terms [i0, i1), one warp each, to out (term i0 at its start).
// The host's own copy of the text is larger than its caches: collecting the
// terms there took 0.8 ms for 22,000 of them.
__global__ void __launch_bounds__(kBlock) term_texts_kernel(const uint8_t* __restrict__ text,
                                                            const uint64_t* __restrict__ loc,
                                                            const uint64_t* __restrict__ at, uint64_t i0, uint64_t i1,
                                                            uint32_t len_bits, uint8_t* __restrict__ out) {
  const uint64_t nw = static_cast<uint64_t>(gridDim.x) * (kBlock / 32);
  const uint64_t start = at[i0];
  for (uint64_t i = i0 + static_cast<uint64_t>(blockIdx.x) * (kBlock / 32) + (threadIdx.x >> 5); i < i1; i += nw) {
    const uint64_t l = loc[i], len = l & ((1ull << len_bits) - 1);
    const uint8_t* src = text + (l >> len_bits);
    uint8_t* dst = out + (at[i] - start);
    for (uint64_t k = lane_id(); k <= len; k += 32) dst[k] = k < len ? src[k] : 0;
  }
}

unsigned grid(const Ctx& ctx, uint64_t units) {
  uint64_t g = div_up(units, static_cast<uint64_t>(kBlock));
  const uint64_t gmax = static_cast<uint64_t>(ctx.num_sms) * 16;
  if (g > gmax) g = gmax;
  return static_cast<unsigned>(g < 1 ? 1 : g);
}

// The text's way to the device, a part at a time, on a stream of its own: a
// part is parsed while the next one is copied.
class TextUpload {
 public:
  TextUpload(Ctx& ctx, const char* text, uint8_t* dev, uint64_t len)
      : ctx_(ctx), text_(text), dev_(dev), len_(len),
        part_(std::min<uint64_t>(std::max<uint64_t>(div_up(len, 4), kUploadLeast), kUploadMost)) {
    s_ = ctx.dl_stream();
    ev_ = ctx.take_event();
    // (the block may have been another's on the context's stream)
    VG_CUDA(cudaEventRecord(ev_, ctx.stream));
    VG_CUDA(cudaStreamWaitEvent(s_, ev_, 0));
  }
  TextUpload(const TextUpload&) = delete;
  TextUpload& operator=(const TextUpload&) = delete;
  ~TextUpload() {   // (the text's block goes back by the context's stream)
    cudaStreamSynchronize(s_);
    std::lock_guard<std::recursive_mutex> lk(ctx_.host_mu);
    ctx_.event_pool.push_back(ev_);
  }
  // Copies the next part; what follows on the context's stream finds the first
  // next() bytes of the text.
  uint64_t next() {
    const uint64_t n = std::min<uint64_t>(part_, len_ - at_);
    if (n) {
      VG_CUDA(cudaMemcpyAsync(dev_ + at_, text_ + at_, n, cudaMemcpyHostToDevice, s_));
      VG_CUDA(cudaEventRecord(ev_, s_));
      VG_CUDA(cudaStreamWaitEvent(ctx_.stream, ev_, 0));
    }
    return at_ += n;
  }

 private:
  Ctx& ctx_;
  const char* text_;
  uint8_t* dev_;
  uint64_t len_, part_, at_ = 0;
  cudaStream_t s_;
  cudaEvent_t ev_;
};

// Runs parse_kernel over the text (up given: as it arrives) into arrays of
// `rows` lines; false when it gave up (nothing but `newlines` is of use then,
// nor where there are more lines than rows).
bool parse(Ctx& ctx, const uint8_t* dtext, uint64_t len, uint64_t rows, const Table& tb, uint32_t* slots,
           const Spans& sp, bool literal_dict, TextUpload* up, uint64_t* newlines) {
  const uint64_t tiles = div_up(len, static_cast<uint64_t>(kPiece));
  Scratch<uint64_t> z(ctx, tiles + 1);   // look-back words, then the ticket
  Scratch<Flags> flags(ctx, 1);
  std::optional<Scratch<FarLine>> far;
  if (up) far.emplace(ctx, tiles);
  VG_CUDA(cudaMemsetAsync(z.get(), 0, (tiles + 1) * sizeof(uint64_t), ctx.stream));
  VG_CUDA(cudaMemsetAsync(flags.get(), 0, sizeof(Flags), ctx.stream));
  VG_CUDA(cudaMemsetAsync(&flags.get()->bad_line, 0xFF, sizeof(unsigned long long), ctx.stream));
  for (uint64_t done = 0; done < tiles;) {
    const uint64_t have = up ? up->next() : len;
    const uint64_t to = have == len ? tiles : have < kPiece + kHalo ? 0 : (have - kHalo) / kPiece;
    if (to <= done) continue;
    ctx.launch("ingest_parse", static_cast<double>(len) / tiles * (to - done) + 12.0 * rows * (to - done) / tiles, [&] {
      parse_kernel<<<static_cast<unsigned>(to - done), kBlock, 0, ctx.stream>>>(
          dtext, len, rows, tb, slots, sp, literal_dict, z.get(), reinterpret_cast<uint32_t*>(z.get() + tiles),
          far ? far->get() : nullptr, flags.get(), ctx.d_err);
    });
    VG_CUDA(cudaGetLastError());
    done = to;
  }
  if (far) {
    ctx.launch("ingest_far", 0.0, [&] {
      far_lines_kernel<<<grid(ctx, tiles), kBlock, 0, ctx.stream>>>(dtext, len, rows, tb, slots, literal_dict, far->get(),
                                                                    flags.get());
    });
    VG_CUDA(cudaGetLastError());
  }
  VG_CUDA(cudaMemcpyAsync(ctx.h_small, flags.get(), sizeof(Flags), cudaMemcpyDeviceToHost, ctx.stream));
  ctx.sync();
  Flags h;
  std::memcpy(&h, ctx.h_small, sizeof(h));
  ctx.check_device_errors();
  *newlines = h.newlines;
  if (h.bad_line != ~0ull)
    fail(VG_ERR_PARSE, "malformed N-Triples statement on line " + std::to_string(h.bad_line));
  return h.give_up == 0;
}

void check_ids(const uint64_t (&terms)[3], const uint32_t (&base)[3]) {
  for (int k = 0; k < 3; ++k)
    if (base[k] + terms[k] > 0xFFFFFFFFull) fail(VG_ERR_OVERFLOW, "dictionary ids exceed 32 bits");
}

// Steps 2 to 4: out.n and the columns, the counts, and the terms' places in id
// order (none without statements); false when the table gave up or (up given)
// the text has more than `rows` lines.  `lines` is set by then.
bool ids_and_columns(Ctx& ctx, const uint8_t* dtext, uint64_t len, bool open_end, uint64_t rows, uint32_t len_bits,
                     bool literal_dict, TextUpload* up, uint64_t& lines, Ingested& out, Counts& h,
                     std::optional<Scratch<uint64_t>>& loc) {
  Table tb{};
  tb.len_bits = len_bits;
  tb.cap = std::min<uint64_t>(4 * rows + 64, 0xFFFFFFFFull);
  tb.hash_bits = g_hash_bits.load();
  Scratch<Slot> table(ctx, tb.cap);
  tb.slots = table.get();
  VG_CUDA(cudaMemsetAsync(tb.slots, 0, tb.cap * sizeof(Slot), ctx.stream));
  Scratch<uint32_t> slots(ctx, 3 * rows);
  uint64_t newlines = 0;
  const bool took = parse(ctx, dtext, len, rows, tb, slots.get(), Spans{}, literal_dict, up, &newlines);
  lines = newlines + (open_end ? 1 : 0);
  if (!took || lines > rows) return false;
  // 3. ids
  const uint32_t base[3] = {1u, 1u, kLiteralStartId};
  const uint3 base3 = make_uint3(base[0], base[1], base[2]);
  const uint64_t tiles = div_up(lines, kTileLines);
  const size_t words = 4 * tiles + sizeof(Counts) / 8 + 1;   // look-back words, counts, ticket
  Scratch<uint64_t> z(ctx, words), first(ctx, tiles);
  VG_CUDA(cudaMemsetAsync(z.get(), 0, words * sizeof(uint64_t), ctx.stream));
  auto* counts = reinterpret_cast<Counts*>(z.get() + 4 * tiles);
  ctx.launch("ingest_ids", 12.0 * lines, [&] {
    ids_kernel<<<static_cast<unsigned>(tiles), kBlock, 0, ctx.stream>>>(
        slots.get(), tb.slots, rows, lines, tiles, len_bits, base3, z.get(), reinterpret_cast<uint32_t*>(counts + 1),
        first.get(), counts, ctx.d_err);
  });
  VG_CUDA(cudaGetLastError());
  VG_CUDA(cudaMemcpyAsync(ctx.h_small, counts, sizeof(Counts), cudaMemcpyDeviceToHost, ctx.stream));
  ctx.sync();
  std::memcpy(&h, ctx.h_small, sizeof(h));
  ctx.check_device_errors();
  if (h.n[0] > 0x7FFFFFFFull) fail(VG_ERR_OVERFLOW, "ingest is limited to 2^31 triples");
  const uint64_t nterms[3] = {h.n[1], h.n[2], h.n[3]};
  check_ids(nterms, base);
  // 4. columns
  out.n = h.n[0];
  out.s = ctx.alloc<uint32_t>(out.n);
  out.p = ctx.alloc<uint32_t>(out.n);
  out.o = ctx.alloc<uint32_t>(out.n);
  if (out.n == 0) return true;
  loc.emplace(ctx, nterms[0] + nterms[1] + nterms[2]);
  uint64_t* l = loc->get();
  const TermList tl{{l, l + nterms[0], l + nterms[0] + nterms[1]}};
  ctx.launch("ingest_scatter", 24.0 * lines, [&] {
    columns_kernel<<<static_cast<unsigned>(tiles), kBlock, 0, ctx.stream>>>(slots.get(), tb.slots, rows, lines, base3,
                                                                           first.get(), out.s, out.p, out.o, tl);
  });
  VG_CUDA(cudaGetLastError());
  return true;
}

// The dictionaries' terms: places by a scan, texts collected on the device
// (at most kTextChunk bytes at a time, or one term) and copied to the host.
void term_texts(Ctx& ctx, const uint8_t* dtext, uint32_t len_bits, const uint64_t* loc, const Counts& h, Dict& dict) {
  constexpr uint64_t kTextChunk = 64ull << 20;
  const uint64_t all = h.n[1] + h.n[2] + h.n[3], bytes = h.bytes[0] + h.bytes[1] + h.bytes[2];
  const uint64_t tiles = div_up(all + 1, kTileLines);
  Scratch<uint64_t> at(ctx, all + 1), z(ctx, tiles + 1);   // z: look-back words, ticket
  VG_CUDA(cudaMemsetAsync(z.get(), 0, (tiles + 1) * sizeof(uint64_t), ctx.stream));
  ctx.launch("ingest_terms", 16.0 * all, [&] {
    term_places_kernel<<<static_cast<unsigned>(tiles), kBlock, 0, ctx.stream>>>(
        loc, all, len_bits, at.get(), z.get(), reinterpret_cast<uint32_t*>(z.get() + tiles), ctx.d_err);
  });
  VG_CUDA(cudaGetLastError());
  auto collect = [&](uint64_t i0, uint64_t i1, uint8_t* out) {
    ctx.launch("ingest_terms", static_cast<double>(bytes), [&] {
      term_texts_kernel<<<grid(ctx, 32 * (i1 - i0)), kBlock, 0, ctx.stream>>>(dtext, loc, at.get(), i0, i1, len_bits,
                                                                             out);
    });
    VG_CUDA(cudaGetLastError());
  };
  TermTexts* terms[3] = {&dict.so, &dict.p, &dict.l};
  char* text[3];
  uint64_t *host_at[3], first = 0;
  for (int k = 0; k < 3; ++k) {
    text[k] = terms[k]->fill(h.n[1 + k], h.bytes[k], &host_at[k]);
    // the next dictionary's first place comes along as this one's end
    VG_CUDA(cudaMemcpyAsync(host_at[k], at.get() + first, (h.n[1 + k] + 1) * sizeof(uint64_t), cudaMemcpyDeviceToHost,
                            ctx.stream));
    first += h.n[1 + k];
  }
  if (bytes <= kTextChunk) {
    Scratch<uint8_t> buf(ctx, bytes);
    if (all) collect(0, all, buf.get());
    uint64_t off = 0;
    for (int k = 0; k < 3; ++k) {
      if (h.bytes[k])
        VG_CUDA(cudaMemcpyAsync(text[k], buf.get() + off, h.bytes[k], cudaMemcpyDeviceToHost, ctx.stream));
      off += h.bytes[k];
    }
    ctx.sync();
  } else {
    ctx.sync();
    first = 0;
    for (int k = 0; k < 3; ++k) {
      const uint64_t n = h.n[1 + k], *a = host_at[k];
      for (uint64_t i = 0; i < n;) {
        uint64_t e = i + 1;   // the first term past the chunk
        e = std::max<uint64_t>(e, std::upper_bound(a + i, a + n + 1, a[i] + kTextChunk) - a - 1);
        Scratch<uint8_t> buf(ctx, a[e] - a[i]);
        collect(first + i, first + e, buf.get());
        VG_CUDA(cudaMemcpyAsync(text[k] + (a[i] - a[0]), buf.get(), a[e] - a[i], cudaMemcpyDeviceToHost, ctx.stream));
        ctx.sync();
        i = e;
      }
      first += n;
    }
  }
  for (int k = 0; k < 3; ++k) {
    const uint64_t a0 = host_at[k][0];
    for (uint64_t i = 0; i <= h.n[1 + k]; ++i) host_at[k][i] -= a0;
  }
  ctx.check_device_errors();
}

// First-appearance ids on the host, for texts that the table cannot take (a
// term too long for a slot's word, 2^32 lines or more, or a hash that fails
// on the text): the statement handler's own rule, src/loader.cu:19-53.
void ingest_on_host(Ctx& ctx, const char* text, uint64_t len, const uint8_t* dtext, uint64_t lines,
                    bool literal_dict, Ingested& out) {
  Scratch<uint64_t> so(ctx, 3 * lines), sl(ctx, 3 * lines);
  Scratch<uint8_t> lit(ctx, lines);
  Spans sp{};
  for (int q = 0; q < 3; ++q) {
    sp.off[q] = so.get() + q * lines;
    sp.len[q] = sl.get() + q * lines;
  }
  sp.lit = lit.get();
  uint64_t newlines;
  parse(ctx, dtext, len, lines, Table{}, nullptr, sp, literal_dict, nullptr, &newlines);
  std::vector<uint64_t> off(3 * lines), ln(3 * lines);
  std::vector<uint8_t> hl(lines);
  VG_CUDA(cudaMemcpyAsync(off.data(), so.get(), 3 * lines * sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx.stream));
  VG_CUDA(cudaMemcpyAsync(ln.data(), sl.get(), 3 * lines * sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx.stream));
  VG_CUDA(cudaMemcpyAsync(hl.data(), lit.get(), lines, cudaMemcpyDeviceToHost, ctx.stream));
  ctx.sync();
  TermTexts* terms[3] = {&out.dict.so, &out.dict.p, &out.dict.l};
  const uint32_t base[3] = {1u, 1u, kLiteralStartId};
  std::unordered_map<std::string_view, uint32_t> ids[3];
  std::vector<uint32_t> col[3];
  for (uint64_t i = 0; i < lines; ++i) {
    if (ln[i] == 0) continue;
    for (int q : {0, 2, 1}) {   // subject, object, predicate
      const int k = q == 1 ? 1 : (q == 2 && literal_dict && hl[i] ? 2 : 0);
      const std::string_view v(text + off[q * lines + i], ln[q * lines + i]);
      auto it = ids[k].find(v);
      if (it == ids[k].end()) {
        it = ids[k].emplace(v, base[k] + static_cast<uint32_t>(terms[k]->size())).first;
        terms[k]->push_back(v);
      }
      col[q].push_back(it->second);
    }
  }
  out.n = col[0].size();
  if (out.n > 0x7FFFFFFFull) fail(VG_ERR_OVERFLOW, "ingest is limited to 2^31 triples");
  const uint64_t sizes[3] = {out.dict.so.size(), out.dict.p.size(), out.dict.l.size()};
  check_ids(sizes, base);
  uint32_t** dst[3] = {&out.s, &out.p, &out.o};
  for (int q = 0; q < 3; ++q) {
    *dst[q] = ctx.alloc<uint32_t>(out.n);
    if (out.n)
      VG_CUDA(cudaMemcpyAsync(*dst[q], col[q].data(), out.n * 4, cudaMemcpyHostToDevice, ctx.stream));
  }
  ctx.sync();
}

}  // namespace

void set_ingest_hash_bits(int bits) { g_hash_bits.store(bits < 1 ? 1 : (bits > 63 ? 63 : bits)); }

void TermTexts::push_back(std::string_view v) {
  const size_t end = at_.back(), need = end + v.size() + 1;
  if (need > cap_) {
    const size_t cap = std::max<size_t>(2 * cap_, need + 64);
    std::unique_ptr<char[]> grown(new char[cap]);
    if (end) std::memcpy(grown.get(), text_.get(), end);
    text_ = std::move(grown);
    cap_ = cap;
  }
  std::memcpy(text_.get() + end, v.data(), v.size());
  text_[end + v.size()] = 0;
  at_.push_back(need);
}

char* TermTexts::fill(size_t count, size_t bytes, uint64_t** at) {
  text_.reset(new char[bytes ? bytes : 1]);
  cap_ = bytes;
  at_.assign(count + 1, 0);
  *at = at_.data();
  return text_.get();
}

bool Dict::has(int kind, uint32_t id, size_t* at) const {
  const uint32_t base = kind == 2 ? kLiteralStartId : 1u;
  if (id < base || id - base >= terms(kind).size()) return false;
  *at = id - base;
  return true;
}

uint32_t Dict::lookup(int kind, const std::string& t) {
  if (kind < 0 || kind > 2) return 0;
  auto& rev = rev_[kind];
  const TermTexts& v = terms(kind);
  const uint32_t base = kind == 2 ? kLiteralStartId : 1u;
  if (rev.size() != v.size()) {
    rev.clear();
    rev.reserve(v.size());
    for (size_t i = 0; i < v.size(); ++i) rev.emplace(v[i], base + static_cast<uint32_t>(i));
  }
  auto it = rev.find(t);
  return it == rev.end() ? 0 : it->second;
}

// Lines that a long text is taken to have at most, before it has been read: a
// quarter more than 32 samples of it promise.
static uint64_t lines_guess(const char* text, uint64_t len) {
  constexpr uint64_t kSamples = 32, kBytes = 4096;
  uint64_t n = 0;
  for (uint64_t k = 0; k < kSamples; ++k) {
    const char* at = text + (len - kBytes) / (kSamples - 1) * k;
    n += static_cast<uint64_t>(std::count(at, at + kBytes, '\n'));
  }
  return static_cast<uint64_t>(static_cast<double>(n) / (kSamples * kBytes) * 1.25 * static_cast<double>(len)) + 4096;
}

void ingest_ntriples(Ctx& ctx, const char* text, uint64_t len, bool literal_dict, Ingested& out) {
  out = Ingested();
  out.dict.literal_dict = literal_dict;
  if (len == 0) return;
  if (div_up(len, static_cast<uint64_t>(kPiece)) > 0x7FFFFFFFull) fail(VG_ERR_OVERFLOW, "ingest text too long");
  // the text, padded to whole 16-byte words
  Scratch<uint8_t> dtext(ctx, div_up(len, 16) * 16);
  const bool open_end = text[len - 1] != '\n';
  // Three terms a line, four slots of the table for every three of them (2^32
  // slots at most).
  int off_bits = 1;
  while (len >> off_bits) ++off_bits;
  const uint32_t len_bits = static_cast<uint32_t>(62 - off_bits < off_bits ? 62 - off_bits : off_bits);
  std::optional<Scratch<uint64_t>> loc;   // the terms' places in the text, in id order
  Counts h{};
  bool done = false, counted = false, copied = false;
  uint64_t lines = 0;
  // A text of several parts is parsed as it arrives, into room for a guess of
  // its lines, where the scratch holds that easily (slots and table take 76
  // bytes a line; columns, terms' places and texts follow).  For 101 MB the
  // copy takes 0.56 ms, and the lines' count (0.03) and parse (0.23) ran after it.
  const uint64_t rows = len > 2 * kUploadLeast ? lines_guess(text, len) : 0;
  if (rows && rows < 0xFFFFFFFFull && ctx.arena.largest_free() > 160 * rows + std::min<uint64_t>(len, 64ull << 20)) {
    TextUpload up(ctx, text, dtext.get(), len);
    done = ids_and_columns(ctx, dtext.get(), len, open_end, rows, len_bits, literal_dict, &up, lines, out, h, loc);
    counted = copied = true;
  }
  if (!copied) VG_CUDA(cudaMemcpyAsync(dtext.get(), text, len, cudaMemcpyHostToDevice, ctx.stream));
  if (!counted) {
    // 1. lines
    Scratch<unsigned long long> ncount(ctx, 1);
    VG_CUDA(cudaMemsetAsync(ncount.get(), 0, sizeof(unsigned long long), ctx.stream));
    ctx.launch("ingest_newlines", static_cast<double>(len), [&] {
      newline_count_kernel<<<grid(ctx, div_up(len, 64)), kBlock, 0, ctx.stream>>>(dtext.get(), len, ncount.get());
    });
    VG_CUDA(cudaGetLastError());
    VG_CUDA(cudaMemcpyAsync(ctx.h_small, ncount.get(), sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    lines = ctx.h_small[0] + (open_end ? 1 : 0);
  }
  // 2. statements and terms
  if (!done && lines < 0xFFFFFFFFull && (!counted || lines > rows))
    done = ids_and_columns(ctx, dtext.get(), len, open_end, lines, len_bits, literal_dict, nullptr, lines, out, h, loc);
  if (done && loc) term_texts(ctx, dtext.get(), len_bits, loc->get(), h, out.dict);
  if (!done) {
    ++out.collisions;
    ingest_on_host(ctx, text, len, dtext.get(), lines, literal_dict, out);
  }
  ctx.sync();
  ctx.check_device_errors();
}

DictResolver::DictResolver(const Dict* d) {
  for (int k = 0; k < 3; ++k) {
    const TermTexts& v = d->terms(k);
    const uint32_t base = k == 2 ? kLiteralStartId : 1u;
    rev_[k].reserve(v.size());
    for (size_t i = 0; i < v.size(); ++i) rev_[k].emplace(std::string(v[i]), base + static_cast<uint32_t>(i));
  }
}

vedas::TYPEID DictResolver::resolve(int pos, const std::string& term) const {
  int kind = pos == 1 ? 1 : 0;
  std::string key = term;
  if (pos == 2 && !term.empty() && term[0] == '"') {
    kind = 2;
    key = term.substr(0, term.find('"', 1) + 1);   // "text" without @lang / ^^<type>
  }
  auto it = rev_[kind].find(key);
  return it == rev_[kind].end() ? 0 : it->second;
}

std::string decode_rows(const Dict& d, const std::vector<const uint32_t*>& cols, uint64_t nrows) {
  // rows are decoded in parallel blocks, then joined
  constexpr uint64_t kRowsPerPart = 4096;
  const uint64_t parts = (nrows + kRowsPerPart - 1) / kRowsPerPart;
  std::vector<std::string> out(parts);
  parallel_for(parts, [&](size_t b) {
    std::string& o = out[b];
    const uint64_t r1 = std::min<uint64_t>(nrows, (b + 1) * kRowsPerPart);
    for (uint64_t r = b * kRowsPerPart; r < r1; ++r) {
      for (size_t c = 0; c < cols.size(); ++c) {
        if (c) o += '\t';
        const uint32_t id = cols[c][r];
        const int kind = d.literal_dict && id >= kLiteralStartId ? 2 : 0;
        size_t at;
        if (d.has(kind, id, &at)) o += d.terms(kind)[at];
        else o += "?" + std::to_string(id);
      }
      o += '\n';
    }
  });
  size_t total = 0;
  for (const auto& x : out) total += x.size();
  std::string all;
  all.reserve(total);
  for (const auto& x : out) all += x;
  return all;
}

void write_vdd(const Dict& d, const char* path) {
  std::ofstream out(path);
  if (!out) fail(VG_ERR_INVALID, std::string("cannot write ") + path);
  auto section = [&](const TermTexts& v, uint32_t base) {
    out << v.size() << "\n";
    for (size_t i = 0; i < v.size(); ++i) out << (base + i) << " " << v[i] << "\n";
  };
  section(d.so, 1u);
  section(d.p, 1u);
  section(d.l, kLiteralStartId);
  if (!out) fail(VG_ERR_INVALID, std::string("write failed: ") + path);
}

void read_vdd(const char* path, Dict& d) {
  std::ifstream in(path);
  if (!in) fail(VG_ERR_INVALID, std::string("cannot open ") + path);
  d = Dict();
  auto section = [&](TermTexts& v, uint32_t base) {
    std::string line;
    if (!std::getline(in, line)) fail(VG_ERR_INVALID, "truncated .vdd");
    const uint64_t count = std::stoull(line);
    // entries may come in any order (the reference writes hash-map order); their
    // texts lie in one block until then (400,000 terms: 74 ms with a string each
    // to be copied and freed, 55 so)
    struct Entry {
      uint32_t id;
      size_t at, len;
    };
    std::vector<Entry> e;
    e.reserve(count);
    std::string text;
    for (uint64_t i = 0; i < count; ++i) {
      if (!std::getline(in, line)) fail(VG_ERR_INVALID, "truncated .vdd");
      const size_t sp = line.find(' ');
      if (sp == std::string::npos) fail(VG_ERR_INVALID, "malformed .vdd line");
      e.push_back({static_cast<uint32_t>(std::stoul(line.substr(0, sp))), text.size(), line.size() - sp - 1});
      text.append(line, sp + 1, std::string::npos);
    }
    std::sort(e.begin(), e.end(), [](const Entry& a, const Entry& b) { return a.id < b.id; });
    for (size_t i = 0; i < e.size(); ++i)
      if (e[i].id != base + i) fail(VG_ERR_INVALID, ".vdd ids are not dense");
    uint64_t* at;
    char* to = v.fill(e.size(), text.size() + e.size(), &at);
    size_t end = 0;
    for (size_t i = 0; i < e.size(); ++i) {
      at[i] = end;
      std::memcpy(to + end, text.data() + e[i].at, e[i].len);
      to[end + e[i].len] = 0;
      end += e[i].len + 1;
    }
    at[e.size()] = end;
  };
  section(d.so, 1u);
  section(d.p, 1u);
  section(d.l, kLiteralStartId);
  d.literal_dict = d.l.size() > 0;
}

}  // namespace vg
