#pragma once

#include <vector>

#include "vg_ctx.h"

namespace vg {

// A device relation: ncols uint32 columns of nrows rows (column-major).
// Bit c of `borrowed` marks column c as a view into memory the relation does
// not own (a slice of an index array): it is never freed or written through
// the relation, and it may start at any 4-byte boundary.
struct Rel {
  uint32_t ncols = 0;
  uint64_t nrows = 0;
  uint32_t* cols[VG_MAX_COLS] = {nullptr};
  uint32_t borrowed = 0;
};

Rel rel_alloc(Ctx& ctx, uint32_t ncols, uint64_t nrows);
// Frees the owned columns.
void rel_free(Ctx& ctx, Rel& r);
// Frees column c if the relation owns it, and marks the slot owned (the
// caller stores an owned column there or drops it).
void rel_drop_col(Ctx& ctx, Rel& r, uint32_t c);
// Replaces every borrowed column by an owned copy (stream-ordered).
void rel_own(Ctx& ctx, Rel& r);

// One contiguous copy src[0, len) -> dst[0, len).
struct CopyPiece {
  const uint32_t* src;
  uint32_t* dst;
  uint64_t len;
};
// All pieces in one launch (up to 16).
void multi_copy(Ctx& ctx, const CopyPiece* pieces, int np);

// First and last value of a join's column 0 (when it has rows), and all of it
// when it has fewer than 100.
struct JoinEnds {
  uint32_t first = 0, last = 0;
  std::vector<uint32_t> c0;
};

// Sorted inner join of l and r on column 0 (two_keys: on columns 0 and 1).
// Output layout: key column(s), l's other columns, r's other columns; rows
// ordered by (left row, right row).  Allocates `out` from the arena, no more
// than its rows take; waits for the result and raises device errors.  True
// when a copy of the output to blocks of its size is still on the stream.
bool join(Ctx& ctx, const Rel& l, const Rel& r, bool two_keys, Rel& out, JoinEnds* ends = nullptr);

// What a join's count leaves in device memory.  Left rows come in groups of
// kJoinGroup (one thread's): match has a bit for each of a group's rows that has
// matches, and only groups with one have their rows' lower bounds (lo) and
// output offsets (offs) stored, a sector of 32 bytes each; start is the group's
// first output row, for the searches.  offs and start count from the tile's
// first output row, which is base[tile] (tiles of 2048 left rows).  The arrays
// cover whole groups; lo and offs start on 16 bytes.  (With an offset and a
// bound for every row instead, a wave of joins of which few left rows match
// moved twice the bytes.)
// Off: 32 bits hold every offset of a join that is written (one with 2^32 rows
// or more is refused, by its 64-bit total); 64 bits for the join that takes any.
constexpr int kJoinGroup = 8;
constexpr uint64_t kMaxJoinRows = 0xFFFFFFFFull;   // of an output with 32-bit offsets
template <typename Off>
struct JoinCounts {
  uint32_t* lo;
  Off* offs;
  Off* start;
  uint8_t* match;
  uint64_t* base;
};

// The same join on a caller's stream with caller-provided scratch (c) and
// output columns (nothing is allocated); done and err must be zero.  Returns
// the result row count; the outputs are written only when it fits `capacity`.
uint64_t join_into(cudaStream_t stream, const Rel& l, const Rel& r, uint32_t* const* out_cols, uint64_t capacity,
                   const JoinCounts<uint64_t>& c, uint32_t* done, uint64_t* total, DeviceErrors* err);

// out[c][i] = in[c][perm[i]] for every column.
void gather_cols(Ctx& ctx, const uint32_t* const* in, uint32_t* const* out, uint32_t ncols,
                 const uint32_t* perm, uint64_t n);

// Stable sort of the rows by column 0 (in place; columns are replaced).
void sort_by_first(Ctx& ctx, Rel& r);
// Lexicographic sort of the rows over all columns (in place); waits for the
// result and raises device errors.
void sort_rows(Ctx& ctx, Rel& r);
// Adjacent duplicate-row removal (synchronizes and raises device errors).  A
// relation without any keeps its columns; views stay views.  repeats: whether
// some are expected (for speed only).
void unique_in_place(Ctx& ctx, Rel& r, bool repeats);

// Copies `n` values of a device column to the host (synchronizes).
void download(Ctx& ctx, const uint32_t* dev, uint64_t n, uint32_t* host);

}  // namespace vg
