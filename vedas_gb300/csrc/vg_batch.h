// Batched (multi-query) versions of the relation kernels: every call takes
// the work of many queries and issues a fixed, small number of launches.
//
// They only enqueue work on the context stream.  The values they hand back
// are stored by the kernels into page-locked host memory (the *_host
// arguments), valid once the stream has passed that point (the caller records
// an event).
#pragma once

#include <memory>
#include <vector>

#include "vg_relops.h"

namespace vg {

// Page-locked host words for device->host reads of one pipeline stage,
// taken from and returned to the context's pool of page-locked chunks.
class PinnedWords {
 public:
  explicit PinnedWords(Ctx& ctx) : ctx_(ctx) {}
  PinnedWords(const PinnedWords&) = delete;
  PinnedWords& operator=(const PinnedWords&) = delete;
  ~PinnedWords();
  // At least `words` 64-bit words; may switch buffers, so only call it while
  // no copy into the buffer is pending.
  uint64_t* reserve(size_t words);
  uint64_t* data() const { return p_; }

 private:
  Ctx& ctx_;
  uint64_t* p_ = nullptr;
  size_t cap_ = 0;   // bytes
};

// The calls of one pipeline stage whose tables go up in one copy: each call
// given the stage adds its tables and leaves its launches to run(), in the
// order of the calls.  What the calls were given must live until then.  (A
// copy, its event and the ring's bookkeeping for each call: 24 of them in a
// 64-query batch.)
class BatchStage {
 public:
  explicit BatchStage(Ctx& ctx);
  ~BatchStage();
  void run();
  struct Impl;
  Impl& impl() { return *impl_; }

 private:
  std::unique_ptr<Impl> impl_;
};

// All pieces in one launch (any number of pieces).
void batched_copy(Ctx& ctx, const std::vector<CopyPiece>& pieces, BatchStage* stage = nullptr);

// One relation segment: ncols columns of n rows, read from `in`, written to `out`.
struct SegRows {
  uint32_t ncols = 0;
  uint64_t n = 0;
  const uint32_t* in[VG_MAX_COLS] = {nullptr};
  uint32_t* out[VG_MAX_COLS] = {nullptr};
};

// Adjacent-unique compaction of every segment; each segment's kept row count
// goes to counts_host[s].
void batched_unique_enqueue(Ctx& ctx, const std::vector<SegRows>& segs, uint64_t* counts_host,
                            BatchStage* stage = nullptr);
// Adds the compaction's written bytes to the kernel statistics once the
// counts are known.
void note_unique_writes(Ctx& ctx, const std::vector<SegRows>& segs, const uint64_t* counts);

// Stable sort of every relation by its column 0: those of up to 1024 rows by
// one launch, the others by one radix sort over (segment, key) composite keys
// and one gather.  Columns are replaced.  key_bits (1..32) bounds every key
// (keys < 2^key_bits); 0: 32 bits.
void batched_sort_by_first(Ctx& ctx, const std::vector<Rel*>& rels, int key_bits);

// Inner joins on column 0 (l[j] with r[j], both sorted by column 0 and
// non-empty), in two halves.  batched_join_count enqueues the per-key match
// counts and their scan and copies each join's output size to
// totals_host[j]; batched_join_write, given those sizes, allocates the
// outputs from the arena, enqueues the output write, and stores column 0's
// first and last value of out[j] to first_last_host[2j], [2j+1] (zero for an
// empty output).  The relations must stay alive and unchanged in between.
struct JoinBatch {
  uint32_t J = 0;
  std::vector<const Rel*> l, r;
  std::vector<uint64_t> row0, base_at;   // offsets of each join's left rows and tiles in cnt's arrays
  JoinCounts<uint32_t> cnt{};
  uint64_t* d_totals = nullptr; // every join's output rows, on the device
  // Frees the arrays (in stream order).
  void release(Ctx& ctx);
};
void batched_join_count(Ctx& ctx, const std::vector<const Rel*>& l, const std::vector<const Rel*>& r, JoinBatch& jb,
                        uint64_t* totals_host);
// skip (optional, J flags): joins whose outputs are in out[] already; the
// others are allocated and written.  Releases jb's device arrays.
void batched_join_write(Ctx& ctx, JoinBatch& jb, const uint64_t* totals, std::vector<Rel>& out,
                        uint32_t* first_last_host, const uint8_t* skip = nullptr);

constexpr uint32_t kSmallC0Words = 100;   // staged column-0 words per small join output

// Count and write without a host round trip in between: the outputs are placed
// on the device in `region` (its bump pointer at d_bump) and written.  Outputs
// that do not fit stay unplaced.  jb's device arrays stay alive:
// place_outputs_on_host then tells which joins were placed (the same
// arithmetic on the copied totals), and the caller writes the others with
// batched_join_write(..., skip = placed), or releases jb.
struct PlacedHost {       // page-locked
  uint64_t* totals;       // every join's output rows
  uint64_t* bump;         // the region's bump pointer after the wave
  DeviceErrors* err;      // the error record after the count; nothing is placed when it holds a timeout
  uint32_t* first_last;   // of the placed outputs with rows
  uint32_t* c0;           // for joins with c0_slot[j] >= 0 and 2 < rows < kSmallC0Words: column 0 at slot * kSmallC0Words
};
void batched_join_placed(Ctx& ctx, const std::vector<const Rel*>& l, const std::vector<const Rel*>& r, JoinBatch& jb,
                         const Arena::Region* region, uint64_t* d_bump, const std::vector<int32_t>& c0_slot,
                         uint32_t nslots, const PlacedHost& host, BatchStage* stage = nullptr);
// Returns the region's bump after the wave; out[j] is the placed output of
// join j (placed[j] = 1) and `blocks` the number of its columns in the region.
uint64_t place_outputs_on_host(const JoinBatch& jb, const uint64_t* totals, const Arena::Region* region,
                               uint64_t bump, std::vector<Rel>& out, std::vector<uint8_t>& placed,
                               int64_t& blocks);

// Column 0 of each relation stored to the host, back to back (one launch):
// col0_words(rels) uint32 words.
uint64_t col0_words(const std::vector<const Rel*>& rels);
void batched_col0_enqueue(Ctx& ctx, const std::vector<const Rel*>& rels, uint32_t* host, BatchStage* stage = nullptr);

}  // namespace vg
