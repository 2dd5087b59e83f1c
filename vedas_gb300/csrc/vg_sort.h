#pragma once

#include <vector>

#include "vg_ctx.h"

namespace vg {

// One radix pass: the digit (key >> shift) & (2^bits - 1), bits <= 8.
struct RadixDigit {
  uint32_t shift;
  uint32_t bits;
};
// Appends the digits that cover key bits [begin, end) from the lowest up, as
// few as 8-bit digits allow and of widths as equal as can be.
void radix_plan(std::vector<RadixDigit>& digits, int begin, int end);

constexpr int kRadixMaxPasses = 20;

// Stable LSD radix sort of n keys over bits [0, end_bit).  When `vals` is
// non-null the uint32 values move with their keys; with vals_iota the values
// are generated as 0..n-1 (the input value buffer is not read).  Double
// buffered: returns true when the result is in (keys_alt, vals_alt).  The host
// waits once, for the digits that are the same for every key: their passes are
// skipped.
bool radix_sort_u32(Ctx& ctx, uint32_t* keys, uint32_t* keys_alt, uint32_t* vals, uint32_t* vals_alt,
                    uint64_t n, int end_bit, bool vals_iota);
bool radix_sort_u64(Ctx& ctx, uint64_t* keys, uint64_t* keys_alt, uint64_t n, int end_bit);
// By the given digits in order (what lies outside them travels with the key
// and does not count: equal digits keep their input order), with the bases of
// each digit's 256 values already on the device.  Counts do not depend on the
// keys' order, so one count serves several sorts.  Nothing is waited for.
bool radix_sort_u64_counted(Ctx& ctx, uint64_t* keys, uint64_t* keys_alt, uint32_t* vals, uint32_t* vals_alt,
                            uint64_t n, const std::vector<RadixDigit>& digits,
                            const std::vector<const uint64_t*>& bases, bool vals_iota = false);
void fill_iota(Ctx& ctx, uint32_t* out, uint64_t n);

}  // namespace vg
