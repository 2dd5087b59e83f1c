// Host-side check of the placement of join outputs in a region (the arithmetic
// that the device uses too): for joins of one left and two right columns (two
// output columns) and the output row counts given as arguments, prints which
// are placed, the region's bump pointer afterwards and the placed columns'
// number.  The region's memory is never touched.
#include <cstdio>
#include <cstdlib>

#include "../vedas_gb300/csrc/vg_batch.h"

int main(int argc, char** argv) {
  vg::Arena::Region region;
  region.begin = reinterpret_cast<char*>(uintptr_t{1} << 20);
  region.bytes = std::strtoull(argv[1], nullptr, 10);
  std::vector<uint64_t> totals;
  for (int i = 2; i < argc; ++i) totals.push_back(std::strtoull(argv[i], nullptr, 10));
  vg::Rel l, r;
  l.ncols = 1;
  r.ncols = 2;
  vg::JoinBatch jb;
  jb.J = static_cast<uint32_t>(totals.size());
  jb.l.assign(jb.J, &l);
  jb.r.assign(jb.J, &r);
  std::vector<vg::Rel> out;
  std::vector<uint8_t> placed;
  int64_t blocks = 0;
  const uint64_t bump = vg::place_outputs_on_host(jb, totals.data(), &region, 512, out, placed, blocks);
  for (size_t j = 0; j < placed.size(); ++j) std::printf("%d", placed[j]);
  std::printf(" %llu %lld\n", static_cast<unsigned long long>(bump), static_cast<long long>(blocks));
  return 0;
}
