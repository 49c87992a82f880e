// Checks of the host-side size rules (headers without device code).  Prints
// "ok"; exits 1 with the failing expression.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <initializer_list>

#include "msshape.h"
#include "tclist.h"

#define EXPECT(x)                                    \
  do {                                               \
    if (!(x)) {                                      \
      std::printf("%s:%d: %s\n", __FILE__, __LINE__, #x); \
      std::exit(1);                                  \
    }                                                \
  } while (0)

// A list's counter at the sizes a graph can have: the place and the work of
// the last vertex come back out of it as they went in.
static void triangle_lists() {
  using namespace ug;
  for (uint64_t mo : std::initializer_list<uint64_t>{1ull << 18, 65ull << 20, kTcLargeEdges - 1, kTcLargeEdges,
                                                    68'000'000ull * 25, kTcMaxEdges}) {
    EXPECT(tc_counter_fits(mo));
    const uint64_t vertices = tc_max_listed(mo), units = tc_max_units(mo);
    const uint64_t counter = (vertices << kTcWorkBits) + units;
    EXPECT(counter >> kTcWorkBits == vertices);
    EXPECT((counter & ((1ull << kTcWorkBits) - 1)) == units);
  }
  // a ring lattice of 68 million nodes with 25 neighbours a side: every node has 25 oriented edges
  const uint64_t ring = 68'000'000;
  EXPECT(25 <= tc_split(ring * 25).search_max || ring < (1ull << (64 - kTcWorkBits)));
}

// Every grid fits the blocks that are resident at once, whatever the GPU (or
// the part of one) has: the groups' blocks wait for one another.
static void many_source_grids() {
  using namespace ug;
  for (uint64_t sms = 1; sms <= 160; sms++)
    for (uint64_t per_sm : {1, 2, 4, 5, 8})
      for (int W : {1, 4})
        for (uint64_t n : std::initializer_list<uint64_t>{1, 31, 256, 257, 8192, 65536, 1u << 20, 1u << 21, 1u << 28})
          for (uint64_t sources : std::initializer_list<uint64_t>{1, 64, 65, 256, 1000, 65536, 1u << 20}) {
            const uint64_t resident = sms * per_sm;
            const MsShape x = ms_shape(n, sources, W, resident);
            EXPECT(x.groups >= 1 && x.group_blocks >= 1);
            EXPECT((uint64_t)x.groups * x.group_blocks <= resident);
            EXPECT(x.groups <= (sources + 64 * W - 1) / (64 * W) && x.groups <= kMsGroups);
            EXPECT(x.groups == 1 || x.groups * n * W * 32 <= kMsMaskBytes);
          }
}

int main() {
  many_source_grids();
  triangle_lists();
  std::printf("ok\n");
}
