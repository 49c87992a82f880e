// Checks of the host-side size rules (headers without device code).  Prints
// "ok"; exits 1 with the failing expression.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <initializer_list>

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

int main() {
  triangle_lists();
  std::printf("ok\n");
}
