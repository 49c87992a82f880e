// tclist.h -- limits of the triangle kernels' vertex lists (tc.cu).  Host code
// only, so that they can be checked without a GPU.
//
// The vertices whose oriented list N+(v) takes a table are listed per kind
// with the work before them; one 64-bit counter per kind holds both, so that
// one atomic gives a vertex its place and its work's start together:
// vertices << kTcWorkBits | units of work.  With mo oriented edges
//  * a listed vertex has more than search_max of them, so at most
//    mo / (search_max + 1) are listed;
//  * no N+(u) has more than D = sqrt(2 mo) elements (each of those neighbours
//    has at least as many edges), so the probes, and one for each in-list
//    entry, are at most mo * (D + 1) / 2; a unit is 2^unit_shift of them, and
//    every vertex rounds up to a whole one.
// From 2^30 edges on, 24 elements could list 2^26 vertices and more, and 256
// probes a unit could pass 2^38: longer lists are searched and units doubled.
#pragma once

#include <stdint.h>

namespace ug {

constexpr int kTcWorkBits = 38;
constexpr uint64_t kTcMaxEdges = (1ull << 31) - 1;  // mo: the undirected CSR has below 2^32 entries
constexpr uint64_t kTcLargeEdges = 1ull << 30;

struct TcSplit {
  uint32_t search_max;  // N+(v) of up to this many elements is searched where it lies
  uint32_t unit_shift;
};

constexpr TcSplit tc_split(uint64_t mo) { return mo < kTcLargeEdges ? TcSplit{24, 8} : TcSplit{31, 9}; }

constexpr uint64_t tc_max_listed(uint64_t mo) { return mo / (tc_split(mo).search_max + 1); }

constexpr uint64_t tc_isqrt(uint64_t x) {
  uint64_t lo = 0, hi = 1ull << 32;
  while (hi - lo > 1) {
    const uint64_t mid = (lo + hi) / 2;
    if (mid * mid <= x) lo = mid; else hi = mid;
  }
  return lo;
}

constexpr uint64_t tc_max_units(uint64_t mo) {
  return ((mo * (tc_isqrt(2 * mo) + 1) / 2) >> tc_split(mo).unit_shift) + tc_max_listed(mo);
}

constexpr bool tc_counter_fits(uint64_t mo) {
  return tc_max_listed(mo) < (1ull << (64 - kTcWorkBits)) && tc_max_units(mo) < (1ull << kTcWorkBits);
}

// both bounds grow with mo on either side of the line
static_assert(tc_counter_fits(kTcLargeEdges - 1) && tc_counter_fits(kTcMaxEdges), "a list's counter does not wrap");
static_assert(tc_split(0).search_max < 32 && tc_split(kTcMaxEdges).search_max < 32, "five halvings find an element");

}  // namespace ug
