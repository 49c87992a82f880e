// tcstream.cuh -- the probe loop of the triangle kernels (tc.cu, batch.cu).
#pragma once

#include <stdint.h>

namespace ug {

constexpr uint32_t kTcEmpty = 0xFFFFFFFFu;  // no element

// Streams up to 32 lists back to back through a warp: lane l
// takes probe pb + l of the concatenation; hit(j, w) is called by every lane
// with the list's lane j and the element (kTcEmpty without a probe) and says
// whether it closes a triangle.  Lane k holds list k: the first slot b and the
// length len (0: no list).  The lists with probes are first moved to the
// front, so that each owns at least one probe and a round finds its lists with
// one ballot and one OR of the ends inside the round, in place of a five-step
// shuffle search; and each lane counts the hits of the list that moved to it
// from the ballot of the round's hits, in place of an atomic per hit or run.
// Returns that count, and the lane the list came from in *from_lane.  pack: 32
// words of shared memory of the warp.
// kAhead: the next round's elements load while this one's are probed (a few
// registers more: worth it where shared memory bounds the warps per SM).
template <bool kAhead, class F>
__device__ __forceinline__ uint32_t tc_stream(uint32_t* pack, uint32_t b, uint32_t len,
                                              const uint32_t* __restrict__ tgt,
                                              uint32_t* from_lane, F&& hit) {
  const uint32_t FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t some = __ballot_sync(FULL, len != 0);
  const int count = __popc(some);
  if (len) pack[__popc(some & lt)] = lane;
  __syncwarp();
  const uint32_t from = lane < count ? pack[lane] : 0u;
  __syncwarp();
  *from_lane = from;
  b = __shfl_sync(FULL, b, from);
  len = __shfl_sync(FULL, len, from);
  if (lane >= count) len = 0;
  uint32_t incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += t;
  }
  const uint32_t total = __shfl_sync(FULL, incl, 31);
  const uint32_t excl = incl - len;
  const uint32_t start = b - excl;  // probe p of pair k is tgt[start_k + p]
  // the round at pb: this lane's list and element
  auto round = [&](uint32_t pb, uint32_t& j) {
    // lists that end at or before pb, and those that end inside the round:
    // one that ends after `at` probes leaves the lanes from `at` to the next
    const uint32_t first = __popc(__ballot_sync(FULL, lane < count && incl <= pb));
    const uint32_t at = incl - pb;
    const bool inside = lane < count && incl > pb && at < 32;
    const uint32_t ends = __reduce_or_sync(FULL, inside ? 1u << (at & 31) : 0u);
    const uint32_t k = first + __popc(ends & (lt | (1u << lane)));
    const uint32_t sk = __shfl_sync(FULL, start, k & 31);
    j = __shfl_sync(FULL, from, k & 31);
    const uint32_t p = pb + lane;
    return p < total ? tgt[sk + p] : kTcEmpty;
  };
  uint32_t c = 0, j = 0;
  uint32_t w = kAhead && total ? round(0, j) : kTcEmpty;
  for (uint32_t pb = 0; pb < total; pb += 32) {
    uint32_t next_j = 0, next_w = kTcEmpty;
    if (!kAhead)
      w = round(pb, j);
    else if (pb + 32 < total)
      next_w = round(pb + 32, next_j);
    const bool h = hit(j, w);
    __syncwarp();
    const uint32_t hits = __ballot_sync(FULL, h);
    if (len && incl > pb && excl < pb + 32) {  // this lane's list is in the round
      const uint32_t lo = excl > pb ? excl - pb : 0u;
      const uint32_t upto = incl - pb < 32 ? (1u << (incl - pb)) - 1u : FULL;
      c += __popc(hits & upto & ~((1u << lo) - 1u));
    }
    if (kAhead) {
      j = next_j;
      w = next_w;
    }
  }
  return c;
}

}  // namespace ug
