// unionfind.cuh -- lock-free union-find over a parent array (global or
// shared memory through a generic pointer), used by weak connected components
// (ursa-core/src/algo/components.rs:14-68).
//
// A union always hooks the larger root under the smaller one with a
// compare-and-swap (a failed CAS means the root moved; the walk continues from
// the new parent), and finds compress paths by pointer jumping: the find with
// intermediate pointer jumping and the hooking of ECL-CC (Jaiganesh and
// Burtscher, "A High-Performance Connected Components Implementation for
// GPUs").  Parents only ever decrease, so each tree's root is the minimum id of
// its component.
#pragma once

#include <stdint.h>

namespace ug {

__device__ __forceinline__ uint32_t uf_parent(const uint32_t* p, uint32_t x) {
  return *(const volatile uint32_t*)&p[x];
}

// The same read through L1 (global memory only).  A cached parent may be
// stale, which costs steps and no correctness: a jump may have taken it off
// x's path, but two nodes once in one set stay in one, parents stay smaller
// than their children, and a stale root is found out by the compare-and-swap
// that hooks it.  Reads past L1 all meet at
// the L2 slice that holds the largest tree's root.
__device__ __forceinline__ uint32_t uf_parent_l1(const uint32_t* p, uint32_t x) {
  uint32_t v;
  asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(v) : "l"(p + x) : "memory");
  return v;
}

// Root of x with intermediate pointer jumping (parent[x] < x off the root).
__device__ __forceinline__ uint32_t uf_find(uint32_t* p, uint32_t x) {
  uint32_t par = uf_parent(p, x);
  if (par != x) {
    uint32_t prev = x, next;
    while (par > (next = uf_parent(p, par))) {
      p[prev] = next;
      prev = par;
      par = next;
    }
  }
  return par;
}

// The same through L1.  Short walks store x's parent alone: the nodes further
// up are those that every walk passes, and their stores would meet at a few
// addresses.  Past kUfShort links a walk reads past L1, wanting the jumps that
// others have stored, and stores its own.  Four links are too few where trees
// are a dozen deep: the last ones, near a root that all walks share, then meet
// at its L2 slice.  Kernels of a call with 4 / 8 / 16 / 32 (and before, with
// jumps from the first link on, past L1), us: four million nodes with twice as
// many random edges 1,864 / 828 / 765 / 939 (922), with 1.5 times 718 / 519 /
// 615 / 797 (524), three times 934 / 675 / 688 / 902 (793); a path of four
// million nodes in random order 889 / 511 / 426 / 424 (1,212); R-MAT with four
// million nodes 384 / 398 / 405 / 396 (1,933).  With 4 / 8: R-MAT with one
// million nodes 325 / 265 (717); sixteen random edges a node, a million nodes,
// 297 / 345 (752).
constexpr int kUfShort = 8;
__device__ __forceinline__ uint32_t uf_find_l1(uint32_t* p, uint32_t x) {
  uint32_t par = uf_parent_l1(p, x);
  if (par != x) {
    uint32_t prev = x, next;
    int links = 0;
    while (par > (next = links < kUfShort ? uf_parent_l1(p, par) : uf_parent(p, par))) {
      if (++links > kUfShort) p[prev] = next;
      prev = par;
      par = next;
    }
    if (links) p[x] = par;
  }
  return par;
}

template <bool kL1 = false>
__device__ __forceinline__ void uf_unite(uint32_t* p, uint32_t a, uint32_t b) {
  uint32_t ra = kL1 ? uf_find_l1(p, a) : uf_find(p, a);
  uint32_t rb = kL1 ? uf_find_l1(p, b) : uf_find(p, b);
  // bounded by the depth of the forest; each failed CAS moves one link up
  while (ra != rb) {
    if (ra < rb) {
      uint32_t old = atomicCAS(&p[rb], rb, ra);
      if (old == rb) return;
      rb = old;
    } else {
      uint32_t old = atomicCAS(&p[ra], ra, rb);
      if (old == ra) return;
      ra = old;
    }
  }
}

// Final root of x without writes (valid once every union has finished).
__device__ __forceinline__ uint32_t uf_root(const uint32_t* p, uint32_t x) {
  uint32_t par = uf_parent(p, x);
  while (par != x) {
    x = par;
    par = uf_parent(p, x);
  }
  return par;
}

}  // namespace ug
