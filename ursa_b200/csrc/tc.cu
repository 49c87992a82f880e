// tc.cu -- triangle_count and clustering_coefficient
// (ursa-core/src/algo/triangle.rs:23-62, clustering.rs:21-40).
//
// The reference counts, for every node u and neighbour a = N(u)[i], the
// common elements of N(u)[i+1..] and N(a): every triangle is counted once at
// each of its three vertices.  Here the vertices are ranked by (undirected
// degree, id) and each undirected edge is oriented from the lower to the
// higher rank, which bounds every oriented list N+ by O(sqrt(m)).  Each
// triangle u < v < w (in rank) is found exactly once, at its middle vertex
// v: w is in N+(v) and in N+(u) for an in-neighbour u of v, and only the
// elements of N+(u) ranked above v can be.  So a warp puts N+(v) in a hash
// table and probes, for each u with u -> v, the elements of N+(u) above v:
// sum over u of C(|N+(u)|, 2) probes (7.2 G at R-MAT-22, against 28.9 G for
// probing every N+(v), v in N+(u), into a table of N+(u)).  A hit credits u
// (one atomic per (u, v) pair), v (one per v) and w (a counter beside w's
// hash slot, flushed once per v).  Integer results are order-independent, so
// the counts are bit-identical to the reference.
#include "frontier.cuh"
#include "tclist.h"
#include "tcstream.cuh"

namespace ug {

namespace {

__device__ __forceinline__ bool rank_less(uint32_t du, uint32_t u, uint32_t dv, uint32_t v) {
  return du < dv || (du == dv && u < v);
}

__global__ void orient_flags_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                               uint64_t n, uint64_t ms, uint32_t* __restrict__ flag) {
  if (blockIdx.x == 0 && threadIdx.x == 0) flag[ms] = 0u;
  for_each_slot_owner(off, n, ms, [&](uint64_t k, uint32_t u) {
    uint32_t v = tgt[k];
    uint32_t du = off[u + 1] - off[u], dv = off[v + 1] - off[v];
    flag[k] = rank_less(du, u, dv, v) ? 1u : 0u;
  });
}

__global__ void orient_fill_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                              uint64_t n, uint64_t ms, const uint32_t* __restrict__ pos,
                              uint32_t* __restrict__ o_off, uint32_t* __restrict__ o_tgt) {
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < ms;
       k += (uint64_t)gridDim.x * blockDim.x) {
    if (pos[k + 1] != pos[k]) o_tgt[pos[k]] = tgt[k];
  }
  for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u <= n;
       u += (uint64_t)gridDim.x * blockDim.x)
    o_off[u] = pos[off[u]];
}

constexpr uint32_t kTcGrab = 16;

__device__ __forceinline__ uint32_t tc_hash(uint32_t w, uint32_t bits) {
  return (w * 0x9E3779B1u) >> (32 - bits);
}

// N+(v) of up to search_max elements (tclist.h: 24 below 2^30 edges) is
// searched where it lies, a lane per probe whatever its v; up to kTcWarpMax a
// warp's hash table; larger ones a block's.  Most vertices have short lists and few probes: a table for each
// of them was all latency (1,024 probes could take 300 tables).  Searched up
// to 16 / 24 / 32 elements: R-MAT-16 884 / 892 / 935 us a call, a Poisson graph
// of mean degree 32 3,345 / 3,168 / 3,129.
constexpr uint32_t kTcWarpMax = 256;
constexpr uint32_t kTcBlockWarps = 8;
constexpr uint32_t kTcMidSlots = 2048;  // a block's table in shared memory

// The vertices that take a table are listed per kind (warp, block), and the
// probes of a list's vertices, back to back, are cut into chunks of equal
// size (an entry's probes stay together) whatever vertices they span: a
// vertex's in-list is cut where it is long, and the next table starts where
// the last one ended.  At most kTcChunks chunks, so that the last ones end
// together on a large graph; at least kTcMinWork probes each.  (Pieces of up to 16K probes of one in-list, sixteen to a grab, left
// R-MAT-16's 7,000 warps waiting for the few that drew the hubs: 4.85 ms of
// warp tables against 0.41; one cut over all vertices left them skipping
// thousands of other kinds' lists: 13.7 ms of block tables on R-MAT-20 against
// 3.6.)
constexpr uint32_t kTcChunks[2] = {1u << 17, 1u << 13};
constexpr uint64_t kTcMinWork[2] = {1024, 8192};
constexpr uint32_t kTcSearchEntries = 256;  // most in-list entries per grab of a searching warp
constexpr int kTcKinds = 2;                 // warp tables, block tables

// One middle vertex v (original id) at a time: N+(v) = rank ids tgt[ob, oe)
// (all ranked above v, ascending) in a hash table T/C of 2^bits slots (load
// <= 1/2), shared by `threads` consecutive threads starting at `t0` (one warp,
// or a whole block); its in-neighbours' entries i in [ib, ie): u = in_src[i],
// the elements of N+(u) above v are tgt[in_pos[i] + 1, off[u + 1]).
__device__ __forceinline__ void tc_table_fill(uint32_t* T, uint32_t bits, uint32_t ob, uint32_t oe,
                                              const uint32_t* __restrict__ tgt, uint32_t t0,
                                              uint32_t threads) {
  const uint32_t bmask = (1u << (bits - 2)) - 1u;  // buckets of four slots
  for (uint32_t k = ob + t0; k < oe; k += threads) {
    const uint32_t x = tgt[k];
    for (uint32_t b = tc_hash(x, bits - 2);; b = (b + 1) & bmask) {
      uint32_t s = 0;
      while (s < 4 && atomicCAS(&T[4 * b + s], kTcEmpty, x) != kTcEmpty) s++;
      if (s < 4) break;
    }
  }
}

// Slot of w in the table (buckets of four keys, one 16-byte load each), or
// kTcEmpty if absent or w is kTcEmpty.  The warp takes every step together
// until its last lane is done, so that it is converged for the ballot that
// follows.
__device__ __forceinline__ uint32_t tc_find(const uint32_t* T, uint32_t bits, uint32_t w) {
  const uint32_t bmask = (1u << (bits - 2)) - 1u;
  uint32_t b = tc_hash(w, bits - 2), h = kTcEmpty;
  bool open = w != kTcEmpty;
  do {
    const uint4 q = *reinterpret_cast<const uint4*>(T + 4 * b);
    if (open) {
      if (q.x == w) h = 4 * b;
      if (q.y == w) h = 4 * b + 1;
      if (q.z == w) h = 4 * b + 2;
      if (q.w == w) h = 4 * b + 3;
      // slots fill in order: a bucket with room ends the chain
      open = h == kTcEmpty && q.w != kTcEmpty;
    }
    b = (b + 1) & bmask;
  } while (__any_sync(0xffffffffu, open));
  return h;
}

// Credits the counts kept beside the table to their w and empties it.
__device__ __forceinline__ void tc_table_flush(uint32_t* T, uint32_t* C, uint32_t bits,
                                               const uint32_t* __restrict__ vertex_of,
                                               uint32_t* __restrict__ tri, uint32_t t0,
                                               uint32_t threads) {
  const uint32_t mask = (1u << bits) - 1u;
  for (uint32_t h = t0; h <= mask; h += threads) {
    const uint32_t t = T[h];
    if (t != kTcEmpty) {
      const uint32_t c = C[h];
      if (c) atomicAdd(&tri[vertex_of[t]], c);
      C[h] = 0;
      T[h] = kTcEmpty;
    }
  }
}

// One warp: `group` (at most 32) entries of [i0, ie) at a time, `stride`
// apart; credits each u and returns the warp's hit count (all lanes).
__device__ __forceinline__ uint32_t tc_pairs(uint32_t* T, uint32_t* C, uint32_t* pack, uint32_t bits,
                                             uint32_t i0, uint32_t ie, uint32_t group, uint32_t stride,
                                             const uint32_t* __restrict__ off,
                                             const uint32_t* __restrict__ tgt,
                                             const uint32_t* __restrict__ in_src,
                                             const uint32_t* __restrict__ in_pos,
                                             uint32_t* __restrict__ tri) {
  const uint32_t FULL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31;
  uint32_t cv = 0;  // per lane; summed at the end
  for (; i0 < ie; i0 += stride) {
    // (u, v) pairs, one per lane: u and the part of N+(u) above v
    uint32_t u = 0, b = 0, len = 0;
    if (lane < group && i0 + lane < ie) {
      u = in_src[i0 + lane];
      b = in_pos[i0 + lane] + 1;
      len = off[u + 1] - b;
    }
    uint32_t from;
    const uint32_t c = tc_stream<false>(pack, b, len, tgt, &from, [&](uint32_t, uint32_t w) {
      const uint32_t h = tc_find(T, bits, w);
      if (h != kTcEmpty) atomicAdd(&C[h], 1u);
      return h != kTcEmpty;
    });
    u = __shfl_sync(FULL, u, from);
    if (c) atomicAdd(&tri[u], c);
    cv += c;
  }
  return __reduce_add_sync(FULL, cv);
}

// One kind's vertices, in no order: ranks, and the work (in units) of the
// ones before; its chunks: index of the vertex and in-list entry where each
// starts (one past the last closes the list).
struct TcList {
  uint32_t* rank;
  uint64_t* at;
  uint32_t* chunk_i;
  uint32_t* chunk_e;
};
// Device words of a call: per kind, the list's vertices and work (tclist.h),
// chunks in use, and the grab counters.
struct TcCtl {
  unsigned long long size[kTcKinds];
  unsigned long long next[kTcKinds + 1];
  uint32_t chunks[kTcKinds];
};

struct TcArgs {
  const uint32_t* off;        // oriented CSR rows by original id
  const uint32_t* tgt;        // ... targets as rank ids, ascending in each row
  const uint32_t* in_off;     // in-lists of the oriented graph, by rank
  const uint32_t* in_src;     // ... holding original ids
  const uint32_t* in_pos;     // ... and the entry's slot in its row of tgt
  const uint32_t* in_rank;    // ... and the rank of the list
  const uint32_t* vertex_of;  // rank -> original id
  uint64_t entries;           // in-list entries of all ranks
  uint32_t search_max;
  uint32_t grab;              // ... taken at a time by a searching warp
  TcList list;                // this launch's kind
  int kind;
  TcCtl* ctl;
  uint32_t* tri;
};

// A list's vertices i .. i + 31 (a lane each) between chunk starts (i0, e0)
// and (i1, e1): vertex, N+(v) and the in-list entries to walk (ib < ie).
struct TcRank {
  uint32_t v, ob, dv, ib, ie;
};
__device__ __forceinline__ TcRank tc_rank(const TcArgs& a, uint32_t i, uint32_t count, uint32_t i0,
                                          uint32_t e0, uint32_t i1, uint32_t e1) {
  TcRank x{0, 0, 0, 0, 0};
  if (i < count && i <= i1) {
    const uint32_t r = a.list.rank[i];
    x.v = a.vertex_of[r];
    x.ob = a.off[x.v];
    x.dv = a.off[x.v + 1] - x.ob;
    x.ib = i == i0 ? e0 : a.in_off[r];
    x.ie = i == i1 ? e1 : a.in_off[r + 1];
  }
  return x;
}

// log2 of the table's slots: load <= 1/2, at least two buckets of four slots.
__device__ __forceinline__ uint32_t tc_bits(uint32_t dv) {
  return max(3u, 32u - (uint32_t)__clz(2 * dv - 1));
}

// Middle vertices with |N+(v)| <= search_max: a warp takes 32 entries at a
// time whatever their v; each probe is searched in N+(v) by bisection.
__global__ void __launch_bounds__(256) tc_middle_search_k(TcArgs a) {
  __shared__ uint32_t pack[8][32];
  const uint32_t FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  while (true) {
    unsigned long long g = 0;
    if (lane == 0) g = atomicAdd(&a.ctl->next[kTcKinds], (unsigned long long)a.grab);
    g = __shfl_sync(FULL, g, 0);
    if (g >= a.entries) break;
    const uint32_t e1 = (uint32_t)min(a.entries, (uint64_t)g + a.grab);
    for (uint32_t e = (uint32_t)g; e < e1; e += 32) {
      uint32_t u = 0, b = 0, len = 0, v = 0, ob = 0, dv = 0;
      if (e + lane < e1) {
        v = a.vertex_of[a.in_rank[e + lane]];
        ob = a.off[v];
        dv = a.off[v + 1] - ob;
        if (dv != 0 && dv <= a.search_max) {
          u = a.in_src[e + lane];
          b = a.in_pos[e + lane] + 1;
          len = a.off[u + 1] - b;
        }
      }
      if (!__any_sync(FULL, len != 0)) continue;
      uint32_t from;
      const uint32_t c = tc_stream<true>(pack[wid], b, len, a.tgt, &from, [&](uint32_t j, uint32_t w) {
        uint32_t lo = __shfl_sync(FULL, ob, j);
        uint32_t left = __shfl_sync(FULL, dv, j);
        if (w == kTcEmpty) left = 0;
#pragma unroll
        for (int step = 0; step < 5; step++) {  // the last element <= w, or the first one
          const uint32_t half = left >> 1;
          if (half && a.tgt[lo + half] <= w) lo += half;
          left -= half;
        }
        const bool h = left && a.tgt[lo] == w;
        if (h) atomicAdd(&a.tri[a.vertex_of[w]], 1u);
        return h;
      });
      u = __shfl_sync(FULL, u, from);
      v = __shfl_sync(FULL, v, from);
      if (c) {
        atomicAdd(&a.tri[u], c);
        atomicAdd(&a.tri[v], c);
      }
    }
  }
}

// Middle vertices with |N+(v)| <= kSlots / 2: a warp per chunk, a table per
// warp in shared memory (kWarps warps per block).
template <int kSlots, int kWarps>
__global__ void __launch_bounds__(kWarps * 32) tc_middle_warp_k(TcArgs a) {
  extern __shared__ __align__(16) uint32_t tc_sm[];  // read as uint4
  const uint32_t FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t* T = tc_sm + (size_t)wid * 2 * kSlots;
  uint32_t* C = T + kSlots;
  uint32_t* pack = tc_sm + (size_t)kWarps * 2 * kSlots + wid * 32;
  for (int i = lane; i < kSlots; i += 32) {
    T[i] = kTcEmpty;
    C[i] = 0;
  }
  __syncwarp();
  const uint32_t n_chunks = a.ctl->chunks[a.kind];
  const uint32_t count = (uint32_t)(a.ctl->size[a.kind] >> kTcWorkBits);
  while (true) {
    unsigned long long g = 0;
    if (lane == 0) g = atomicAdd(&a.ctl->next[a.kind], 1ull);
    g = __shfl_sync(FULL, g, 0);
    if (g >= n_chunks) break;
    const uint32_t i0 = a.list.chunk_i[g], e0 = a.list.chunk_e[g];
    const uint32_t i1 = a.list.chunk_i[g + 1], e1 = a.list.chunk_e[g + 1];
    for (uint32_t i = i0; i < count && i <= i1; i += 32) {
      const TcRank x = tc_rank(a, i + lane, count, i0, e0, i1, e1);
      for (unsigned todo = __ballot_sync(FULL, x.ib < x.ie); todo; todo &= todo - 1) {
        const int l = __ffs(todo) - 1;
        const uint32_t v = __shfl_sync(FULL, x.v, l), ob = __shfl_sync(FULL, x.ob, l);
        const uint32_t dv = __shfl_sync(FULL, x.dv, l);
        const uint32_t ib = __shfl_sync(FULL, x.ib, l), ie = __shfl_sync(FULL, x.ie, l);
        const uint32_t bits = tc_bits(dv);
        tc_table_fill(T, bits, ob, ob + dv, a.tgt, lane, 32);
        __syncwarp();
        const uint32_t cv = tc_pairs(T, C, pack, bits, ib, ie, 32, 32, a.off, a.tgt, a.in_src, a.in_pos, a.tri);
        __syncwarp();
        tc_table_flush(T, C, bits, a.vertex_of, a.tri, lane, 32);
        if (cv && lane == 0) atomicAdd(&a.tri[v], cv);
        __syncwarp();
      }
    }
  }
}

// The larger ones: one block of kWarps warps per chunk, sharing one table:
// kTcMidSlots slots in shared memory up to half as many elements, else
// table[block * 2 * slots, +2 * slots) in global memory (keys, then counts;
// all empty on entry, left empty).  Every warp reads the vertices by itself:
// the same values, so the same loop.
template <int kWarps>
__global__ void __launch_bounds__(kWarps * 32) tc_middle_block_k(TcArgs a, uint32_t* table,
                                                                 uint32_t slots) {
  extern __shared__ __align__(16) uint32_t tc_sm[];  // read as uint4
  __shared__ uint32_t pack[kWarps][32];
  __shared__ unsigned long long s_g;
  const uint32_t FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (uint32_t i = threadIdx.x; i < kTcMidSlots; i += blockDim.x) {
    tc_sm[i] = kTcEmpty;
    tc_sm[kTcMidSlots + i] = 0;
  }
  __syncthreads();
  const uint32_t n_chunks = a.ctl->chunks[a.kind];
  const uint32_t count = (uint32_t)(a.ctl->size[a.kind] >> kTcWorkBits);
  while (true) {
    if (threadIdx.x == 0) s_g = atomicAdd(&a.ctl->next[a.kind], 1ull);
    __syncthreads();
    const unsigned long long g = s_g;
    __syncthreads();  // read by all before thread 0 takes the next chunk
    if (g >= n_chunks) break;
    const uint32_t i0 = a.list.chunk_i[g], e0 = a.list.chunk_e[g];
    const uint32_t i1 = a.list.chunk_i[g + 1], e1 = a.list.chunk_e[g + 1];
    for (uint32_t i = i0; i < count && i <= i1; i += 32) {
      const TcRank x = tc_rank(a, i + lane, count, i0, e0, i1, e1);
      for (unsigned todo = __ballot_sync(FULL, x.ib < x.ie); todo; todo &= todo - 1) {
        const int l = __ffs(todo) - 1;
        const uint32_t v = __shfl_sync(FULL, x.v, l), ob = __shfl_sync(FULL, x.ob, l);
        const uint32_t dv = __shfl_sync(FULL, x.dv, l);
        const uint32_t ib = __shfl_sync(FULL, x.ib, l), ie = __shfl_sync(FULL, x.ie, l);
        const uint32_t bits = tc_bits(dv);
        uint32_t* T = tc_sm;
        uint32_t* C = tc_sm + kTcMidSlots;
        if (dv > kTcMidSlots / 2) {
          T = table + (size_t)blockIdx.x * 2 * slots;
          C = T + slots;
        }
        tc_table_fill(T, bits, ob, ob + dv, a.tgt, threadIdx.x, blockDim.x);
        __syncthreads();
        // the entries spread over all warps: suffixes are long here, so a
        // few tens of entries can be all the work
        const uint32_t group = min(32u, (ie - ib + kWarps - 1) / kWarps);
        const uint32_t cv = tc_pairs(T, C, pack[wid], bits, ib + group * wid, ie, group,
                                     group * kWarps, a.off, a.tgt, a.in_src, a.in_pos, a.tri);
        if (cv && lane == 0) atomicAdd(&a.tri[v], cv);
        __syncthreads();
        tc_table_flush(T, C, bits, a.vertex_of, a.tri, threadIdx.x, blockDim.x);
        __syncthreads();
      }
    }
  }
}

// ---- small graphs (the per-graph calls of a batch's plain path): the
// rank relabelling, its two radix sorts and the host reads of the
// middle-vertex path are a fixed cost of about a millisecond, more than the
// whole count takes on a graph of a few tens of thousands of edges.  Below
// kSmallEntries undirected CSR entries one kernel over the (degree, id)
// orientation counts instead: a warp per vertex u puts N+(u) in a
// shared-memory hash set (open addressing, load <= 1/2; longer lists are
// searched by binary search in global memory) and streams the concatenation
// of N+(v), v in N+(u), 32 lists at a time; a hit w is the triangle (u, v, w),
// credited to w at once and to v and u by the lists' counts.
constexpr uint64_t kSmallEntries = 1u << 18;
constexpr int kSmThreads = 256;
constexpr int kSmWarps = kSmThreads / 32;
constexpr uint32_t kSmSlots = 2048;  // hash slots per warp
constexpr uint32_t kSmHashMax = kSmSlots / 2;

__global__ void __launch_bounds__(kSmThreads) count_small_k(const uint32_t* __restrict__ o_off,
                                                          const uint32_t* __restrict__ o_tgt,
                                                          uint64_t n, uint32_t* __restrict__ tri,
                                                          unsigned long long* __restrict__ next) {
  extern __shared__ __align__(16) uint32_t tc_sm[];
  const uint32_t FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t* T = tc_sm + (size_t)w * kSmSlots;
  uint32_t* pack = tc_sm + (size_t)kSmWarps * kSmSlots + w * 32;
  for (uint32_t i = lane; i < kSmSlots; i += 32) T[i] = kTcEmpty;
  __syncwarp();
  while (true) {
    unsigned long long g = 0;
    if (lane == 0) g = atomicAdd(next, (unsigned long long)kTcGrab);
    g = __shfl_sync(FULL, g, 0);
    if (g >= n) break;
    const uint64_t g_end = g + kTcGrab < n ? g + kTcGrab : n;
    for (uint64_t u = g; u < g_end; u++) {
      const uint32_t ob = o_off[u], oe = o_off[u + 1], du = oe - ob;
      if (du < 2) continue;  // u is the lowest vertex of no triangle
      const bool hashed = du <= kSmHashMax;
      uint32_t bits = 6;
      while ((1u << bits) < 2 * du) bits++;
      const uint32_t mask = (1u << bits) - 1;
      if (hashed) {
        for (uint32_t i = ob + lane; i < oe; i += 32) {
          const uint32_t x = o_tgt[i];
          uint32_t h = tc_hash(x, bits);
          while (atomicCAS(&T[h], kTcEmpty, x) != kTcEmpty) h = (h + 1) & mask;
        }
        __syncwarp();
      }
      uint32_t cu = 0;
      for (uint32_t vb = ob; vb < oe; vb += 32) {
        const uint32_t i = vb + lane;
        uint32_t v = 0, st = 0, len = 0;
        if (i < oe) {
          v = o_tgt[i];
          st = o_off[v];
          len = o_off[v + 1] - st;
        }
        uint32_t from;
        const uint32_t c = tc_stream<true>(pack, st, len, o_tgt, &from, [&](uint32_t, uint32_t x) {
          bool hit = false;
          if (hashed) {  // the warp steps together until its last lane is done
            uint32_t h = tc_hash(x, bits);
            bool open = x != kTcEmpty;
            do {
              const uint32_t t = T[h];
              hit |= open && t == x;
              open = open && t != x && t != kTcEmpty;
              h = (h + 1) & mask;
            } while (__any_sync(FULL, open));
          } else if (x != kTcEmpty) {
            uint32_t lo = ob, left = oe - ob;
            while (left > 1) {  // the last element <= x, or the first one
              const uint32_t half = left >> 1;
              if (o_tgt[lo + half] <= x) lo += half;
              left -= half;
            }
            hit = o_tgt[lo] == x;
          }
          if (hit) atomicAdd(&tri[x], 1u);
          return hit;
        });
        v = __shfl_sync(FULL, v, from);
        if (c) atomicAdd(&tri[v], c);
        cu += c;
      }
      cu = __reduce_add_sync(FULL, cu);
      if (lane == 0 && cu) atomicAdd(&tri[u], cu);
      if (hashed) {
        __syncwarp();
        for (uint32_t k = lane; k <= mask; k += 32) T[k] = kTcEmpty;
        __syncwarp();
      }
    }
  }
}


size_t small_smem_bytes() { return ((size_t)kSmWarps * kSmSlots + kSmWarps * 32) * sizeof(uint32_t); }

// ---- preparation: ranks, the rank-oriented CSR and its in-lists
__global__ void und_degree_k(const uint32_t* __restrict__ off, uint64_t n, uint32_t* __restrict__ deg) {
  for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n;
       u += (uint64_t)gridDim.x * blockDim.x)
    deg[u] = off[u + 1] - off[u];
}

__global__ void rank_scatter_k(const uint32_t* __restrict__ vertex_of, uint64_t n,
                               uint32_t* __restrict__ rank_of) {
  for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n;
       r += (uint64_t)gridDim.x * blockDim.x)
    rank_of[vertex_of[r]] = (uint32_t)r;
}

__global__ void rank_flags_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                             uint64_t n, uint64_t ms, const uint32_t* __restrict__ rank_of,
                             uint32_t* __restrict__ flag) {
  if (blockIdx.x == 0 && threadIdx.x == 0) flag[ms] = 0u;
  for_each_slot_owner(off, n, ms, [&](uint64_t k, uint32_t u) {
    flag[k] = rank_of[u] < rank_of[tgt[k]] ? 1u : 0u;
  });
}

__global__ void rank_fill_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                            uint64_t n, uint64_t ms, const uint32_t* __restrict__ rank_of,
                            const uint32_t* __restrict__ pos, uint32_t* __restrict__ o_off,
                            uint32_t* __restrict__ o_tgt, uint32_t* __restrict__ o_src) {
  for_each_slot_owner(off, n, ms, [&](uint64_t k, uint32_t u) {
    if (pos[k + 1] != pos[k]) {
      o_tgt[pos[k]] = rank_of[tgt[k]];
      o_src[pos[k]] = u;
    }
  });
  for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u <= n;
       u += (uint64_t)gridDim.x * blockDim.x)
    o_off[u] = pos[off[u]];
}

// in_pos[order[p]] = p: the final slot of each in-list entry in the sorted rows.
__global__ void pos_scatter_k(const uint32_t* __restrict__ order, uint64_t m,
                              uint32_t* __restrict__ in_pos) {
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < m;
       p += (uint64_t)gridDim.x * blockDim.x)
    in_pos[order[p]] = (uint32_t)p;
}

// Probes of in-list entry i: the elements of N+(u) above v.
__global__ void entry_work_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ in_src,
                             const uint32_t* __restrict__ in_pos, uint64_t m,
                             uint64_t* __restrict__ work) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (uint64_t)gridDim.x * blockDim.x)
    work[i] = off[in_src[i] + 1] - in_pos[i];  // and one for the entry itself
}

// The ranks that take a table, listed per kind with their work (probes in
// units, and one for the table itself).  One atomic per warp and kind gives
// the vertices' places and the work before them together.
__global__ void tc_lists_k(const uint32_t* __restrict__ in_off, const uint32_t* __restrict__ off,
                           const uint32_t* __restrict__ vertex_of, const uint64_t* __restrict__ wp,
                           uint64_t n, TcSplit split, TcList warp_list, TcList block_list, TcCtl* ctl) {
  const uint32_t FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t r0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull; r0 < n; r0 += stride) {
    const uint64_t r = r0 + lane;
    int kind = -1;
    unsigned long long x = 0;
    if (r < n) {
      const uint32_t b = in_off[r], e = in_off[r + 1];
      if (b != e) {
        const uint32_t v = vertex_of[r];
        const uint32_t dv = off[v + 1] - off[v];
        if (dv > split.search_max) {
          kind = dv > kTcWarpMax ? 1 : 0;
          x = (1ull << kTcWorkBits) + ((wp[e] - wp[b]) >> split.unit_shift) + 1;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kTcKinds; k++) {
      if (!__any_sync(FULL, kind == k)) continue;
      const unsigned long long mine = kind == k ? x : 0ull;
      unsigned long long incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += t;
      }
      unsigned long long base = 0;
      if (lane == 31) base = atomicAdd(&ctl->size[k], incl);
      base = __shfl_sync(FULL, base, 31) + incl - mine;
      if (kind == k) {
        const TcList& l = k ? block_list : warp_list;
        const uint32_t i = (uint32_t)(base >> kTcWorkBits);
        l.rank[i] = (uint32_t)r;
        l.at[i] = base & ((1ull << kTcWorkBits) - 1);
      }
    }
  }
}

// Chunk c of a kind starts c * step units into its list's work: in the last
// vertex that starts at or before, at the first entry whose probes begin at
// or after.
__global__ void tc_chunks_k(const uint32_t* __restrict__ in_off, const uint64_t* __restrict__ wp,
                            TcList list, int kind, uint64_t min_work,
                            uint64_t max_chunks, uint32_t unit_shift, TcCtl* ctl) {
  const unsigned long long size = ctl->size[kind];
  const uint32_t count = (uint32_t)(size >> kTcWorkBits);
  const uint64_t work = size & ((1ull << kTcWorkBits) - 1);
  const uint64_t step = max(min_work, (work + max_chunks - 1) / max_chunks);
  const uint32_t used = (uint32_t)((work + step - 1) / step);
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->chunks[kind] = used;
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c <= used; c += gridDim.x * blockDim.x) {
    if (c == used) {
      list.chunk_i[c] = count;
      list.chunk_e[c] = 0;
      continue;
    }
    const uint64_t want = c * step;
    uint32_t lo = 0, hi = count;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (list.at[mid] <= want) lo = mid; else hi = mid;
    }
    const uint32_t r = list.rank[lo];
    uint32_t e = in_off[r], end = in_off[r + 1];
    const uint64_t cut = wp[e] + ((want - list.at[lo]) << unit_shift);
    while (e < end) {
      const uint32_t mid = e + ((end - e) >> 1);
      if (wp[mid] < cut) e = mid + 1; else end = mid;
    }
    list.chunk_i[c] = lo;
    list.chunk_e[c] = e;
  }
}

// Global tables, one per block: keys (empty) then counts (zero), slots each.
__global__ void fill_tables_k(uint32_t* __restrict__ table, uint64_t tables, uint32_t slots) {
  const uint64_t total = tables * 2 * slots;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (uint64_t)gridDim.x * blockDim.x)
    table[i] = ((i / slots) & 1) ? 0u : kTcEmpty;
}

__global__ void max_outdeg_k(const uint32_t* __restrict__ off, uint64_t n, unsigned* __restrict__ mx) {
  uint32_t best = 0;
  for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n;
       u += (uint64_t)gridDim.x * blockDim.x)
    best = max(best, off[u + 1] - off[u]);
  best = __reduce_max_sync(0xffffffffu, best);
  if ((threadIdx.x & 31) == 0 && best) atomicMax(mx, best);
}

// clustering.rs:21-40: 2 T / (k (k - 1)), 0.0 for k < 2, in f64.
__global__ void clustering_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tri,
                             uint64_t n, double* __restrict__ out) {
  for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n;
       u += (uint64_t)gridDim.x * blockDim.x) {
    double k = (double)(off[u + 1] - off[u]);
    out[u] = k < 2.0 ? 0.0 : __ddiv_rn(__dmul_rn(2.0, (double)tri[u]), __dmul_rn(k, __dsub_rn(k, 1.0)));
  }
}

}  // namespace

// Orientation of the undirected CSR by (degree, id), targets as original ids
// (the batched triangle kernel's input; host-synchronising, done once).
void orient_build(TopoImpl* t, OrientedCsr& o, cudaStream_t s) {
  const uint64_t n = t->n;
  ensure_undirected(t, s);
  const uint64_t ms = t->m_und;
  o.off.alloc(n + 1, s);
  o.mo = 0;
  if (ms == 0) {
    UG_CUDA(cudaMemsetAsync(o.off.get(), 0, (n + 1) * sizeof(uint32_t), s));
    o.tgt.alloc(1, s);
    return;
  }
  Scratch<uint32_t> pos(ms + 1, s);
  orient_flags_k<<<grid_for(ms), kBlock, 0, s>>>(t->und_off.get(), t->und_tgt.get(), n, ms,
                                                 pos.get());
  UG_LAUNCH_CHECK();
  Scratch<uint32_t> total(1, s);
  exclusive_scan_u32(pos.get(), pos.get(), ms + 1, total.get(), s);
  o.mo = read_u32(total.get(), s);
  o.tgt.alloc(o.mo ? o.mo : 1, s);
  orient_fill_k<<<grid_for(ms), kBlock, 0, s>>>(t->und_off.get(), t->und_tgt.get(), n, ms,
                                                pos.get(), o.off.get(), o.tgt.get());
  UG_LAUNCH_CHECK();
}

// Blocks per SM for a kernel and dynamic shared memory size, once per device
// (the shared-memory limit is raised on first use).
template <class K>
static int tc_blocks_per_sm(K kernel, int threads, size_t smem, int dev, int* cache,
                            std::mutex& mu) {
  std::lock_guard<std::mutex> g(mu);
  if (!cache[dev]) {
    UG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    UG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&cache[dev], kernel, threads, smem));
    UG_CHECK(cache[dev] > 0, URSA_GPU_ECUDA, "triangle kernel cannot be resident");
  }
  return cache[dev];
}

void triangle_count_run(TopoImpl* t, uint32_t* d_tri, cudaStream_t s) {
  const uint64_t n = t->n;
  if (n == 0) return;
  UG_CUDA(cudaMemsetAsync(d_tri, 0, n * sizeof(uint32_t), s));
  ensure_undirected(t, s);
  const uint64_t ms = t->m_und;
  if (ms == 0) return;
  int dev = 0;
  UG_CUDA(cudaGetDevice(&dev));
  UG_CHECK(dev >= 0 && dev < 64, URSA_GPU_EINVAL, "device index out of range");
  if (ms < kSmallEntries) {
    OrientedCsr o;
    orient_build(t, o, s);
    if (o.mo) {
      static std::mutex mu;
      static int cache[64] = {0};
      const int per_sm = tc_blocks_per_sm(count_small_k, kSmThreads, small_smem_bytes(), dev, cache, mu);
      Scratch<unsigned long long> next(1, s);
      UG_CUDA(cudaMemsetAsync(next.get(), 0, sizeof(unsigned long long), s));
      count_small_k<<<per_sm * sm_count(dev), kSmThreads, small_smem_bytes(), s>>>(
          o.off.get(), o.tgt.get(), n, d_tri, next.get());
      UG_LAUNCH_CHECK();
      count_launch();
    }
    UG_CUDA(cudaStreamSynchronize(s));  // o's buffers are released on return
    return;
  }
  // ranks by (undirected degree, id): a stable sort by degree
  Scratch<uint32_t> vertex_of(n, s), rank_of(n, s);
  {
    Scratch<uint32_t> deg(n, s), deg_sorted(n, s);
    und_degree_k<<<grid_for(n), kBlock, 0, s>>>(t->und_off.get(), n, deg.get());
    UG_LAUNCH_CHECK();
    radix_sort_pairs(deg.get(), nullptr, n, bits_for(ms), deg_sorted.get(), vertex_of.get(),
                     nullptr, nullptr, s);
    rank_scatter_k<<<grid_for(n), kBlock, 0, s>>>(vertex_of.get(), n, rank_of.get());
    UG_LAUNCH_CHECK();
  }
  // every undirected edge once, from the lower to the higher rank; targets
  // as rank ids, rows by original id
  Scratch<uint32_t> pos(ms + 1, s);
  rank_flags_k<<<grid_for(ms), kBlock, 0, s>>>(t->und_off.get(), t->und_tgt.get(), n, ms,
                                               rank_of.get(), pos.get());
  UG_LAUNCH_CHECK();
  Scratch<uint32_t> total(1, s);
  exclusive_scan_u32(pos.get(), pos.get(), ms + 1, total.get(), s);
  const uint64_t mo = read_u32(total.get(), s);
  Scratch<uint32_t> o_off(n + 1, s), o_tgt(mo ? mo : 1, s), o_src(mo ? mo : 1, s);
  rank_fill_k<<<grid_for(ms), kBlock, 0, s>>>(t->und_off.get(), t->und_tgt.get(), n, ms,
                                              rank_of.get(), pos.get(), o_off.get(), o_tgt.get(),
                                              o_src.get());
  UG_LAUNCH_CHECK();
  pos.release();
  rank_of.release();
  if (mo == 0) return;
  // in-lists: the oriented edges grouped by target rank (sources in row
  // order), then the rows re-sorted by target rank (a stable sort of the
  // in-list order by source), and each in-list entry's slot in its sorted row
  Scratch<uint32_t> in_off(n + 1, s), in_src(mo, s), in_pos(mo, s), in_rank(mo, s);
  {
    uint32_t* const keys = in_rank.get();
    radix_sort_pairs(o_tgt.get(), o_src.get(), mo, bits_for(n - 1), keys, in_src.get(),
                     nullptr, nullptr, s);
    offsets_from_sorted(keys, mo, n, in_off.get(), s);
    Scratch<uint32_t> rows(mo, s), order(mo, s);
    radix_sort_pairs(in_src.get(), nullptr, mo, bits_for(n - 1), rows.get(), order.get(),
                     keys, o_tgt.get(), s);
    pos_scatter_k<<<grid_for(mo), kBlock, 0, s>>>(order.get(), mo, in_pos.get());
    UG_LAUNCH_CHECK();
  }
  o_src.release();
  UG_CHECK(mo <= kTcMaxEdges, URSA_GPU_EINVAL, "triangle count: too many undirected edges");
  const TcSplit split = tc_split(mo);
  uint32_t max_dv = 0;
  {
    Scratch<unsigned> mx(1, s);
    UG_CUDA(cudaMemsetAsync(mx.get(), 0, sizeof(unsigned), s));
    max_outdeg_k<<<grid_for(n), kBlock, 0, s>>>(o_off.get(), n, mx.get());
    UG_LAUNCH_CHECK();
    max_dv = read_u32(mx.get(), s);
  }
  Scratch<TcCtl> ctl(1, s);
  UG_CUDA(cudaMemsetAsync(ctl.get(), 0, sizeof(TcCtl), s));
  // chunks of equal probes over the lists of vertices that take a table, where
  // there are any (a star of a million nodes 847 us with empty lists, 812
  // without)
  Scratch<uint64_t> wp, before;
  Scratch<uint32_t> ranks, chunk_at;
  TcList lists[kTcKinds] = {};
  if (max_dv > split.search_max) {
    wp.alloc(mo + 1, s);
    entry_work_k<<<grid_for(mo), kBlock, 0, s>>>(o_off.get(), in_src.get(), in_pos.get(), mo, wp.get());
    UG_LAUNCH_CHECK();
    UG_CUDA(cudaMemsetAsync(wp.get() + mo, 0, sizeof(uint64_t), s));
    exclusive_scan_u64(wp.get(), wp.get(), mo + 1, nullptr, s);
    const uint64_t listed = std::min<uint64_t>(n, tc_max_listed(mo) + 1);  // at most, of a kind
    ranks.alloc(kTcKinds * listed, s);
    before.alloc(kTcKinds * listed, s);
    chunk_at.alloc(2 * (kTcChunks[0] + kTcChunks[1] + 2ull), s);
    for (int k = 0; k < kTcKinds; k++) {
      uint32_t* at = chunk_at.get() + (k ? 2 * (kTcChunks[0] + 1ull) : 0);
      lists[k] = TcList{ranks.get() + k * listed, before.get() + k * listed, at, at + kTcChunks[k] + 1};
    }
    tc_lists_k<<<grid_for(n), kBlock, 0, s>>>(in_off.get(), o_off.get(), vertex_of.get(), wp.get(), n,
                                              split, lists[0], lists[1], ctl.get());
    UG_LAUNCH_CHECK();
    for (int k = 0; k < kTcKinds; k++) {
      tc_chunks_k<<<grid_for(kTcChunks[k] + 1), kBlock, 0, s>>>(
          in_off.get(), wp.get(), lists[k], k, kTcMinWork[k] >> split.unit_shift, kTcChunks[k],
          split.unit_shift, ctl.get());
      UG_LAUNCH_CHECK();
    }
  }
  TcArgs a;
  a.off = o_off.get();
  a.tgt = o_tgt.get();
  a.in_off = in_off.get();
  a.in_src = in_src.get();
  a.in_pos = in_pos.get();
  a.in_rank = in_rank.get();
  a.vertex_of = vertex_of.get();
  a.entries = mo;
  a.search_max = split.search_max;
  a.list = lists[0];
  a.kind = 0;
  a.ctl = ctl.get();
  a.tri = d_tri;
  {  // |N+(v)| <= search_max: searched
    static std::mutex mu;
    static int cache[64] = {0};
    const int per_sm = tc_blocks_per_sm(tc_middle_search_k, 256, 0, dev, cache, mu);
    const uint64_t warps = 8ull * per_sm * sm_count(dev);
    a.grab = (uint32_t)std::min<uint64_t>(kTcSearchEntries, (mo / (4 * warps) + 31) / 32 * 32 + 32);
    tc_middle_search_k<<<per_sm * sm_count(dev), 256, 0, s>>>(a);
    UG_LAUNCH_CHECK();
    count_launch();
  }
  constexpr int kSmallSlots = 2 * kTcWarpMax, kWarpsW = 8, kWarpsB = kTcBlockWarps;
  if (max_dv > split.search_max) {  // up to 256: a warp per chunk
    static std::mutex mu;
    static int cache[64] = {0};
    const size_t smem = ((size_t)kWarpsW * 2 * kSmallSlots + kWarpsW * 32) * sizeof(uint32_t);
    const int per_sm = tc_blocks_per_sm(tc_middle_warp_k<kSmallSlots, kWarpsW>, kWarpsW * 32, smem,
                                        dev, cache, mu);
    tc_middle_warp_k<kSmallSlots, kWarpsW><<<per_sm * sm_count(dev), kWarpsW * 32, smem, s>>>(a);
    UG_LAUNCH_CHECK();
    count_launch();
  }
  a.list = lists[1];
  a.kind = 1;
  Scratch<uint32_t> table;
  if (max_dv > (uint32_t)kSmallSlots / 2) {  // above: a block per chunk
    static std::mutex mu;
    static int cache[64] = {0};
    const size_t smem = (size_t)2 * kTcMidSlots * sizeof(uint32_t);
    const int per_sm = tc_blocks_per_sm(tc_middle_block_k<kWarpsB>, kWarpsB * 32, smem, dev, cache, mu);
    const unsigned blocks = (unsigned)(per_sm * sm_count(dev));
    uint32_t slots = 1;
    while (slots < 2ull * max_dv) slots <<= 1;
    if (max_dv > kTcMidSlots / 2) {  // keys empty (all ones), counts zero
      table.alloc((size_t)blocks * 2 * slots, s);
      fill_tables_k<<<grid_for((uint64_t)blocks * 2 * slots), kBlock, 0, s>>>(table.get(), blocks,
                                                                                slots);
      UG_LAUNCH_CHECK();
    }
    tc_middle_block_k<kWarpsB><<<blocks, kWarpsB * 32, smem, s>>>(a, table.get(), slots);
    UG_LAUNCH_CHECK();
    count_launch();
  }
  UG_CUDA(cudaStreamSynchronize(s));  // the scratch above is released on return
}

void clustering_run(TopoImpl* t, double* d_out, cudaStream_t s) {
  const uint64_t n = t->n;
  if (n == 0) return;
  Scratch<uint32_t> tri(n, s);
  triangle_count_run(t, tri.get(), s);
  clustering_k<<<grid_for(n), kBlock, 0, s>>>(t->und_off.get(), tri.get(), n, d_out);
  UG_LAUNCH_CHECK();
}

}  // namespace ug

using namespace ug;

extern "C" {

int ursa_gpu_triangle_count(ursa_gpu_topo* t, uint32_t* out) {
  return guard([&] {
    UG_CHECK(t, URSA_GPU_EINVAL, "topology is NULL");
    TopoImpl* ti = &t->impl;
    if (ti->n == 0) return;  // triangle.rs:56-58
    UG_CHECK(out, URSA_GPU_EINVAL, "out is NULL");
    cudaStream_t s = thread_stream(ti->device);
    Scratch<uint32_t> d(ti->n, s);
    triangle_count_run(ti, d.get(), s);
    UG_CUDA(cudaMemcpyAsync(out, d.get(), ti->n * 4, cudaMemcpyDeviceToHost, s));
    UG_CUDA(cudaStreamSynchronize(s));
  });
}

int ursa_gpu_clustering_coefficient(ursa_gpu_topo* t, double* out) {
  return guard([&] {
    UG_CHECK(t, URSA_GPU_EINVAL, "topology is NULL");
    TopoImpl* ti = &t->impl;
    if (ti->n == 0) return;  // clustering.rs:23-25
    UG_CHECK(out, URSA_GPU_EINVAL, "out is NULL");
    cudaStream_t s = thread_stream(ti->device);
    Scratch<double> d(ti->n, s);
    clustering_run(ti, d.get(), s);
    UG_CUDA(cudaMemcpyAsync(out, d.get(), ti->n * 8, cudaMemcpyDeviceToHost, s));
    UG_CUDA(cudaStreamSynchronize(s));
  });
}

}  // extern "C"
