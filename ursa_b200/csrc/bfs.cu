// bfs.cu -- bfs_distances from one source (ursa-core/src/algo/bfs.rs:18-42).
//
// Level-synchronous and direction-optimising (Beamer et al.); levels are
// exact, so the output is bit-identical to the reference's serial BFS.  A
// level is ONE launch that reads what to do from device memory, and its last
// block to finish decides the next level's way, so levels are enqueued
// several at a time and the host reads one word per run of them: with a
// prefix scan of the frontier's degrees and a host read per level, three
// quarters of a call on 50,000 nodes was launches and round trips (297 us for
// 70 us of kernels; 101 us now).  R-MAT-22 takes 619 us against 875, 305 of
// them the distances' copy to the host; its pull levels read every unvisited
// node's row up to its first parent and are bound by those random reads.
//
// A level goes one of three ways:
//   list: the frontier is a list of (node, first slot) entries of at most
//     kSpan edges each (a hub is many entries), a lane per edge; new
//     nodes are appended as entries (CAS on dist);
//   pull: every unvisited node looks for a neighbour on the last level, four
//     at a time; only counts are kept;
//   scan: the first top-down level after pulling: nodes on the last level are
//     found by scanning dist, 32 at a time, and expanded as they are found.
#include <algorithm>

#include "frontier.cuh"

namespace ug {

namespace {

constexpr uint32_t kLongRow = 1024;  // scan: rows above are walked by the block
constexpr uint32_t kLongList = 64;
constexpr double kAlpha = 14.0, kBeta = 24.0;
constexpr int kBfsBlocks = 8;  // per SM
// The grid has a thread per node, or per this many edges: a level's list can
// hold them all (256 nodes, 50M edges: 951 us with one block, 123 so).
constexpr uint64_t kBfsLaneEdges = 64;

enum Mode : uint32_t { kList = 0, kPull = 1, kScan = 2, kDone = 3 };

struct BfsState {
  uint32_t mode;
  int32_t level;  // of the frontier
  uint32_t entries[2];  // frontier entries, by level parity
  unsigned ticket;
  uint32_t limit;  // entries from which the next level is a pull
  unsigned long long f, left;          // the frontier's nodes; edges not yet walked from
  unsigned long long next_f, next_T;   // being counted: the next frontier's nodes and edges
};

struct BfsArgs {
  DirView fw, rv;
  uint64_t n;
  int32_t* dist;
  uint2* list[2];  // by level parity
  BfsState* st;
};

// With this many entries the next frontier's edges pass left / kAlpha (at most
// one entry a node is not full), so it is pulled and nobody reads its list.
// (256 nodes, 50M edges, both directions: 257 us with all of them written, a
// warp a hub, 150 so.)
__device__ __forceinline__ uint32_t bfs_limit(uint64_t n, unsigned long long left) {
  return (uint32_t)min(0xFFFFFFFFull, n + left / (unsigned long long)(kAlpha * kSpan) + 2ull);
}

__global__ void bfs_init_k(BfsArgs a, uint32_t source, unsigned long long edges) {
  const uint32_t deg = dv_deg(a.fw, source);
  const uint32_t k = (deg + kSpan - 1) / kSpan;
  for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) a.list[0][i] = make_uint2(source, i * kSpan);
  if (threadIdx.x) return;
  a.dist[source] = 0;
  BfsState s{};
  const bool pull = (double)deg > (double)edges / kAlpha;
  s.mode = deg == 0 ? kDone : pull ? kPull : kList;
  s.entries[0] = k;
  s.f = 1;
  s.left = edges - (pull ? 0 : deg);
  s.limit = bfs_limit(a.n, s.left);
  *a.st = s;
}

// One step of a warp along edges: every lane has a neighbour w (or none).
__device__ __forceinline__ void bfs_visit(const BfsArgs& a, int32_t level, uint32_t limit, bool have, uint32_t w,
                                          unsigned long long& f, unsigned long long& T) {
  bool take = false;
  uint32_t deg = 0;
  if (have && a.dist[w] < 0) take = atomicCAS(&a.dist[w], -1, level + 1) == -1;
  if (take) {
    deg = dv_deg(a.fw, w);
    f++;
    T += deg;
  }
  append_entries(a.list[(level + 1) & 1], &a.st->entries[(level + 1) & 1], take, w, deg, limit);
}

__global__ void __launch_bounds__(kBlock) bfs_level_k(BfsArgs a) {
  const uint32_t FULL = 0xffffffffu;
  const BfsState* sp = a.st;
  const uint32_t mode = sp->mode;
  if (mode == kDone) return;
  const int32_t level = sp->level;
  const int lane = threadIdx.x & 31;
  const uint64_t gtid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nthr = (uint64_t)gridDim.x * blockDim.x;
  unsigned long long f = 0, T = 0;  // this thread's new nodes and their edges
  const uint32_t limit = sp->limit;
  if (mode == kList) {
    const uint32_t count = sp->entries[level & 1];
    const uint2* list = a.list[level & 1];
    const uint32_t sub = threadIdx.x & (kEntryLanes - 1);
    const uint64_t per_grid = nthr / kEntryLanes;
    const uint64_t rounds = (count + per_grid - 1) / per_grid;  // whole warps step together
    for (uint64_t r = 0; r < rounds; r++) {
      const uint64_t i = r * per_grid + gtid / kEntryLanes;
      uint32_t u = 0, j = 0, end = 0;
      if (i < count) {
        const uint2 e = list[i];
        u = e.x;
        j = e.y + sub;
        end = min(dv_deg(a.fw, u), e.y + kSpan);
      }
      while (__any_sync(FULL, j < end)) {
        const bool have = j < end;
        bfs_visit(a, level, limit, have, have ? dv_nbr(a.fw, u, j) : 0u, f, T);
        j += kEntryLanes;
      }
    }
  } else if (mode == kPull) {
    for (uint64_t v = gtid; v < a.n; v += nthr) {
      if (a.dist[v] >= 0) continue;
      bool found = false;
      for (int part = 0; part < 2 && !found; part++) {
        const uint32_t* off = part ? a.rv.off1 : a.rv.off0;
        const uint32_t* tgt = part ? a.rv.tgt1 : a.rv.tgt0;
        if (!off) break;
        uint32_t k = off[v];
        const uint32_t e = off[v + 1];
        // the first neighbour alone (it decides most nodes on a full level), then four in flight
        if (k < e) found = a.dist[tgt[k++]] == level;
        for (; k < e && !found; k += 4) {
          uint32_t u[4];
#pragma unroll
          for (int q = 0; q < 4; q++) u[q] = tgt[min(k + q, e - 1)];
          int32_t d[4];
#pragma unroll
          for (int q = 0; q < 4; q++) d[q] = a.dist[u[q]];
          found = d[0] == level || d[1] == level || d[2] == level || d[3] == level;
        }
      }
      if (found) {
        a.dist[v] = level + 1;
        f++;
        T += dv_deg(a.fw, (uint32_t)v);
      }
    }
  } else {
    __shared__ uint32_t longs[kLongList];
    __shared__ unsigned n_long;
    if (threadIdx.x == 0) n_long = 0;
    __syncthreads();
    const uint64_t span = (a.n + nthr - 1) / nthr * nthr;
    for (uint64_t v = gtid; v < span; v += nthr) {
      uint32_t deg = 0;
      if (v < a.n && a.dist[v] == level) deg = dv_deg(a.fw, (uint32_t)v);
      if (deg > kLongRow) {
        const unsigned at = atomicAdd(&n_long, 1u);
        if (at < kLongList) {
          longs[at] = (uint32_t)v;
          deg = 0;
        }
      }
      for (uint32_t todo = __ballot_sync(FULL, deg != 0); todo; todo &= todo - 1) {
        const int l = __ffs(todo) - 1;
        const uint32_t u = __shfl_sync(FULL, (uint32_t)v, l), d = __shfl_sync(FULL, deg, l);
        for (uint32_t j0 = 0; j0 < d; j0 += 32) {
          const bool have = j0 + lane < d;
          bfs_visit(a, level, limit, have, have ? dv_nbr(a.fw, u, j0 + lane) : 0u, f, T);
        }
      }
    }
    __syncthreads();
    const unsigned listed = min(n_long, kLongList);
    for (unsigned i = 0; i < listed; i++) {
      const uint32_t u = longs[i], d = dv_deg(a.fw, u);
      for (uint32_t j0 = 0; j0 < d; j0 += blockDim.x) {
        const bool have = j0 + threadIdx.x < d;
        bfs_visit(a, level, limit, have, have ? dv_nbr(a.fw, u, j0 + threadIdx.x) : 0u, f, T);
      }
    }
  }
  // the block's counts, and the last block's decision
  __shared__ unsigned long long sums[2][kBlock / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    f += __shfl_down_sync(FULL, f, o);
    T += __shfl_down_sync(FULL, T, o);
  }
  if (lane == 0) {
    sums[0][threadIdx.x >> 5] = f;
    sums[1][threadIdx.x >> 5] = T;
  }
  __syncthreads();
  if (threadIdx.x) return;
  f = T = 0;
  for (int w = 0; w < kBlock / 32; w++) {
    f += sums[0][w];
    T += sums[1][w];
  }
  BfsState* s = a.st;
  if (f) {
    atomicAdd(&s->next_f, f);
    atomicAdd(&s->next_T, T);
  }
  __threadfence();
  if (atomicAdd(&s->ticket, 1u) != gridDim.x - 1) return;
  __threadfence();
  const unsigned long long nf = __ldcg(&s->next_f), nT = __ldcg(&s->next_T), left = s->left;
  // top-down while the frontier's edges are few, pull while its nodes are many
  bool pull = mode == kPull && !((double)nf < (double)a.n / kBeta && nf < s->f);
  if (!pull && (double)nT > (double)left / kAlpha) pull = true;
  s->mode = nf == 0 || nT == 0 ? kDone : pull ? kPull : mode == kPull ? kScan : kList;
  s->left = pull ? left : left - min(left, nT);
  s->limit = bfs_limit(a.n, s->left);
  s->f = nf;
  s->level = level + 1;
  s->entries[level & 1] = 0;  // the list after the next
  s->next_f = s->next_T = 0;
  s->ticket = 0;
}

}  // namespace

// Distances into d_dist (n i32) and from there into `out` (host, n i32).
void bfs_distances_run(TopoImpl* t, uint32_t source, int dir, int32_t* d_dist, int32_t* out,
                       cudaStream_t s) {
  const uint64_t n = t->n;
  if (n == 0) return;
  UG_CUDA(cudaMemsetAsync(d_dist, 0xFF, n * sizeof(int32_t), s));
  auto copy = [&] { UG_CUDA(cudaMemcpyAsync(out, d_dist, n * sizeof(int32_t), cudaMemcpyDeviceToHost, s)); };
  if ((uint64_t)source >= n) {  // bfs.rs:21-23
    copy();
    UG_CUDA(cudaStreamSynchronize(s));
    return;
  }
  const uint64_t edges = t->m * (dir == 2 ? 2 : 1);
  const uint64_t entries = n + edges / kSpan + 1;
  Scratch<uint2> list(2 * entries, s);
  Scratch<BfsState> st(1, s);
  BfsArgs a;
  a.fw = dir_view(t, dir, s);
  a.rv = reverse_view(t, dir, s);
  a.n = n;
  a.dist = d_dist;
  a.list[0] = list.get();
  a.list[1] = list.get() + entries;
  a.st = st.get();
  bfs_init_k<<<1, kBlock, 0, s>>>(a, source, edges);
  UG_LAUNCH_CHECK();
  const unsigned grid = grid_for(std::max(n, edges / kBfsLaneEdges), kBlock,
                                 (unsigned)sm_count(t->device) * kBfsBlocks);
  uint32_t mode = kList;
  for (int run = 8; mode != kDone; run = run < 64 ? 2 * run : run) {
    for (int i = 0; i < run; i++) {
      bfs_level_k<<<grid, kBlock, 0, s>>>(a);
      UG_LAUNCH_CHECK();
    }
    // a copy to pageable memory returns once it is done: the levels are over
    UG_CUDA(cudaMemcpyAsync(&mode, &st.get()->mode, sizeof(mode), cudaMemcpyDeviceToHost, s));
  }
  copy();
  UG_CUDA(cudaStreamSynchronize(s));
}

}  // namespace ug

using namespace ug;

extern "C" int ursa_gpu_bfs_distances(ursa_gpu_topo* t, uint32_t source, int dir, int32_t* out) {
  return guard([&] {
    UG_CHECK(t, URSA_GPU_EINVAL, "topology is NULL");
    UG_CHECK(dir >= 0 && dir <= 2, URSA_GPU_EINVAL, "direction must be 0, 1 or 2");
    TopoImpl* ti = &t->impl;
    if (ti->n == 0) return;
    UG_CHECK(out, URSA_GPU_EINVAL, "out is NULL");
    cudaStream_t s = thread_stream(ti->device);
    Scratch<int32_t> d(ti->n, s);
    bfs_distances_run(ti, source, dir, d.get(), out, s);
  });
}
