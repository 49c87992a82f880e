// cc.cu -- weak connected components (ursa-core/src/algo/components.rs:14-68).
//
// The reference runs a serial union-find (path halving, union by rank) over
// the out-edges and labels each node with its representative.  Here the
// lock-free union-find of unionfind.cuh links trees so that each root is the
// minimum id of its component, so the final labels are the minimum member
// ids: the reference's partition with a canonical representative.
//
// A pass that unites every edge is bound by its finds: two dependent random
// reads per edge, almost all of which learn that both ends already share a
// tree (1,813 us of a 2,168 us call on R-MAT-22, 65M edges).  So the edges
// of the component that holds most of them are not visited (Sutton, Ben-Nun
// and Barak's sampling scheme, "Optimizing Parallel Graph Connectivity
// Computation via Subgraph Sampling"): every node first links to a few of
// its neighbours, the root that owns most edges is found by sampling, and
// then only nodes outside that root's tree walk their edges, along both
// CSRs -- an edge with an end outside is seen from that end, and one with
// both ends inside joins nothing.  R-MAT-22's kernels took 1,859 us and take
// about 380 (270 of them the second link's finds); the rest of a 677 us call is
// the labels' copy to the host.
#include "frontier.cuh"
#include "unionfind.cuh"

namespace ug {

namespace {

constexpr uint32_t kNoGiant = 0xFFFFFFFFu;
// Fewer edges than this take the pass over all slots at once, which is four
// launches fewer: 70,000 edges 78 us against 89 sampled, a million 193 against
// 153.  So do graphs of fewer edges than three quarters of their nodes, whose
// passes over the nodes are most of the work: four million nodes with two
// million edges 154 us of kernels against 287, with four million 624 and 503.
constexpr uint64_t kSampleEdges = 1u << 18;
constexpr uint32_t kLinkMin = 8;      // first link: the smallest of these many out-neighbours
constexpr uint32_t kLinkMore = 1;     // second link: this many neighbours united (2: 743 us a call, 1: 732)
constexpr unsigned kRuns = 148u * 8u; // blocks of the passes that take nodes in runs
constexpr uint32_t kSamples = 1024;   // edges whose roots are sampled
constexpr uint32_t kLaneEdges = 16;   // rows up to this are walked by their lane
constexpr uint32_t kWarpEdges = 4096; // ... up to this by the warp; longer ones by slot

// Words shared by the passes of one call: the sampled root (kNoGiant: none
// owns enough) and whether a row was left to the pass over all slots.
struct CcCtl {
  uint32_t giant, by_slot;
};

// First link, without atomics: parent[v] = the smallest of v and its first
// out-neighbours (or in-neighbours if it has none); parent ids only go down, so
// this is a forest.  The neighbours are one or two 32-byte sectors.
// Where neighbours have close ids (a path, a ring) its trees would be chains
// that the finds of the next pass walk.  So a link inside a tile of kBlock nodes
// is followed to its end by the block that stores it, and a node with no smaller
// out-neighbour takes its first in-neighbour if that one is in the tile; a chain
// is no longer than two links a tile.  (A path of two million nodes from high
// ids to low ones: 1,700 us of finds in one chain, the old pass over all edges
// 990; a ring with 8 neighbours a side 500 and 430.)
__global__ void __launch_bounds__(kBlock) cc_first_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                                                     const uint32_t* __restrict__ in_off,
                                                     const uint32_t* __restrict__ in_tgt, uint64_t n,
                                                     uint32_t* __restrict__ parent) {
  __shared__ volatile uint32_t tile[kBlock];
  for (uint64_t first = (uint64_t)blockIdx.x * kBlock; first < n; first += (uint64_t)gridDim.x * kBlock) {
    const uint64_t v = first + threadIdx.x;
    uint32_t best = 0;
    if (v < n) {
      uint32_t b = off[v], e = off[v + 1];
      const uint32_t* t = tgt;
      if (b == e && in_off) {
        b = in_off[v];
        e = in_off[v + 1];
        t = in_tgt;
      }
      best = (uint32_t)v;
      const uint32_t k = min(e - b, kLinkMin);
#pragma unroll
      for (uint32_t j = 0; j < kLinkMin; j++)
        if (j < k) best = min(best, t[b + j]);
      if (best == v && in_off && t == tgt && in_off[v] != in_off[v + 1]) {
        const uint32_t w = in_tgt[in_off[v]];
        if (w < v && w >= first) best = w;
      }
    }
    bool more = v < n && best < v && best >= first;
    if (__syncthreads_or(more)) {
      tile[threadIdx.x] = best;
      do {
        __syncthreads();
        if (more) {
          const uint32_t q = tile[best - first];
          more = q != best;
          best = q;
          tile[threadIdx.x] = q;
          more = more && q >= first;
        }
      } while (__syncthreads_or(more));
    }
    if (v < n) parent[v] = best;
  }
}

// A block's own run of the n nodes: [first, last).  The linking passes take
// nodes in runs: a grid-wide stride links a whole wave of consecutive nodes
// at once, which on a path (or a road grid) is one chain as long as the wave,
// and every find walks it (89 ms at a million nodes; 1 ms in runs).
__device__ __forceinline__ void cc_run(uint64_t n, uint64_t& first, uint64_t& last) {
  const uint64_t per = (n + gridDim.x - 1) / gridDim.x;
  first = min(n, blockIdx.x * per);
  last = min(n, first + per);
}

// Second link: the first neighbours of each row united.
__global__ void cc_link_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                          const uint32_t* __restrict__ in_off, const uint32_t* __restrict__ in_tgt,
                          uint64_t n, uint32_t* parent) {
  uint64_t first, last;
  cc_run(n, first, last);
  for (uint64_t v = first + threadIdx.x; v < last; v += blockDim.x) {
    uint32_t b = off[v], e = off[v + 1];
    const uint32_t* t = tgt;
    if (b == e && in_off) {
      b = in_off[v];
      e = in_off[v + 1];
      t = in_tgt;
    }
    const uint32_t k = min(e - b, kLinkMore);
    for (uint32_t j = 0; j < k; j++) {
      const uint32_t w = t[b + j];
      if (w != (uint32_t)v) uf_unite<true>(parent, (uint32_t)v, w);
    }
  }
}

__global__ void cc_compress_k(uint32_t* parent, uint64_t n) {
  uint64_t first, last;
  cc_run(n, first, last);
  for (uint64_t v = first + threadIdx.x; v < last; v += blockDim.x)
    uf_find_l1(parent, (uint32_t)v);  // stores what it finds
}

// One block: the roots of kSamples edges' targets (a fixed stride over the
// slots, so a root is met in proportion to the edges it owns), counted in a
// hash table.  The most frequent one is the giant if it owns at least half of
// the sample: walking both directions of the other rows then reads no more
// than the one pass over all out-edges that is taken otherwise.
__global__ void __launch_bounds__(kSamples) cc_sample_k(const uint32_t* __restrict__ tgt, uint64_t m,
                                                        const uint32_t* __restrict__ parent,
                                                        bool have_in, CcCtl* ctl) {
  constexpr uint32_t kSlots = 2 * kSamples;
  __shared__ uint32_t key[kSlots];
  __shared__ uint32_t cnt[kSlots];
  for (uint32_t i = threadIdx.x; i < kSlots; i += kSamples) {
    key[i] = kNoGiant;
    cnt[i] = 0;
  }
  __shared__ uint32_t s_best, s_root;
  if (threadIdx.x == 0) {
    s_best = 0;
    s_root = kNoGiant;
  }
  __syncthreads();
  const uint64_t k = m <= kSamples ? threadIdx.x : (m / kSamples) * threadIdx.x;
  const uint32_t taken = (uint32_t)(m < kSamples ? m : kSamples);
  uint32_t h = 0;
  if (k < m) {
    const uint32_t r = parent[tgt[k]];
    h = (r * 0x9E3779B1u) >> 21;
    for (;; h = (h + 1) & (kSlots - 1)) {
      const uint32_t old = atomicCAS(&key[h], kNoGiant, r);
      if (old == kNoGiant || old == r) break;
    }
    atomicAdd(&cnt[h], 1u);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < kSlots; i += kSamples)
    if (cnt[i]) atomicMax(&s_best, cnt[i]);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < kSlots; i += kSamples)
    if (cnt[i] && cnt[i] == s_best) s_root = key[i];
  __syncthreads();
  if (threadIdx.x == 0) {
    const bool giant = have_in && 2 * s_best >= taken;
    ctl->giant = giant ? s_root : kNoGiant;
    ctl->by_slot = giant ? 0u : 1u;
  }
}

// Rows outside the giant's tree walk their edges, out and in.  A pointer to
// the giant is read as it stands: a node that ever pointed there is in that
// component, whatever the other threads link meanwhile.
__global__ void cc_rest_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                          const uint32_t* __restrict__ in_off, const uint32_t* __restrict__ in_tgt,
                          uint64_t n, uint32_t* parent, CcCtl* ctl) {
  const uint32_t giant = ctl->giant;
  if (giant == kNoGiant) return;
  const int lane = threadIdx.x & 31;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t base = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; base < n;
       base += warps * 32) {
    const uint64_t v = base + lane;
    const bool outside = v < n && uf_parent(parent, (uint32_t)v) != giant;
    uint32_t b0 = 0, d0 = 0, b1 = 0, d1 = 0;
    if (outside) {
      b0 = off[v];
      d0 = off[v + 1] - b0;
      b1 = in_off[v];
      d1 = in_off[v + 1] - b1;
    }
    const uint64_t deg = (uint64_t)d0 + d1;
    if (deg <= kLaneEdges)
      for (uint32_t j = 0; j < (uint32_t)deg; j++) {
        const uint32_t w = j < d0 ? tgt[b0 + j] : in_tgt[b1 + j - d0];
        if (w != (uint32_t)v) uf_unite<true>(parent, (uint32_t)v, w);
      }
    if (deg > kWarpEdges) ctl->by_slot = 1u;
    unsigned todo = __ballot_sync(0xffffffffu, deg > kLaneEdges && deg <= kWarpEdges);
    while (todo) {
      const int l = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint32_t x = (uint32_t)(base + l);
      const uint32_t xb0 = __shfl_sync(0xffffffffu, b0, l), xd0 = __shfl_sync(0xffffffffu, d0, l);
      const uint32_t xb1 = __shfl_sync(0xffffffffu, b1, l), xd1 = __shfl_sync(0xffffffffu, d1, l);
      for (uint32_t j = lane; j < xd0; j += 32) {
        const uint32_t w = tgt[xb0 + j];
        if (w != x) uf_unite<true>(parent, x, w);
      }
      for (uint32_t j = lane; j < xd1; j += 32) {
        const uint32_t w = in_tgt[xb1 + j];
        if (w != x) uf_unite<true>(parent, x, w);
      }
      __syncwarp();
    }
  }
}

// Every out-edge that the giant does not hold on both ends, one thread per
// slot: only when no root owns half of the edges, or a row outside the giant
// is too long for a warp (balanced whatever the degrees).
template <bool kL1>
__global__ void cc_slots_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                           uint64_t n, uint64_t m, uint32_t* parent, const CcCtl* ctl) {
  if (ctl && !ctl->by_slot) return;
  const uint32_t giant = ctl ? ctl->giant : kNoGiant;
  for_each_slot_owner(off, n, m, [&](uint64_t k, uint32_t u) {
    const uint32_t v = tgt[k];
    if (u == v) return;
    if (giant != kNoGiant && uf_parent(parent, u) == giant && uf_parent(parent, v) == giant) return;
    uf_unite<kL1>(parent, u, v);
  });
}

__global__ void iota_k(uint32_t* p, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    p[i] = (uint32_t)i;
}

__global__ void flatten_k(uint32_t* parent, uint64_t n, uint32_t* __restrict__ out) {
  uint64_t first, last;
  cc_run(n, first, last);
  for (uint64_t i = first + threadIdx.x; i < last; i += blockDim.x) {
    out[i] = uf_find_l1(parent, (uint32_t)i);
  }
}

}  // namespace

// The whole call with a caller-supplied parent array (n u32, overwritten);
// allocates nothing: the passes' control words sit in d_out, which the last
// pass overwrites.
void cc_weak_with_parent(TopoImpl* t, uint32_t* parent, uint32_t* d_out, cudaStream_t s) {
  const uint64_t n = t->n, m = t->m;
  if (n == 0) return;
  if (n == 1) {
    UG_CUDA(cudaMemsetAsync(d_out, 0, sizeof(uint32_t), s));
    return;
  }
  const uint32_t *off = t->out.off.get(), *tgt = t->out.tgt.get();
  const uint32_t* in_off = t->has_in ? t->in.off.get() : nullptr;
  const uint32_t* in_tgt = t->has_in ? t->in.tgt.get() : nullptr;
  CcCtl* ctl = reinterpret_cast<CcCtl*>(d_out);
  if (m < kSampleEdges || m < n / 4 * 3) {
    iota_k<<<grid_for(n), kBlock, 0, s>>>(parent, n);
    UG_LAUNCH_CHECK();
    if (m) {
      // finds past L1 where trees stay small (four million nodes, two million edges: 155 us, 163 through L1)
      auto slots = m < kSampleEdges ? cc_slots_k<true> : cc_slots_k<false>;
      slots<<<grid_for(m, kBlock, 148u * 64u), kBlock, 0, s>>>(off, tgt, n, m, parent, nullptr);
      UG_LAUNCH_CHECK();
    }
  } else {
    cc_first_k<<<grid_for(n), kBlock, 0, s>>>(off, tgt, in_off, in_tgt, n, parent);
    UG_LAUNCH_CHECK();
    cc_link_k<<<grid_for(n, kBlock, kRuns), kBlock, 0, s>>>(off, tgt, in_off, in_tgt, n, parent);
    UG_LAUNCH_CHECK();
    cc_compress_k<<<grid_for(n, kBlock, kRuns), kBlock, 0, s>>>(parent, n);
    UG_LAUNCH_CHECK();
    cc_sample_k<<<1, kSamples, 0, s>>>(tgt, m, parent, in_off != nullptr, ctl);
    UG_LAUNCH_CHECK();
    cc_rest_k<<<grid_for(n), kBlock, 0, s>>>(off, tgt, in_off, in_tgt, n, parent, ctl);
    UG_LAUNCH_CHECK();
    cc_slots_k<true><<<grid_for(m, kBlock, 148u * 64u), kBlock, 0, s>>>(off, tgt, n, m, parent, ctl);
    UG_LAUNCH_CHECK();
  }
  flatten_k<<<grid_for(n, kBlock, kRuns), kBlock, 0, s>>>(parent, n, d_out);
  UG_LAUNCH_CHECK();
}

void cc_weak_run(TopoImpl* t, uint32_t* d_out, cudaStream_t s) {
  if (t->n == 0) return;
  Scratch<uint32_t> parent(t->n, s);
  cc_weak_with_parent(t, parent.get(), d_out, s);
}

}  // namespace ug

using namespace ug;

extern "C" int ursa_gpu_connected_components_weak(ursa_gpu_topo* t, uint32_t* out) {
  return guard([&] {
    UG_CHECK(t, URSA_GPU_EINVAL, "topology is NULL");
    TopoImpl* ti = &t->impl;
    if (ti->n == 0) return;
    UG_CHECK(out, URSA_GPU_EINVAL, "out is NULL");
    cudaStream_t s = thread_stream(ti->device);
    Scratch<uint32_t> d(ti->n, s);
    cc_weak_run(ti, d.get(), s);
    UG_CUDA(cudaMemcpyAsync(out, d.get(), ti->n * 4, cudaMemcpyDeviceToHost, s));
    UG_CUDA(cudaStreamSynchronize(s));
  });
}
