// bc.cu -- Brandes betweenness (ursa-core/src/algo/betweenness.rs, rng.rs).
//
// Sources: all nodes, or the reference's seeded sample -- the first
// ceil(frac * n) entries of a SplitMix64 Fisher-Yates shuffle
// (betweenness.rs:349-362, rng.rs:12-72) -- in exactly the reference's order
// for a given seed.
//
// Per source, on the device:
//  * unweighted (brandes_from, :185-230): level-synchronous BFS over the
//    out-CSR; sigma[w] += sigma[v] for every CSR slot v->w with
//    dist[w] = dist[v] + 1 (parallel edges count, as in the reference), as f64
//    atomics -- shortest-path counts are integers, exact below 2^53, so the
//    order of those additions does not matter;
//  * weighted (brandes_from_weighted, :278-339): Dijkstra-equivalent f64
//    distances (frontier Bellman-Ford), then the tight-edge DAG
//    (fl(dist[u] + w) == dist[v], exact equality as the reference's tie rule)
//    is walked in Kahn order to accumulate sigma;
//  * reverse accumulation (reverse_accumulate, :81-98): levels in reverse,
//    one warp per node sums sigma[v] * ((1 + delta[w]) / sigma[w]) over its
//    DAG successors with a fixed-order reduction, then bc += delta (source
//    excluded).
// Sources go in 64-source chunks whose partial vectors are added in chunk
// order, and sampled results are scaled by n / k (accumulate_sources,
// :45-70; :171-176).  The dependency sums run in a different order than the
// reference's predecessor lists, so results agree to f64 rounding.
#include <algorithm>
#include <cmath>
#include <vector>

#include "frontier.cuh"

namespace ug {

void sssp_run(const DirView& d, const double* w0, const double* w1, uint64_t n, uint64_t m,
              uint32_t source, unsigned long long* dist, cudaStream_t s);

namespace {

constexpr unsigned long long kInfBits = 0x7FF0000000000000ull;
constexpr uint32_t kSrcChunk = 64;  // betweenness.rs:51
constexpr bool kBatchedWeighted = true;  // weighted sources 64 at a time (else one by one)

// ---------------------------------------------------------------- rng.rs
constexpr uint64_t kDefaultSeed = 0x5EED5EED5EED5EEDull;  // rng.rs:9

constexpr uint64_t kGamma = 0x9E3779B97F4A7C15ull;

// The shuffle's swap partner of position i (rng.rs:64-72: i from n - 1 down to
// 1).  SplitMix64's state is a counter, so any step can be computed alone.
__host__ __device__ __forceinline__ uint64_t shuffle_partner(uint64_t state, uint64_t n, uint64_t i) {
  uint64_t z = state + (n - i) * kGamma;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return (z ^ (z >> 31)) % (i + 1);
}

// Followed backwards, from step 1 up, what ends at one of the first k
// positions came from position x, until the first step i > x whose partner is
// x; it came from i then.  One pass finds that step for every x, and the k
// chains, of about ln(n / k) steps each, are walked.  The n swaps one after
// another took 3.8 ms at a million nodes, a tenth of a 256-source call.
// Fewer steps than this run on the host (a one-source call on 32,760 nodes 194 us
// so, on 32,900 by the device 130; about equal at half of that).
constexpr uint64_t kShuffleMin = 1u << 15;

__global__ void shuffle_steps_k(uint64_t state, uint64_t n, uint64_t k, uint32_t* __restrict__ next) {
  for (uint64_t i = k + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t j = shuffle_partner(state, n, i);
    if (j != i) atomicMin(&next[j], (uint32_t)i);
  }
}

__global__ void shuffle_trace_k(uint64_t k, const uint32_t* __restrict__ next, uint32_t* __restrict__ from) {
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < k;
       p += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t x = (uint32_t)p, i;
    while ((i = next[x]) != 0xFFFFFFFFu) x = i;  // i > x
    from[p] = x;
  }
}

// sample_sources (betweenness.rs:349-362) with shuffled_order (rng.rs:64-72).
std::vector<uint32_t> sample_sources(uint64_t n, bool has_sample, double frac, bool has_seed,
                                     uint64_t seed, cudaStream_t s) {
  std::vector<uint32_t> out;
  if (!has_sample) {
    out.resize(n);
    for (uint64_t i = 0; i < n; i++) out[i] = (uint32_t)i;
    return out;
  }
  double f = frac;
  if (f < 0.0) f = 0.0;
  if (f > 1.0) f = 1.0;
  double kf = std::ceil((double)n * f);
  uint64_t k = (std::isnan(kf) || kf <= 0.0) ? 0 : (kf >= 1.8446744073709552e19 ? UINT64_MAX : (uint64_t)kf);
  if (k < 1) k = 1;
  if (k > n) k = n;
  if (k == 0) return out;
  const uint64_t st = (has_seed ? seed : kDefaultSeed) ^ 0xD1B54A32D192ED03ull;
  if (n - k < kShuffleMin) {
    std::vector<uint32_t> order(n);
    for (uint64_t i = 0; i < n; i++) order[i] = (uint32_t)i;
    for (uint64_t i = n; i-- > 1;) std::swap(order[i], order[shuffle_partner(st, n, i)]);
    out.assign(order.begin(), order.begin() + k);
    return out;
  }
  std::vector<uint32_t> from(k), at(k);  // at[x]: which of the k positions is traced to x by steps below k
  {
    Scratch<uint32_t> next(n, s), d_from(k, s);
    UG_CUDA(cudaMemsetAsync(next.get(), 0xFF, n * sizeof(uint32_t), s));
    shuffle_steps_k<<<grid_for(n - k), kBlock, 0, s>>>(st, n, k, next.get());
    UG_LAUNCH_CHECK();
    shuffle_trace_k<<<grid_for(k), kBlock, 0, s>>>(k, next.get(), d_from.get());
    UG_LAUNCH_CHECK();
    UG_CUDA(cudaMemcpyAsync(from.data(), d_from.get(), k * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    for (uint64_t i = 0; i < k; i++) at[i] = (uint32_t)i;
    for (uint64_t i = 1; i < k; i++) std::swap(at[i], at[shuffle_partner(st, n, i)]);
    UG_CUDA(cudaStreamSynchronize(s));
  }
  out.resize(k);
  for (uint64_t x = 0; x < k; x++) out[at[x]] = from[x];
  return out;
}

// ------------------------------------------------------------ kernels
__device__ __forceinline__ void append_bc(uint32_t* Q, uint32_t* cnt, bool take, uint32_t v) {
  uint32_t mask = __ballot_sync(0xffffffffu, take);
  if (!take) return;
  int lane = threadIdx.x & 31;
  int leader = __ffs(mask) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(cnt, (uint32_t)__popc(mask));
  base = __shfl_sync(mask, base, leader);
  Q[base + __popc(mask & ((1u << lane) - 1u))] = v;
}

__global__ void bfs_discover_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                               const uint32_t* __restrict__ F, uint64_t f,
                               const uint64_t* __restrict__ pos, uint64_t T, int32_t* dist,
                               int32_t level, uint32_t* __restrict__ N, uint32_t* __restrict__ cnt) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t span = ((T + stride - 1) / stride) * stride;
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < span; e += stride) {
    bool take = false;
    uint32_t v = 0;
    if (e < T) {
      uint64_t i = owner_in_pos(pos, f, e);
      v = tgt[off[F[i]] + (uint32_t)(e - pos[i])];
      if (dist[v] < 0) take = atomicCAS(&dist[v], -1, level + 1) == -1;
    }
    append_bc(N, cnt, take, v);
  }
}

__global__ void bfs_sigma_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                            const uint32_t* __restrict__ F, uint64_t f,
                            const uint64_t* __restrict__ pos, uint64_t T,
                            const int32_t* __restrict__ dist, int32_t level, double* sigma) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < T;
       e += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t i = owner_in_pos(pos, f, e);
    uint32_t u = F[i];
    uint32_t v = tgt[off[u] + (uint32_t)(e - pos[i])];
    if (dist[v] == level + 1) atomicAdd(&sigma[v], sigma[u]);
  }
}

__device__ __forceinline__ bool tight(const unsigned long long* __restrict__ dist, uint32_t u,
                                      uint32_t v, double w) {
  unsigned long long du = dist[u], dv = dist[v];
  if (du == kInfBits || u == v) return false;
  double nd = __dadd_rn(__longlong_as_double((long long)du), w);
  if ((unsigned long long)__double_as_longlong(nd) != dv) return false;
  return du < dv || (du == dv && u < v);  // zero weights: keep the DAG acyclic
}

// tight in-slot counts over every out-slot
__global__ void tight_indeg_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                              const double* __restrict__ w, uint64_t n, uint64_t m,
                              const unsigned long long* __restrict__ dist,
                              uint32_t* __restrict__ indeg) {
  for_each_slot_owner(off, n, m, [&](uint64_t k, uint32_t u) {
    uint32_t v = tgt[k];
    if (tight(dist, u, v, w[k])) atomicAdd(&indeg[v], 1u);
  });
}

__global__ void kahn_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                       const double* __restrict__ w, const uint32_t* __restrict__ F, uint64_t f,
                       const uint64_t* __restrict__ pos, uint64_t T,
                       const unsigned long long* __restrict__ dist, uint32_t* indeg, double* sigma,
                       uint32_t* __restrict__ N, uint32_t* __restrict__ cnt) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t span = ((T + stride - 1) / stride) * stride;
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < span; e += stride) {
    bool take = false;
    uint32_t v = 0;
    if (e < T) {
      uint64_t i = owner_in_pos(pos, f, e);
      uint32_t u = F[i];
      uint32_t k = off[u] + (uint32_t)(e - pos[i]);
      v = tgt[k];
      if (tight(dist, u, v, w[k])) {
        atomicAdd(&sigma[v], sigma[u]);
        take = atomicSub(&indeg[v], 1u) == 1u;
      }
    }
    append_bc(N, cnt, take, v);
  }
}

// One warp per node of the level: delta[v] = sum over DAG successors of
// sigma[v] * ((1 + delta[w]) / sigma[w]); bc[v] += delta[v] unless v == s.
template <bool kWeighted>
__global__ void dependency_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                             const double* __restrict__ w, const uint32_t* __restrict__ L,
                             uint64_t cnt, const int32_t* __restrict__ hop,
                             const unsigned long long* __restrict__ dist,
                             const double* __restrict__ sigma, double* delta, double* bc,
                             uint32_t source) {
  const int lane = threadIdx.x & 31;
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t i = warp; i < cnt; i += nwarps) {
    const uint32_t v = L[i];
    const double sv = sigma[v];
    double acc = 0.0;
    for (uint32_t k = off[v] + lane; k < off[v + 1]; k += 32) {
      const uint32_t x = tgt[k];
      bool succ = kWeighted ? tight(dist, v, x, w[k]) : (hop[x] == hop[v] + 1);
      if (succ) acc += __dmul_rn(sv, __ddiv_rn(__dadd_rn(1.0, delta[x]), sigma[x]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) {
      delta[v] = acc;
      if (v != source) bc[v] += acc;
    }
  }
}

__global__ void add_into_k(double* __restrict__ dst, const double* __restrict__ src, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    dst[i] = __dadd_rn(dst[i], src[i]);
}

__global__ void scale_k(double* __restrict__ x, uint64_t n, double s) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    x[i] = __dmul_rn(x[i], s);
}

__global__ void seed_source_k(int32_t* hop, double* sigma, uint32_t* L, uint32_t s) {
  if (hop) hop[s] = 0;
  sigma[s] = 1.0;
  L[0] = s;
}

__global__ void fdeg_out_k(const uint32_t* __restrict__ off, const uint32_t* __restrict__ F,
                           uint64_t f, uint64_t* __restrict__ pos) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= f;
       i += (uint64_t)gridDim.x * blockDim.x)
    pos[i] = i < f ? (uint64_t)(off[F[i] + 1] - off[F[i]]) : 0ull;
}

// ---- 64 sources at once (unweighted) -------------------------------------
// Batch b holds sources [64 b, 64 b + 64) of the source list, the
// reference's accumulation chunk (betweenness.rs:45-70).  Per node v the
// batch keeps a row of 64 f64 (node-major: lane l of a warp holds sources 2 l
// and 2 l + 1, one 16-byte access), and per level a mask of the sources that
// reach v there (bit q = source q).
//  forward level L: one warp per node v still missing some sources; over v's
//    in-edges u -> v in CSR order, the sources in front[u] & need reach v at
//    level L, sigma_q[v] += sigma_q[u] for each (per slot, as brandes_from
//    counts parallel edges);
//  backward level L (deepest first): one warp per node v with some source at
//    level L; over v's out-edges v -> w in CSR order, an edge is on the
//    shortest-path DAG of the sources in mask_L[v] & mask_L+1[w]:
//    delta_q[v] = sigma_q[v] * the sum of c_q[w], c = (1 + delta) / sigma
//    (reverse_accumulate, :81-98, summed per successor instead of per
//    predecessor list); c_q[v] then takes the place of sigma_q[v], which
//    nobody reads any more;
//  fold: per node, the batch's partial = sum over q in source order of
//    delta_q[v] (v != source q), added to the result in batch order.
// What bounds it is the rows: 512 bytes per edge and level that lies on some
// source's DAG, from HBM.  So a warp finds the edges with a source in common
// first (32 at a time, 8-byte masks that stay in L2) and has eight rows in
// flight; the masks per level take the place of a DAG mask per edge (a random
// read-modify-write per edge in the forward pass) and of a hop per (node,
// source), and c that of a second row and a division per edge and source.
// 256 sources on a Poisson graph of a million nodes, 16.8M edges: forward
// 15.8 ms against 37.4, backward 14.9 against 51.4; the deepest level, where
// most edges meet, moves 4.1 TB/s from DRAM forward and 6.3 backward.
constexpr int kBcB = 64;

struct BcBatchArgs {
  const uint32_t* in_off;
  const uint32_t* in_src;
  const uint32_t* in_to_out;  // in-CSR slot -> out-CSR slot of the same edge
  const uint32_t* out_off;
  const uint32_t* out_tgt;
  uint64_t n;
  uint64_t qmask;
  uint64_t* vis;
  const uint64_t* front;
  uint64_t* next;
  int32_t* hop;      // n x 64
  double* sigma;     // n x 64
  double* delta;     // n x 64
  uint64_t* dag;     // per out-CSR slot
  int32_t level;
  unsigned* found;
};

constexpr int kBcRows = 8;            // rows in flight per warp (4: 41.3 ms a call, 8: 40.8, 16: 42.9)
constexpr int kBcOcc = 4;             // blocks per SM: registers for those rows (3: 47.9 ms, 5: 42.4)
constexpr uint32_t kBcLong = 1024;     // longer rows are walked by the whole block
constexpr int kBcLongList = 32;        // ... as many as it can list; the rest by their warp
constexpr int kBcWarps = kBlock / 32;
constexpr uint32_t kBcNone = 0xFFFFFFFFu;
constexpr uint32_t kBcGroup = 32;      // most nodes a warp takes at a time
// Mask levels kept, in no more memory than a hop per (node, source) takes;
// deeper searches (roads, chains) go on from there with bc_forward_k, and
// later batches of the call take it from the start.
constexpr size_t kBcMaxLevels = 32;

struct BcLevelArgs {
  const uint32_t* off;   // forward: the in-CSR; backward: the out-CSR
  const uint32_t* adj;
  uint64_t n;
  uint64_t qmask;
  uint64_t* vis;          // forward
  const uint64_t* front;  // forward: masks of the last level; backward: of the next one
  uint64_t* mask;         // this level's masks (forward: written)
  double* row;            // n x 64: sigma, then c
  double* delta;          // n x 64 (backward)
  unsigned* found;
  uint32_t group;         // nodes a warp takes at a time
};

// Two f64 of a row past L1, or zeros without the predicate.  Volatile, so that
// a warp's eight loads are issued before the first sum waits for one.
__device__ __forceinline__ double2 bc_load(const double* p, bool take) {
  double2 r;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %3, 0;\n\t"
      "mov.f64 %0, 0d0000000000000000;\n\t"
      "mov.f64 %1, 0d0000000000000000;\n\t"
      "@p ld.global.cg.v2.f64 {%0, %1}, [%2];\n\t}"
      : "=d"(r.x), "=d"(r.y)
      : "l"(p), "r"((uint32_t)take));
  return r;
}

// A warp's list of the edges of a step that share a source: the neighbour and
// the sources shared (two words: lanes 0..15 hold sources 0..31).
struct BcStep {
  uint32_t f[32 + kBcRows][2];
  uint32_t u[32 + kBcRows];
};

// Adds, in order, the rows of a step of up to 32 edges (a lane each: the
// neighbour u and the sources f it shares) into every lane's two sums.
__device__ __forceinline__ void bc_add_step(BcStep& st, uint32_t u, uint64_t f, const double* row,
                                            double2& sum) {
  const uint32_t FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint32_t some = __ballot_sync(FULL, f != 0);
  if (!some) return;
  const int count = __popc(some);
  if (f) {
    const int at = __popc(some & ((1u << lane) - 1u));
    st.f[at][0] = (uint32_t)f;
    st.f[at][1] = (uint32_t)(f >> 32);
    st.u[at] = u;
  }
  if (lane < kBcRows) st.f[count + lane][0] = st.f[count + lane][1] = 0;  // the last rows, unused
  __syncwarp();
  const int word = lane >> 4, shift = 2 * (lane & 15);
  for (int j0 = 0; j0 < count; j0 += kBcRows) {
    double2 r[kBcRows];
    uint32_t bits[kBcRows];
#pragma unroll
    for (int j = 0; j < kBcRows; j++) {
      bits[j] = (st.f[j0 + j][word] >> shift) & 3u;
      r[j] = bc_load(row + (uint64_t)st.u[j0 + j] * kBcB + 2 * lane, bits[j] != 0);
    }
#pragma unroll
    for (int j = 0; j < kBcRows; j++) {
      sum.x = __dadd_rn(sum.x, bits[j] & 1u ? r[j].x : 0.0);
      sum.y = __dadd_rn(sum.y, bits[j] & 2u ? r[j].y : 0.0);
    }
  }
  __syncwarp();
}

// The same over adj[k], k in [b, e), for the sources in mask[adj[k]] & need;
// adds the sources met to the lane's own `met`.
__device__ __forceinline__ void bc_add_rows(BcStep& st, const uint32_t* __restrict__ adj,
                                            const uint64_t* __restrict__ mask, const double* row,
                                            uint32_t b, uint32_t e, uint64_t need, uint64_t& met,
                                            double2& sum) {
  const int lane = threadIdx.x & 31;
  for (uint32_t k0 = b; k0 < e; k0 += 32) {
    uint32_t u = 0;
    uint64_t f = 0;
    if (k0 + lane < e) {
      u = adj[k0 + lane];
      f = mask[u] & need;
    }
    met |= f;
    bc_add_step(st, u, f, row, sum);
  }
}

__device__ __forceinline__ uint64_t bc_or(uint64_t met) {
  return ((uint64_t)__reduce_or_sync(0xffffffffu, (uint32_t)(met >> 32)) << 32) |
         __reduce_or_sync(0xffffffffu, (uint32_t)met);
}

// A warp's nodes, one per lane: need (sources wanted, 0: nothing to do) and
// edges [b, e) of each.  settle(l, need, met, sum) takes the result of lane
// l's node, in lane order (met: per lane, to be ORed over the warp).  The
// next node's neighbours are loaded while a node's rows are added.
template <class Settle>
__device__ __forceinline__ void bc_nodes(const BcLevelArgs& A, BcStep& st, uint64_t need, uint32_t b,
                                         uint32_t e, Settle&& settle) {
  const uint32_t FULL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31;
  uint32_t todo = __ballot_sync(FULL, need != 0);
  uint32_t u1 = kBcNone, b1 = 0, e1 = 0;
  int l1 = -1;
  auto next = [&]() {
    l1 = __ffs(todo) - 1;  // -1 after the last
    todo &= todo - 1;
    b1 = __shfl_sync(FULL, b, l1 & 31);
    e1 = l1 >= 0 ? __shfl_sync(FULL, e, l1 & 31) : b1;
    u1 = lane < e1 - b1 ? A.adj[b1 + lane] : kBcNone;
  };
  next();
  while (l1 >= 0) {
    const int l = l1;
    const uint32_t u = u1, lb = b1, le = e1;
    const uint64_t ln = __shfl_sync(FULL, need, l);
    const uint64_t f = u != kBcNone ? A.front[u] & ln : 0ull;
    next();
    uint64_t met = f;
    double2 sum = make_double2(0.0, 0.0);
    bc_add_step(st, u, f, A.row, sum);
    if (le - lb > 32) bc_add_rows(st, A.adj, A.front, A.row, lb + 32, le, ln, met, sum);
    settle(l, ln, met, sum);
  }
}

// The same over one long row by every warp of the block: runs of 32-edge
// steps per warp, combined in warp order; valid in warp 0.
struct BcShared {
  BcStep step[kBcWarps];
  uint32_t list[kBcLongList];
  unsigned count;
  double2 sum[kBcWarps][32];
  uint64_t met[kBcWarps];
};
__device__ __forceinline__ uint64_t bc_add_rows_block(BcShared& sh, const uint32_t* adj,
                                                      const uint64_t* mask, const double* row,
                                                      uint32_t b, uint32_t e, uint64_t need,
                                                      double2& sum) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t per = ((e - b + kBcWarps - 1) / kBcWarps + 31) / 32 * 32;
  const uint32_t lo = min(e, b + w * per), hi = min(e, lo + per);
  double2 part = make_double2(0.0, 0.0);
  uint64_t met = 0;
  bc_add_rows(sh.step[w], adj, mask, row, lo, hi, need, met, part);
  met = bc_or(met);
  sh.sum[w][lane] = part;
  if (lane == 0) sh.met[w] = met;
  __syncthreads();
  uint64_t all = 0;
  if (w == 0)
    for (int i = 0; i < kBcWarps; i++) {
      all |= sh.met[i];
      sum.x = __dadd_rn(sum.x, sh.sum[i][lane].x);
      sum.y = __dadd_rn(sum.y, sh.sum[i][lane].y);
    }
  __syncthreads();
  return all;
}

__global__ void __launch_bounds__(kBlock, kBcOcc) bc_forward_level_k(BcLevelArgs A) {
  __shared__ BcShared sh;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) sh.count = 0;
  __syncthreads();
  const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  bool any = false;
  auto settle = [&](uint64_t v, uint64_t reached, double2 sigma) {
    if (!reached) return;
    any = true;
    if (lane == 0) {
      A.mask[v] = reached;
      A.vis[v] |= reached;
    }
    double* row = A.row + v * kBcB + 2 * lane;
    const uint32_t bits = (uint32_t)(reached >> (2 * lane)) & 3u;
    if (bits == 3u) {
      *reinterpret_cast<double2*>(row) = sigma;
    } else {
      if (bits & 1u) row[0] = sigma.x;
      if (bits & 2u) row[1] = sigma.y;
    }
  };
  // lane l's node: nw apart, so that a run of long rows (the lowest ids of an
  // R-MAT graph) is spread over the warps
  for (uint64_t v0 = gw; v0 < A.n; v0 += nw * A.group) {
    const uint64_t mine = v0 + lane * nw;
    uint64_t need = 0;
    uint32_t b = 0, e = 0;
    if (lane < A.group && mine < A.n) {
      A.mask[mine] = 0;
      need = A.qmask & ~A.vis[mine];
      if (need) {
        b = A.off[mine];
        e = A.off[mine + 1];
      }
      if (b == e) {
        need = 0;
      } else if (e - b > kBcLong) {
        const unsigned at = atomicAdd(&sh.count, 1u);
        if (at < kBcLongList) {
          sh.list[at] = (uint32_t)mine;
          need = 0;
        }
      }
    }
    __syncwarp();  // the cleared masks, before settle() sets one
    bc_nodes(A, sh.step[threadIdx.x >> 5], need, b, e, [&](int l, uint64_t, uint64_t met, double2 sigma) {
      if (__any_sync(0xffffffffu, met != 0)) settle(v0 + l * nw, bc_or(met), sigma);
    });
  }
  __syncthreads();
  const unsigned listed = min(sh.count, (unsigned)kBcLongList);
  for (unsigned i = 0; i < listed; i++) {
    const uint64_t v = sh.list[i];
    double2 sigma = make_double2(0.0, 0.0);
    const uint64_t reached = bc_add_rows_block(sh, A.adj, A.front, A.row, A.off[v], A.off[v + 1],
                                               A.qmask & ~A.vis[v], sigma);
    if (threadIdx.x < 32) settle(v, reached, sigma);
  }
  if (lane == 0 && any) atomicOr(A.found, 1u);
}

__global__ void __launch_bounds__(kBlock, kBcOcc) bc_backward_level_k(BcLevelArgs A) {
  __shared__ BcShared sh;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) sh.count = 0;
  __syncthreads();
  const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  auto settle = [&](uint64_t v, uint32_t bits, double2 c) {  // c: the sums of the successors' c
    double* row = A.row + v * kBcB + 2 * lane;
    double* delta = A.delta + v * kBcB + 2 * lane;
    if (bits & 1u) {
      const double sigma = row[0], d = __dmul_rn(sigma, c.x);
      delta[0] = d;
      row[0] = __ddiv_rn(__dadd_rn(1.0, d), sigma);
    }
    if (bits & 2u) {
      const double sigma = row[1], d = __dmul_rn(sigma, c.y);
      delta[1] = d;
      row[1] = __ddiv_rn(__dadd_rn(1.0, d), sigma);
    }
  };
  for (uint64_t v0 = gw; v0 < A.n; v0 += nw * A.group) {
    const uint64_t mine = v0 + lane * nw;
    uint64_t here = 0;
    uint32_t b = 0, e = 0;
    if (lane < A.group && mine < A.n) {
      here = A.mask[mine];
      if (here) {
        b = A.off[mine];
        e = A.off[mine + 1];
        if (e - b > kBcLong) {
          const unsigned at = atomicAdd(&sh.count, 1u);
          if (at < kBcLongList) {
            sh.list[at] = (uint32_t)mine;
            here = 0;
          }
        }
      }
    }
    bc_nodes(A, sh.step[threadIdx.x >> 5], here, b, e, [&](int l, uint64_t at, uint64_t, double2 d) {
      settle(v0 + l * nw, (uint32_t)(at >> (2 * lane)) & 3u, d);
    });
  }
  __syncthreads();
  const unsigned listed = min(sh.count, (unsigned)kBcLongList);
  for (unsigned i = 0; i < listed; i++) {
    const uint64_t v = sh.list[i];
    const uint64_t here = A.mask[v];
    double2 d = make_double2(0.0, 0.0);
    bc_add_rows_block(sh, A.adj, A.front, A.row, A.off[v], A.off[v + 1], here, d);
    if (threadIdx.x < 32) settle(v, (uint32_t)(here >> (2 * lane)) & 3u, d);
  }
}

__global__ void bc_seed_level_k(const uint32_t* __restrict__ src, uint32_t nq, uint64_t* vis,
                                uint64_t* mask, double* sigma) {
  const uint32_t q = threadIdx.x;
  if (q >= nq) return;
  const uint32_t s = src[q];
  atomicOr((unsigned long long*)(vis + s), 1ull << q);
  atomicOr((unsigned long long*)(mask + s), 1ull << q);
  sigma[(uint64_t)s * kBcB + q] = 1.0;
}

// The batch's partial (sources in order, each source's own node excluded),
// added to out in batch order; vis: the sources that reach each node.
__global__ void bc_fold_level_k(const double* __restrict__ delta, const uint64_t* __restrict__ vis,
                                const uint32_t* __restrict__ src, uint32_t nq, uint64_t n,
                                double* __restrict__ out) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t met = vis[v];
    if (!met) continue;
    double p = 0.0;
    for (uint32_t q = 0; q < nq; q++)
      if (((met >> q) & 1ull) && src[q] != v) p = __dadd_rn(p, delta[v * kBcB + q]);
    out[v] = __dadd_rn(out[v], p);
  }
}

// The mask levels of a batch that goes on below them (bc_deep_from_masks).
struct BcMasks {
  const uint64_t* level[kBcMaxLevels];
  uint32_t count;
};

// hop[v * 64 + q]: the level at which source q reaches v, -1 if none here; a
// warp per node.
__global__ void bc_masks_to_hop_k(BcMasks m, uint64_t n, int32_t* __restrict__ hop) {
  const int lane = threadIdx.x & 31;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t v = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += nw) {
    const uint64_t mine = (uint32_t)lane < m.count ? m.level[lane][v] : 0ull;
    int32_t h0 = -1, h1 = -1;
    for (uint32_t l = 0; l < m.count; l++) {
      const uint64_t x = __shfl_sync(0xffffffffu, mine, l);
      if ((x >> lane) & 1ull) h0 = (int32_t)l;
      if ((x >> (lane + 32)) & 1ull) h1 = (int32_t)l;
    }
    hop[v * kBcB + lane] = h0;
    hop[v * kBcB + lane + 32] = h1;
  }
}

// dag[k], k the out-slot of u -> v: the sources that reach v one level after u.
__global__ void bc_masks_to_dag_k(BcMasks m, const uint32_t* __restrict__ off, const uint32_t* __restrict__ tgt,
                                  uint64_t n, uint64_t slots, uint64_t* __restrict__ dag) {
  for_each_slot_owner(off, n, slots, [&](uint64_t k, uint32_t u) {
    const uint32_t v = tgt[k];
    uint64_t f = 0;
    for (uint32_t l = 1; l < m.count; l++) {
      const uint64_t x = m.level[l - 1][u];
      if (x) f |= x & m.level[l][v];
    }
    dag[k] = f;
  });
}
static_assert(kBcMaxLevels <= 32, "a lane per level");

// ---- searches deeper than kBcMaxLevels: the same batch with a hop per (node,
// source) and, per out-slot, a mask of the sources whose DAG holds the edge
__global__ void bc_seed_k(const uint32_t* __restrict__ src, uint32_t nq, uint64_t* vis, uint64_t* front,
                          int32_t* hop, double* sigma) {
  const uint32_t q = threadIdx.x;
  if (q >= nq) return;
  const uint32_t s = src[q];
  atomicOr((unsigned long long*)(vis + s), 1ull << q);
  atomicOr((unsigned long long*)(front + s), 1ull << q);
  hop[(uint64_t)s * kBcB + q] = 0;
  sigma[(uint64_t)s * kBcB + q] = 1.0;
}

__global__ void bc_forward_k(BcBatchArgs A) {
  const int lane = threadIdx.x & 31;
  const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  bool any = false;
  for (uint64_t v = gw; v < A.n; v += nw) {
    const uint64_t need = A.qmask & ~A.vis[v];
    if (need == 0) {
      if (lane == 0) A.next[v] = 0;
      continue;
    }
    const uint32_t b = A.in_off[v], e = A.in_off[v + 1];
    double s0 = 0.0, s1 = 0.0;
    uint64_t reached = 0;
    for (uint32_t k0 = b; k0 < e; k0 += 8) {
      uint32_t u = 0;
      uint64_t f = 0;
      if (lane < 8 && k0 + lane < e) {
        u = A.in_src[k0 + lane];
        f = A.front[u] & need;
        // an edge can be on several sources' DAGs at different levels; the
        // warp owning v is the only writer of v's in-slots within a level
        if (f) A.dag[A.in_to_out[k0 + lane]] |= f;
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const uint64_t fj = __shfl_sync(0xffffffffu, f, j);
        const uint32_t uj = __shfl_sync(0xffffffffu, u, j);
        if (fj) {
          reached |= fj;
          const double* row = A.sigma + (uint64_t)uj * kBcB;
          if ((fj >> lane) & 1ull) s0 += row[lane];
          if ((fj >> (lane + 32)) & 1ull) s1 += row[lane + 32];
        }
      }
    }
    if (lane == 0) A.next[v] = reached;
    if (reached) {
      any = true;
      if (lane == 0) A.vis[v] |= reached;
      if ((reached >> lane) & 1ull) {
        A.sigma[v * kBcB + lane] = s0;
        A.hop[v * kBcB + lane] = A.level;
      }
      if ((reached >> (lane + 32)) & 1ull) {
        A.sigma[v * kBcB + lane + 32] = s1;
        A.hop[v * kBcB + lane + 32] = A.level;
      }
    }
  }
  if (lane == 0 && any) atomicOr(A.found, 1u);
}

__global__ void bc_backward_k(BcBatchArgs A) {
  const int lane = threadIdx.x & 31;
  const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t v = gw; v < A.n; v += nw) {
    const bool h0 = A.hop[v * kBcB + lane] == A.level;
    const bool h1 = A.hop[v * kBcB + lane + 32] == A.level;
    const uint64_t mL = (uint64_t)__ballot_sync(0xffffffffu, h0) |
                        ((uint64_t)__ballot_sync(0xffffffffu, h1) << 32);
    if (mL == 0) continue;
    const double sv0 = h0 ? A.sigma[v * kBcB + lane] : 0.0;
    const double sv1 = h1 ? A.sigma[v * kBcB + lane + 32] : 0.0;
    double d0 = 0.0, d1 = 0.0;
    const uint32_t b = A.out_off[v], e = A.out_off[v + 1];
    for (uint32_t k0 = b; k0 < e; k0 += 8) {
      uint32_t w = 0;
      uint64_t dm = 0;
      if (lane < 8 && k0 + lane < e) {
        dm = A.dag[k0 + lane] & mL;
        if (dm) w = A.out_tgt[k0 + lane];
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const uint64_t dj = __shfl_sync(0xffffffffu, dm, j);
        const uint32_t wj = __shfl_sync(0xffffffffu, w, j);
        if (dj) {
          const uint64_t r = (uint64_t)wj * kBcB;
          if ((dj >> lane) & 1ull)  // coeff = (1 + delta[w]) / sigma[w]; delta[v] += sigma[v] * coeff
            d0 += __dmul_rn(sv0, __ddiv_rn(__dadd_rn(1.0, A.delta[r + lane]), A.sigma[r + lane]));
          if ((dj >> (lane + 32)) & 1ull)
            d1 += __dmul_rn(sv1, __ddiv_rn(__dadd_rn(1.0, A.delta[r + lane + 32]), A.sigma[r + lane + 32]));
        }
      }
    }
    if (h0) A.delta[v * kBcB + lane] = d0;
    if (h1) A.delta[v * kBcB + lane + 32] = d1;
  }
}

// The batch's partial (sources in order, each source's own node excluded),
// added to out in batch order.
__global__ void bc_fold_k(const double* __restrict__ delta, const uint32_t* __restrict__ src,
                          uint32_t nq, uint64_t n, double* __restrict__ out) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x) {
    double p = 0.0;
    for (uint32_t q = 0; q < nq; q++)
      if (src[q] != v) p = __dadd_rn(p, delta[v * kBcB + q]);
    out[v] = __dadd_rn(out[v], p);
  }
}

// ---- weighted, 64 sources at once -----------------------------------------
// brandes_from_weighted (:278-339) for the batch: distances by a multi-source
// frontier Bellman-Ford (lanes are sources; atomicMin on the bit patterns of
// non-negative f64, whose fixpoint is Dijkstra's distances); then the tight
// DAG per source (fl(dist[u] + w) == dist[v] exactly, the reference's tie
// rule; zero-weight ties ordered by id) as a mask per out-CSR slot; then
// sigma in rounds over that DAG -- a (node, source) is settled once every
// tight predecessor was settled in an earlier round, and sigma is the sum
// over them -- with the round as the node's level for the backward pass.
struct BcwArgs {
  const uint32_t* out_off;
  const uint32_t* out_tgt;
  const double* w_out;        // per out-CSR slot
  const uint32_t* in_off;
  const uint32_t* in_src;
  const uint32_t* in_to_out;
  uint64_t n;
  uint64_t qmask;
  unsigned long long* dist;   // n x 64 bit patterns
  const uint64_t* flag_cur;   // sources whose distance at v fell last round
  uint64_t* flag_next;
  uint64_t* dag;              // per out-CSR slot: sources for which the edge is tight
  uint64_t* reach;            // per node: sources that reach it
  const uint64_t* done_prev;
  uint64_t* done_next;
  double* sigma;
  int32_t* round;             // n x 64: the round a (node, source) settled, -1 = never
  int32_t r;
  unsigned* found;
};

__global__ void bcw_seed_k(const uint32_t* __restrict__ src, uint32_t nq, unsigned long long* dist,
                           uint64_t* flag, uint64_t* done, int32_t* round, double* sigma) {
  const uint32_t q = threadIdx.x;
  if (q >= nq) return;
  const uint32_t s = src[q];
  dist[(uint64_t)s * kBcB + q] = 0ull;  // +0.0
  atomicOr((unsigned long long*)(flag + s), 1ull << q);
  atomicOr((unsigned long long*)(done + s), 1ull << q);
  round[(uint64_t)s * kBcB + q] = 0;
  sigma[(uint64_t)s * kBcB + q] = 1.0;
}

// One Bellman-Ford round: every (v, source) whose distance fell last round
// relaxes v's out-edges.
__global__ void bcw_relax_k(BcwArgs A) {
  const int lane = threadIdx.x & 31;
  const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  bool any = false;
  for (uint64_t v = gw; v < A.n; v += nw) {
    const uint64_t fl = A.flag_cur[v];
    if (!fl) continue;
    const bool f0 = (fl >> lane) & 1ull, f1 = (fl >> (lane + 32)) & 1ull;
    const double d0 = f0 ? __longlong_as_double((long long)A.dist[v * kBcB + lane]) : 0.0;
    const double d1 = f1 ? __longlong_as_double((long long)A.dist[v * kBcB + lane + 32]) : 0.0;
    const uint32_t b = A.out_off[v], e = A.out_off[v + 1];
    for (uint32_t k0 = b; k0 < e; k0 += 8) {
      uint32_t wl = 0;
      double xl = 0.0;
      if (lane < 8 && k0 + lane < e) {
        wl = A.out_tgt[k0 + lane];
        xl = A.w_out[k0 + lane];
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        if (k0 + j >= e) break;
        const uint32_t w = __shfl_sync(0xffffffffu, wl, j);
        const double x = __shfl_sync(0xffffffffu, xl, j);
        bool low0 = false, low1 = false;
        if (f0) {
          const unsigned long long nd = (unsigned long long)__double_as_longlong(__dadd_rn(d0, x));
          low0 = nd < atomicMin(&A.dist[(uint64_t)w * kBcB + lane], nd);
        }
        if (f1) {
          const unsigned long long nd = (unsigned long long)__double_as_longlong(__dadd_rn(d1, x));
          low1 = nd < atomicMin(&A.dist[(uint64_t)w * kBcB + lane + 32], nd);
        }
        const uint64_t lowered = (uint64_t)__ballot_sync(0xffffffffu, low0) |
                                 ((uint64_t)__ballot_sync(0xffffffffu, low1) << 32);
        if (lowered) {
          any = true;
          if (lane == 0) atomicOr((unsigned long long*)(A.flag_next + w), lowered);
        }
      }
    }
  }
  if (lane == 0 && any) atomicOr(A.found, 1u);
}

__device__ __forceinline__ bool tight_bits(unsigned long long du, unsigned long long dv, double x,
                                           uint32_t u, uint32_t v) {
  if (du == kInfBits || u == v) return false;
  const unsigned long long nd = (unsigned long long)__double_as_longlong(
      __dadd_rn(__longlong_as_double((long long)du), x));
  if (nd != dv) return false;
  return du < dv || (du == dv && u < v);  // zero weights: keep the DAG acyclic
}

// Tight mask of every out-slot, and the sources that reach each node.
__global__ void bcw_tight_k(BcwArgs A) {
  const int lane = threadIdx.x & 31;
  const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t u = gw; u < A.n; u += nw) {
    const unsigned long long du0 = A.dist[u * kBcB + lane], du1 = A.dist[u * kBcB + lane + 32];
    const uint64_t reach = ((uint64_t)__ballot_sync(0xffffffffu, du0 != kInfBits) |
                            ((uint64_t)__ballot_sync(0xffffffffu, du1 != kInfBits) << 32)) & A.qmask;
    if (lane == 0) A.reach[u] = reach;
    if (!reach) continue;
    const uint32_t b = A.out_off[u], e = A.out_off[u + 1];
    for (uint32_t k = b; k < e; k++) {
      const uint32_t v = A.out_tgt[k];
      const double x = A.w_out[k];
      const bool t0 = tight_bits(du0, A.dist[(uint64_t)v * kBcB + lane], x, (uint32_t)u, v);
      const bool t1 = tight_bits(du1, A.dist[(uint64_t)v * kBcB + lane + 32], x, (uint32_t)u, v);
      const uint64_t m = ((uint64_t)__ballot_sync(0xffffffffu, t0) |
                          ((uint64_t)__ballot_sync(0xffffffffu, t1) << 32)) & A.qmask;
      if (lane == 0) A.dag[k] = m;
    }
  }
}

// Round r of sigma: (w, source) settles when no tight predecessor is still
// unsettled (as of the round's start); sigma = the sum over its tight
// predecessors, in in-CSR order.
__global__ void bcw_sigma_k(BcwArgs A) {
  const int lane = threadIdx.x & 31;
  const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  bool any = false;
  for (uint64_t w = gw; w < A.n; w += nw) {
    const uint64_t dp = A.done_prev[w];
    const uint64_t pend = A.reach[w] & ~dp;
    if (!pend) {
      if (lane == 0) A.done_next[w] = dp;
      continue;
    }
    const uint32_t b = A.in_off[w], e = A.in_off[w + 1];
    uint64_t notready = 0;
    for (uint32_t k = b + lane; k < e; k += 32) {
      const uint64_t tm = A.dag[A.in_to_out[k]] & pend;
      if (tm) notready |= tm & ~A.done_prev[A.in_src[k]];
    }
    notready = ((uint64_t)__reduce_or_sync(0xffffffffu, (unsigned)(notready >> 32)) << 32) |
               __reduce_or_sync(0xffffffffu, (unsigned)notready);
    const uint64_t ready = pend & ~notready;
    if (lane == 0) A.done_next[w] = dp | ready;
    if (!ready) continue;
    any = true;
    double s0 = 0.0, s1 = 0.0;
    for (uint32_t k0 = b; k0 < e; k0 += 8) {
      uint32_t ul = 0;
      uint64_t tl = 0;
      if (lane < 8 && k0 + lane < e) {
        tl = A.dag[A.in_to_out[k0 + lane]] & ready;
        if (tl) ul = A.in_src[k0 + lane];
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const uint64_t tj = __shfl_sync(0xffffffffu, tl, j);
        const uint32_t uj = __shfl_sync(0xffffffffu, ul, j);
        if (tj) {
          if ((tj >> lane) & 1ull) s0 += A.sigma[(uint64_t)uj * kBcB + lane];
          if ((tj >> (lane + 32)) & 1ull) s1 += A.sigma[(uint64_t)uj * kBcB + lane + 32];
        }
      }
    }
    if ((ready >> lane) & 1ull) {
      A.sigma[w * kBcB + lane] = s0;
      A.round[w * kBcB + lane] = A.r;
    }
    if ((ready >> (lane + 32)) & 1ull) {
      A.sigma[w * kBcB + lane + 32] = s1;
      A.round[w * kBcB + lane + 32] = A.r;
    }
  }
  if (lane == 0 && any) atomicOr(A.found, 1u);
}

__global__ void fill_u64_bc_k(unsigned long long* p, uint64_t n, unsigned long long v) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

__global__ void inv_perm_k(const uint32_t* __restrict__ eid, uint64_t m, uint32_t* __restrict__ inv) {
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < m;
       k += (uint64_t)gridDim.x * blockDim.x)
    inv[eid[k]] = (uint32_t)k;
}

__global__ void compose_k(const uint32_t* __restrict__ a, const uint32_t* __restrict__ inv, uint64_t m,
                          uint32_t* __restrict__ out) {
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < m;
       k += (uint64_t)gridDim.x * blockDim.x)
    out[k] = inv[a[k]];
}

}  // namespace

// What the batches of a graph deeper than kBcMaxLevels share, made by the
// first of them.
struct BcDeep {
  Scratch<uint32_t> in_to_out;
  Scratch<uint64_t> fa, fb, dag;
  Scratch<int32_t> hop;
};

static void bc_deep_prepare(TopoImpl* t, BcDeep& d, cudaStream_t s) {
  const uint64_t n = t->n, m = t->m;
  d.in_to_out.alloc(m ? m : 1, s);
  if (m) {
    Scratch<uint32_t> inv(m, s);
    inv_perm_k<<<grid_for(m), kBlock, 0, s>>>(t->out.eid.get(), m, inv.get());
    UG_LAUNCH_CHECK();
    compose_k<<<grid_for(m), kBlock, 0, s>>>(t->in.eid.get(), inv.get(), m, d.in_to_out.get());
    UG_LAUNCH_CHECK();
  }
  d.fa.alloc(n, s);
  d.fb.alloc(n, s);
  d.dag.alloc(m ? m : 1, s);
}

// A batch that met its limit of mask levels goes on with a hop per (node,
// source): hops, DAG masks and the frontier from the levels it has (0 to L).
// The hops are made in delta, which is free until the way back, so that they
// need no memory beside the masks.
static void bc_deep_from_masks(TopoImpl* t, BcDeep& d, std::vector<Scratch<uint64_t>>& masks, size_t L,
                               double* delta, cudaStream_t s) {
  const uint64_t n = t->n, m = t->m;
  BcMasks lv{};
  for (size_t l = 0; l <= L; l++) lv.level[l] = masks[l].get();
  lv.count = (uint32_t)L + 1;
  int32_t* hop = reinterpret_cast<int32_t*>(delta);
  bc_masks_to_hop_k<<<grid_for(n * 32, kBlock, 148u * 8u), kBlock, 0, s>>>(lv, n, hop);
  UG_LAUNCH_CHECK();
  if (m) {
    bc_masks_to_dag_k<<<grid_for(m), kBlock, 0, s>>>(lv, t->out.off.get(), t->out.tgt.get(), n, m, d.dag.get());
    UG_LAUNCH_CHECK();
  }
  UG_CUDA(cudaMemcpyAsync(d.fa.get(), lv.level[L], n * 8, cudaMemcpyDeviceToDevice, s));
  masks.clear();
  d.hop.alloc(n * kBcB, s);
  UG_CUDA(cudaMemcpyAsync(d.hop.get(), hop, n * kBcB * 4, cudaMemcpyDeviceToDevice, s));
}

// A batch (at most 64 sources), added into d_out, from level L on: its
// frontier in d.fa, its nodes so far in vis, hop and sigma.  (64 sources on 34
// layers of 20,000 nodes: 26.8 ms a call with these kernels alone, 30.8 when
// the first batch started over at level 31, 18.8 so; a grid of 300 by 300
// 37.4 / 38.9 / 37.1, with 256 sources 146.6 / 149.0 / 146.5.)
static void bc_deep_batch(TopoImpl* t, BcDeep& d, const uint32_t* d_src, uint32_t nq, int32_t L, uint64_t* vis,
                          double* sigma, double* delta, double* d_out, cudaStream_t s) {
  const uint64_t n = t->n;
  Scratch<unsigned> found(1, s);
  BcBatchArgs a;
  a.in_off = t->in.off.get();
  a.in_src = t->in.tgt.get();
  a.in_to_out = d.in_to_out.get();
  a.out_off = t->out.off.get();
  a.out_tgt = t->out.tgt.get();
  a.n = n;
  a.vis = vis;
  a.hop = d.hop.get();
  a.sigma = sigma;
  a.delta = delta;
  a.dag = d.dag.get();
  a.found = found.get();
  a.qmask = nq == 64 ? ~0ull : ((1ull << nq) - 1ull);
  const unsigned gw = grid_for(n * 32, kBlock, 148u * 8u);
  UG_CUDA(cudaMemsetAsync(delta, 0, n * kBcB * 8, s));
  uint64_t* cur = d.fa.get();
  uint64_t* nxt = d.fb.get();
  while (true) {
    a.level = L + 1;
    a.front = cur;
    a.next = nxt;
    UG_CUDA(cudaMemsetAsync(found.get(), 0, 4, s));
    bc_forward_k<<<gw, kBlock, 0, s>>>(a);
    UG_LAUNCH_CHECK();
    if (!read_u32(found.get(), s)) break;
    L++;
    std::swap(cur, nxt);
  }
  // nodes of the deepest level L have no successors (delta 0)
  for (int32_t lvl = L - 1; lvl >= 0; lvl--) {
    a.level = lvl;
    bc_backward_k<<<gw, kBlock, 0, s>>>(a);
    UG_LAUNCH_CHECK();
  }
  bc_fold_k<<<grid_for(n), kBlock, 0, s>>>(delta, d_src, nq, n, d_out);
  UG_LAUNCH_CHECK();
}

// Unweighted betweenness over `sources`, 64 at a time, added into d_out.
static void betweenness_batched(TopoImpl* t, const std::vector<uint32_t>& sources, double* d_out,
                                cudaStream_t s) {
  const uint64_t n = t->n, m = t->m;
  ensure_in(t, s);
  Scratch<uint64_t> vis(n, s);
  Scratch<double> row(n * kBcB, s), delta(n * kBcB, s);
  Scratch<uint32_t> d_src(kBcB, s);
  Scratch<unsigned> found(1, s);
  std::vector<Scratch<uint64_t>> masks;  // masks[l]: the sources that reach each node at level l
  auto level = [&](size_t l) {
    while (masks.size() <= l) masks.emplace_back(n, s);
    return masks[l].get();
  };
  BcLevelArgs a{};
  a.n = n;
  a.vis = vis.get();
  a.row = row.get();
  a.delta = delta.get();
  a.found = found.get();
  BcDeep d;
  bool deep = false;  // the graph has searches past the levels kept
  const unsigned gw = grid_for(n * 32, kBlock, 148u * kBcOcc);
  // few nodes at a time while there are fewer than four groups per warp
  a.group = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(kBcGroup, n / (4ull * gw * kBcWarps)));
  for (size_t c0 = 0; c0 < sources.size(); c0 += kBcB) {
    const uint32_t nq = (uint32_t)std::min<size_t>(kBcB, sources.size() - c0);
    a.qmask = nq == 64 ? ~0ull : ((1ull << nq) - 1ull);
    UG_CUDA(cudaMemcpyAsync(d_src.get(), sources.data() + c0, nq * 4, cudaMemcpyHostToDevice, s));
    UG_CUDA(cudaMemsetAsync(vis.get(), 0, n * 8, s));
    if (deep) {
      UG_CUDA(cudaMemsetAsync(d.fa.get(), 0, n * 8, s));
      UG_CUDA(cudaMemsetAsync(d.hop.get(), 0xFF, n * kBcB * 4, s));
      if (m) UG_CUDA(cudaMemsetAsync(d.dag.get(), 0, m * 8, s));
      bc_seed_k<<<1, kBcB, 0, s>>>(d_src.get(), nq, vis.get(), d.fa.get(), d.hop.get(), row.get());
      UG_LAUNCH_CHECK();
      bc_deep_batch(t, d, d_src.get(), nq, 0, vis.get(), row.get(), delta.get(), d_out, s);
      continue;
    }
    UG_CUDA(cudaMemsetAsync(level(0), 0, n * 8, s));
    bc_seed_level_k<<<1, kBcB, 0, s>>>(d_src.get(), nq, vis.get(), level(0), row.get());
    UG_LAUNCH_CHECK();
    a.off = t->in.off.get();
    a.adj = t->in.tgt.get();
    size_t L = 0;  // the deepest level met
    bool more = true;
    while (L + 1 < kBcMaxLevels) {
      a.front = level(L);
      a.mask = level(L + 1);
      UG_CUDA(cudaMemsetAsync(found.get(), 0, 4, s));
      bc_forward_level_k<<<gw, kBlock, 0, s>>>(a);
      UG_LAUNCH_CHECK();
      more = read_u32(found.get(), s) != 0;
      if (!more) break;
      L++;
    }
    if (more) {
      deep = true;
      bc_deep_prepare(t, d, s);
      bc_deep_from_masks(t, d, masks, L, delta.get(), s);
      bc_deep_batch(t, d, d_src.get(), nq, (int32_t)L, vis.get(), row.get(), delta.get(), d_out, s);
      continue;
    }
    a.off = t->out.off.get();
    a.adj = t->out.tgt.get();
    for (size_t l = L; l >= 1; l--) {  // level 0, the sources, takes no part in the result
      a.mask = level(l);
      a.front = level(l + 1);
      bc_backward_level_k<<<gw, kBlock, 0, s>>>(a);
      UG_LAUNCH_CHECK();
    }
    bc_fold_level_k<<<grid_for(n), kBlock, 0, s>>>(delta.get(), vis.get(), d_src.get(), nq, n, d_out);
    UG_LAUNCH_CHECK();
  }
}

// Weighted betweenness over `sources`, 64 at a time, added into d_out;
// w_out: the weights in out-CSR slot order.
static void betweenness_weighted_batched(TopoImpl* t, const double* w_out,
                                         const std::vector<uint32_t>& sources, double* d_out,
                                         cudaStream_t s) {
  const uint64_t n = t->n, m = t->m;
  ensure_in(t, s);
  Scratch<uint32_t> in_to_out(m ? m : 1, s);
  if (m) {
    Scratch<uint32_t> inv(m, s);
    inv_perm_k<<<grid_for(m), kBlock, 0, s>>>(t->out.eid.get(), m, inv.get());
    UG_LAUNCH_CHECK();
    compose_k<<<grid_for(m), kBlock, 0, s>>>(t->in.eid.get(), inv.get(), m, in_to_out.get());
    UG_LAUNCH_CHECK();
  }
  Scratch<unsigned long long> dist(n * kBcB, s);
  Scratch<uint64_t> fl0(n, s), fl1(n, s), reach(n, s), dn0(n, s), dn1(n, s), dag(m ? m : 1, s);
  Scratch<int32_t> round(n * kBcB, s);
  Scratch<double> sigma(n * kBcB, s), delta(n * kBcB, s);
  Scratch<uint32_t> d_src(kBcB, s);
  Scratch<unsigned> found(1, s);
  BcwArgs a;
  a.out_off = t->out.off.get();
  a.out_tgt = t->out.tgt.get();
  a.w_out = w_out;
  a.in_off = t->in.off.get();
  a.in_src = t->in.tgt.get();
  a.in_to_out = in_to_out.get();
  a.n = n;
  a.dist = dist.get();
  a.dag = dag.get();
  a.reach = reach.get();
  a.sigma = sigma.get();
  a.round = round.get();
  a.found = found.get();
  BcBatchArgs bk{};  // the backward pass of the unweighted batch, on rounds and the tight DAG
  bk.out_off = t->out.off.get();
  bk.out_tgt = t->out.tgt.get();
  bk.n = n;
  bk.hop = round.get();
  bk.sigma = sigma.get();
  bk.delta = delta.get();
  bk.dag = dag.get();
  const unsigned gw = grid_for(n * 32, kBlock, 148u * 8u);
  auto read_found = [&]() {
    unsigned f = 0;
    UG_CUDA(cudaMemcpyAsync(&f, found.get(), 4, cudaMemcpyDeviceToHost, s));
    UG_CUDA(cudaStreamSynchronize(s));
    return f;
  };
  for (size_t c0 = 0; c0 < sources.size(); c0 += kBcB) {
    const uint32_t nq = (uint32_t)std::min<size_t>(kBcB, sources.size() - c0);
    a.qmask = nq == 64 ? ~0ull : ((1ull << nq) - 1ull);
    UG_CUDA(cudaMemcpyAsync(d_src.get(), sources.data() + c0, nq * 4, cudaMemcpyHostToDevice, s));
    fill_u64_bc_k<<<grid_for(n * kBcB), kBlock, 0, s>>>(dist.get(), n * kBcB, kInfBits);
    UG_LAUNCH_CHECK();
    UG_CUDA(cudaMemsetAsync(fl0.get(), 0, n * 8, s));
    UG_CUDA(cudaMemsetAsync(fl1.get(), 0, n * 8, s));
    UG_CUDA(cudaMemsetAsync(dn0.get(), 0, n * 8, s));
    UG_CUDA(cudaMemsetAsync(round.get(), 0xFF, n * kBcB * 4, s));
    UG_CUDA(cudaMemsetAsync(sigma.get(), 0, n * kBcB * 8, s));
    UG_CUDA(cudaMemsetAsync(delta.get(), 0, n * kBcB * 8, s));
    if (m) UG_CUDA(cudaMemsetAsync(dag.get(), 0, m * 8, s));  // unreached nodes' slots stay 0
    bcw_seed_k<<<1, kBcB, 0, s>>>(d_src.get(), nq, dist.get(), fl0.get(), dn0.get(), round.get(),
                                  sigma.get());
    UG_LAUNCH_CHECK();
    // distances
    uint64_t* cur = fl0.get();
    uint64_t* nxt = fl1.get();
    while (true) {
      a.flag_cur = cur;
      a.flag_next = nxt;
      UG_CUDA(cudaMemsetAsync(found.get(), 0, 4, s));
      bcw_relax_k<<<gw, kBlock, 0, s>>>(a);
      UG_LAUNCH_CHECK();
      UG_CUDA(cudaMemsetAsync(cur, 0, n * 8, s));  // consumed
      if (!read_found()) break;
      std::swap(cur, nxt);
    }
    // tight DAG, then sigma by rounds
    bcw_tight_k<<<gw, kBlock, 0, s>>>(a);
    UG_LAUNCH_CHECK();
    uint64_t* dprev = dn0.get();
    uint64_t* dnext = dn1.get();
    int32_t r = 0;
    while (true) {
      a.r = r + 1;
      a.done_prev = dprev;
      a.done_next = dnext;
      UG_CUDA(cudaMemsetAsync(found.get(), 0, 4, s));
      bcw_sigma_k<<<gw, kBlock, 0, s>>>(a);
      UG_LAUNCH_CHECK();
      if (!read_found()) break;
      r++;
      std::swap(dprev, dnext);
    }
    // backward over rounds, deepest first (round r's nodes have no successors)
    for (int32_t lvl = r - 1; lvl >= 0; lvl--) {
      bk.level = lvl;
      bc_backward_k<<<gw, kBlock, 0, s>>>(bk);
      UG_LAUNCH_CHECK();
    }
    bc_fold_k<<<grid_for(n), kBlock, 0, s>>>(delta.get(), d_src.get(), nq, n, d_out);
    UG_LAUNCH_CHECK();
  }
}

struct BcState {
  Scratch<int32_t> hop;                 // unweighted BFS level (-1 = unreached)
  Scratch<unsigned long long> dist;     // weighted distance bits
  Scratch<uint32_t> indeg;              // weighted: tight in-slots left
  Scratch<double> sigma, delta;
  Scratch<uint32_t> L;                  // nodes in discovery order, by level
  Scratch<uint64_t> pos;
  Scratch<uint32_t> cnt;
};

static uint64_t out_scan(const uint32_t* off, const uint32_t* F, uint64_t f, uint64_t* pos,
                         cudaStream_t s) {
  fdeg_out_k<<<grid_for(f + 1), kBlock, 0, s>>>(off, F, f, pos);
  UG_LAUNCH_CHECK();
  exclusive_scan_u64(pos, pos, f + 1, nullptr, s);
  uint64_t total = 0;
  UG_CUDA(cudaMemcpyAsync(&total, pos + f, 8, cudaMemcpyDeviceToHost, s));
  UG_CUDA(cudaStreamSynchronize(s));
  return total;
}

// One source's dependencies added into acc.
static void brandes_source(TopoImpl* t, const double* w_out, uint32_t src, BcState& st,
                           double* acc, cudaStream_t s) {
  const uint64_t n = t->n, m = t->m;
  const uint32_t* off = t->out.off.get();
  const uint32_t* tgt = t->out.tgt.get();
  const bool weighted = w_out != nullptr;
  UG_CUDA(cudaMemsetAsync(st.sigma.get(), 0, n * 8, s));
  UG_CUDA(cudaMemsetAsync(st.delta.get(), 0, n * 8, s));
  if (weighted) {
    DirView dv{};
    dv.off0 = off;
    dv.tgt0 = tgt;
    dv.eid0 = t->out.eid.get();
    sssp_run(dv, w_out, nullptr, n, m, src, st.dist.get(), s);
    UG_CUDA(cudaMemsetAsync(st.indeg.get(), 0, n * 4, s));
    if (m) {
      tight_indeg_k<<<grid_for(m, kBlock, 148u * 64u), kBlock, 0, s>>>(off, tgt, w_out, n, m,
                                                                        st.dist.get(),
                                                                        st.indeg.get());
      UG_LAUNCH_CHECK();
    }
  } else {
    UG_CUDA(cudaMemsetAsync(st.hop.get(), 0xFF, n * 4, s));
  }
  seed_source_k<<<1, 1, 0, s>>>(weighted ? nullptr : st.hop.get(), st.sigma.get(), st.L.get(), src);
  UG_LAUNCH_CHECK();
  std::vector<uint64_t> lev = {0, 1};  // level l = L[lev[l] .. lev[l+1])
  int32_t level = 0;
  while (true) {
    const uint64_t lo = lev[lev.size() - 2], hi = lev.back();
    const uint64_t f = hi - lo;
    if (f == 0) break;
    const uint32_t* F = st.L.get() + lo;
    uint64_t T = out_scan(off, F, f, st.pos.get(), s);
    if (T == 0) {
      lev.push_back(hi);
      break;
    }
    UG_CUDA(cudaMemsetAsync(st.cnt.get(), 0, 4, s));
    unsigned g = grid_for(T, kBlock, 148u * 64u);
    if (weighted) {
      kahn_k<<<g, kBlock, 0, s>>>(off, tgt, w_out, F, f, st.pos.get(), T, st.dist.get(),
                                  st.indeg.get(), st.sigma.get(), st.L.get() + hi, st.cnt.get());
      UG_LAUNCH_CHECK();
    } else {
      bfs_discover_k<<<g, kBlock, 0, s>>>(off, tgt, F, f, st.pos.get(), T, st.hop.get(), level,
                                          st.L.get() + hi, st.cnt.get());
      UG_LAUNCH_CHECK();
      bfs_sigma_k<<<g, kBlock, 0, s>>>(off, tgt, F, f, st.pos.get(), T, st.hop.get(), level,
                                       st.sigma.get());
      UG_LAUNCH_CHECK();
    }
    uint32_t next = read_u32(st.cnt.get(), s);
    lev.push_back(hi + next);
    level++;
  }
  // reverse accumulation, deepest level first
  for (size_t l = lev.size() - 1; l-- > 0;) {
    const uint64_t lo = lev[l], hi = lev[l + 1];
    if (hi <= lo) continue;
    const uint64_t cnt = hi - lo;
    unsigned g = grid_for(cnt * 32, kBlock, 148u * 64u);
    if (weighted)
      dependency_k<true><<<g, kBlock, 0, s>>>(off, tgt, w_out, st.L.get() + lo, cnt, nullptr,
                                              st.dist.get(), st.sigma.get(), st.delta.get(), acc,
                                              src);
    else
      dependency_k<false><<<g, kBlock, 0, s>>>(off, tgt, nullptr, st.L.get() + lo, cnt,
                                               st.hop.get(), nullptr, st.sigma.get(),
                                               st.delta.get(), acc, src);
    UG_LAUNCH_CHECK();
  }
}

void betweenness_run(TopoImpl* t, const double* d_weights, bool has_sample, double sample,
                     bool has_seed, uint64_t seed, double* d_out, cudaStream_t s) {
  const uint64_t n = t->n, m = t->m;
  if (n == 0) return;
  std::vector<uint32_t> sources = sample_sources(n, has_sample, sample, has_seed, seed, s);
  UG_CUDA(cudaMemsetAsync(d_out, 0, n * 8, s));
  if (sources.empty()) return;
  BcState st;
  st.sigma.alloc(n, s);
  st.delta.alloc(n, s);
  st.L.alloc(n, s);
  st.pos.alloc(n + 1, s);
  st.cnt.alloc(1, s);
  Scratch<double> w_out;
  if (d_weights) {
    st.dist.alloc(n, s);
    st.indeg.alloc(n, s);
    w_out.alloc(m ? m : 1, s);
    DirView dv{};
    dv.off0 = t->out.off.get();
    dv.tgt0 = t->out.tgt.get();
    dv.eid0 = t->out.eid.get();
    DirWeights dw;
    gather_dir_weights(t, dv, d_weights, dw, s);
    swap(w_out, dw.w0);
  } else {
    st.hop.alloc(n, s);
  }
  if (!d_weights) {
    betweenness_batched(t, sources, d_out, s);
  } else if (kBatchedWeighted) {
    betweenness_weighted_batched(t, w_out.get(), sources, d_out, s);
  } else {
  Scratch<double> acc(n, s);
  for (size_t c0 = 0; c0 < sources.size(); c0 += kSrcChunk) {
    UG_CUDA(cudaMemsetAsync(acc.get(), 0, n * 8, s));
    size_t c1 = c0 + kSrcChunk < sources.size() ? c0 + kSrcChunk : sources.size();
    for (size_t i = c0; i < c1; i++)
      brandes_source(t, d_weights ? w_out.get() : nullptr, sources[i], st, acc.get(), s);
    add_into_k<<<grid_for(n), kBlock, 0, s>>>(d_out, acc.get(), n);
    UG_LAUNCH_CHECK();
  }
  }
  if (has_sample) {
    scale_k<<<grid_for(n), kBlock, 0, s>>>(d_out, n, (double)n / (double)sources.size());
    UG_LAUNCH_CHECK();
  }
}

}  // namespace ug

using namespace ug;

extern "C" {

int ursa_gpu_betweenness(ursa_gpu_topo* t, int has_sample, double sample, int has_seed,
                         uint64_t seed, double* out) {
  return guard([&] {
    UG_CHECK(t, URSA_GPU_EINVAL, "topology is NULL");
    TopoImpl* ti = &t->impl;
    if (ti->n == 0) return;  // betweenness.rs:155-157
    UG_CHECK(out, URSA_GPU_EINVAL, "out is NULL");
    cudaStream_t s = thread_stream(ti->device);
    Scratch<double> d(ti->n, s);
    betweenness_run(ti, nullptr, has_sample != 0, sample, has_seed != 0, seed, d.get(), s);
    UG_CUDA(cudaMemcpyAsync(out, d.get(), ti->n * 8, cudaMemcpyDeviceToHost, s));
    UG_CUDA(cudaStreamSynchronize(s));
  });
}

int ursa_gpu_betweenness_weighted(ursa_gpu_topo* t, const double* weights, uint64_t n_weights,
                                  int has_sample, double sample, int has_seed, uint64_t seed,
                                  double* out) {
  return guard([&] {
    UG_CHECK(t, URSA_GPU_EINVAL, "topology is NULL");
    TopoImpl* ti = &t->impl;
    UG_CHECK(n_weights == ti->m, URSA_GPU_EINVAL, "weights length must equal the edge count");
    UG_CHECK(ti->m == 0 || weights, URSA_GPU_EINVAL, "weights is NULL");
    if (ti->n == 0) return;  // betweenness.rs:248-250
    UG_CHECK(out, URSA_GPU_EINVAL, "out is NULL");
    cudaStream_t s = thread_stream(ti->device);
    Scratch<double> dw(ti->m ? ti->m : 1, s), d(ti->n, s);
    if (ti->m) UG_CUDA(cudaMemcpyAsync(dw.get(), weights, ti->m * 8, cudaMemcpyHostToDevice, s));
    check_sssp_weights_device(dw.get(), ti->m, s);
    betweenness_run(ti, dw.get(), has_sample != 0, sample, has_seed != 0, seed, d.get(), s);
    UG_CUDA(cudaMemcpyAsync(out, d.get(), ti->n * 8, cudaMemcpyDeviceToHost, s));
    UG_CUDA(cudaStreamSynchronize(s));
  });
}

}  // extern "C"
