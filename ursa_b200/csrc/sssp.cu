// sssp.cu -- weighted shortest paths (ursa-core/src/algo/bfs.rs:126-259).
//
// dijkstra_distances: frontier Bellman-Ford.  Distances are non-negative
// doubles, whose IEEE bit patterns order like u64, so a relaxation is one
// atomicMin on the bits.  Every improvement re-queues the node (once per
// round, flag-deduplicated) until nothing changes.  The fixpoint is the same
// set of f64 values Dijkstra settles: dist[v] = min over edges of
// fl(dist[u] + w), and fl(a + w) is monotone in a with fl(a + w) >= a for
// w >= 0, so both compute the minimum left-to-right f64 path sum.
//
// shortest_path_weighted_with_cost: distances as above, then the path is
// walked back from the target.  The reference's parent of v is the first
// node, in Dijkstra's settle order, whose relaxation produced dist[v]
// (strict '<' at bfs.rs:237); with positive weights the settle order is the
// heap order (dist, node id), so the parent is the tight predecessor u
// (fl(dist[u] + w) == dist[v]) with the smallest (dist[u], u).  With
// zero-weight edges Dijkstra's settle order among equal distances depends on
// discovery order; there the path is a valid minimum-cost path but may pick
// a different tie.
#include <vector>

#include "frontier.cuh"

namespace ug {

namespace {

constexpr unsigned long long kInfBits = 0x7FF0000000000000ull;
// The first delta, in mean weights: a million nodes of degree 16 with 0.25 /
// 0.5 / 1 / 2 / 4 / infinity 3.98 / 3.72 / 3.73 / 4.06 / 4.38 / 4.38 ms a call
// (2.3 of them the weights' copy to the device).
constexpr double kDeltaWeights = 1.0;
// Fewer edges are walked again sooner than a step more is launched (2,000
// nodes, 20,000 edges: 198 us in one step, 329 in steps).
constexpr uint64_t kPlainEdges = 1u << 20;
constexpr uint64_t kStepEntries = 32768;  // a step of fewer entries is small;
constexpr unsigned kSmallSteps = 4;       // past this many in a row every further one is doubled
constexpr double kGapSteps = 8.0;         // a gap of more is jumped (jumping any: log-normal weights 8.2 -> 8.5 ms)
constexpr int kSsspBlocks = 8;         // per SM

__device__ __forceinline__ void append_w(uint32_t* Q, uint32_t* cnt, bool take, uint32_t v) {
  uint32_t mask = __ballot_sync(0xffffffffu, take);
  if (!take) return;
  int lane = threadIdx.x & 31;
  int leader = __ffs(mask) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(cnt, (uint32_t)__popc(mask));
  base = __shfl_sync(mask, base, leader);
  Q[base + __popc(mask & ((1u << lane) - 1u))] = v;
}

__device__ __forceinline__ unsigned long long ld_bits(const unsigned long long* p) {
  return *(const volatile unsigned long long*)p;
}

// ---- distances: rounds driven from the device ------------------------------
// A round is one launch; its last block to finish decides what the next one
// does, so rounds are enqueued several at a time and the host reads one word
// per run of them.  Near rounds relax the out-edges of the near list (entries
// of 16 edges); a node whose distance falls below the threshold joins the
// next near list (once per round: `stamp`), others the far list (once: `far`).
// With nothing near, the threshold moves up by delta (or, past a wide gap, to the
// nearest far node and delta) and a refill round moves the far nodes below it
// to the near list (the near-far form of
// delta-stepping, Davidson et al.).  Any order reaches the same fixpoint; this
// one relaxes fewer edges whose source is still to fall.
enum SsspMode : uint32_t { kNear = 0, kRefill = 1, kSsspDone = 2 };

struct SsspState {
  uint32_t mode, round;
  uint32_t entries[2];  // near entries, by round parity
  uint32_t fars[2];     // far nodes, in the buffer in use and the one a refill fills
  uint32_t far_buf;
  unsigned ticket, small_steps;
  double threshold, delta;
  unsigned long long walked;  // entries since the threshold moved
  double reached;  // the threshold before: distances below it have been queued as they fell
  unsigned long long far_min;  // of a refill: the least distance left far
};

struct SsspArgs {
  DirView d;
  const double* w0;
  const double* w1;
  uint64_t n;
  unsigned long long* dist;
  uint32_t* stamp;  // the last round v was queued for
  uint32_t* far;    // v is in the far list
  uint2* list[2];
  uint32_t* far_list[2];
  SsspState* st;
};

// One block: distances are +inf but the source's; delta is kDeltaWeights mean weights
// (of up to 1,024 slots a stride apart), +inf if that is no positive number or
// the graph is small.
__global__ void __launch_bounds__(1024) sssp_init_k(SsspArgs a, uint32_t source, uint64_t m) {
  __shared__ double sums[32];
  const uint64_t k = m <= 1024 ? threadIdx.x : (m / 1024) * threadIdx.x;
  double w = k < m ? a.w0[k] : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) w += __shfl_down_sync(0xffffffffu, w, o);
  if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = w;
  const uint32_t deg = dv_deg(a.d, source);
  const uint32_t entries = (deg + kSpan - 1) / kSpan;
  for (uint32_t i = threadIdx.x; i < entries; i += blockDim.x) a.list[0][i] = make_uint2(source, i * kSpan);
  __syncthreads();
  if (threadIdx.x) return;
  double sum = 0.0;
  for (int i = 0; i < 32; i++) sum += sums[i];
  double delta = kDeltaWeights * sum / (double)(m < 1024 ? (m ? m : 1) : 1024);
  if (!(delta > 0.0) || m < kPlainEdges) delta = __longlong_as_double((long long)kInfBits);
  a.dist[source] = 0ull;  // +0.0
  SsspState s{};
  s.mode = entries ? kNear : kSsspDone;
  s.entries[0] = entries;
  s.threshold = s.delta = delta;
  s.far_min = ~0ull;
  *a.st = s;
}

__global__ void __launch_bounds__(kBlock) sssp_round_k(SsspArgs a) {
  const uint32_t FULL = 0xffffffffu;
  const SsspState* sp = a.st;
  const uint32_t mode = sp->mode;
  if (mode == kSsspDone) return;
  const uint32_t round = sp->round, parity = (round + 1) & 1;
  const unsigned long long below = (unsigned long long)__double_as_longlong(sp->threshold);
  const uint64_t gtid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nthr = (uint64_t)gridDim.x * blockDim.x;
  if (mode == kNear) {
    const uint32_t count = sp->entries[round & 1];
    const uint2* list = a.list[round & 1];
    uint32_t* far_list = a.far_list[sp->far_buf];
    uint32_t* fars = &a.st->fars[sp->far_buf];
    const uint32_t sub = threadIdx.x & (kEntryLanes - 1);
    static_assert(kSpan == kEntryLanes, "a lane per edge of an entry");
    const uint64_t per_grid = nthr / kEntryLanes;
    const uint64_t rounds = (count + per_grid - 1) / per_grid;  // whole warps step together
    for (uint64_t r = 0; r < rounds; r++) {
      const uint64_t i = r * per_grid + gtid / kEntryLanes;
      bool near = false, far = false;
      uint32_t v = 0, deg = 0;
      if (i < count) {
        const uint2 e = list[i];
        const uint32_t j = e.y + sub;
        if (j < dv_deg(a.d, e.x)) {
          uint32_t slot;
          bool second;
          v = dv_nbr(a.d, e.x, j, &slot, &second);
          const double w = second ? a.w1[slot] : a.w0[slot];
          const double nd = __dadd_rn(__longlong_as_double((long long)ld_bits(&a.dist[e.x])), w);
          const unsigned long long nb = (unsigned long long)__double_as_longlong(nd);
          if (nb < ld_bits(&a.dist[v]) && nb < atomicMin(&a.dist[v], nb)) {
            if (nb < below)
              near = atomicExch(&a.stamp[v], round + 1) != round + 1;
            else
              far = atomicExch(&a.far[v], 1u) == 0u;
          }
        }
      }
      if (near) deg = dv_deg(a.d, v);
      append_entries(a.list[parity], &a.st->entries[parity], near, v, deg);
      append_w(far_list, fars, far, v);
    }
  } else {
    const unsigned long long done = (unsigned long long)__double_as_longlong(sp->reached);
    const uint32_t from = sp->far_buf, count = sp->fars[from];
    const uint32_t* list = a.far_list[from];
    const uint64_t span = (count + nthr - 1) / nthr * nthr;
    unsigned long long least = ~0ull;
    for (uint64_t i = gtid; i < span; i += nthr) {
      bool near = false, far = false;
      uint32_t v = 0, deg = 0;
      if (i < count) {
        v = list[i];
        const unsigned long long d = a.dist[v];
        far = d >= below;
        if (far) least = min(least, d);
        near = !far && d >= done;
        if (!far) a.far[v] = 0u;
      }
      if (near) deg = dv_deg(a.d, v);
      append_entries(a.list[parity], &a.st->entries[parity], near, v, deg);
      append_w(a.far_list[from ^ 1], &a.st->fars[from ^ 1], far, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) least = min(least, __shfl_xor_sync(FULL, least, o));
    if ((threadIdx.x & 31) == 0 && least != ~0ull) atomicMin(&a.st->far_min, least);
  }
  __syncthreads();
  if (threadIdx.x) return;
  SsspState* s = a.st;
  __threadfence();
  if (atomicAdd(&s->ticket, 1u) != gridDim.x - 1) return;
  __threadfence();
  if (mode == kRefill) {
    s->fars[s->far_buf] = 0;
    s->far_buf ^= 1;
  }
  s->walked += mode == kNear ? s->entries[round & 1] : 0;
  const uint32_t near = __ldcg(&s->entries[parity]), fars = __ldcg(&s->fars[s->far_buf]);
  if (near == 0 && fars != 0) {
    // after a few steps in a row that found little to do they are lengthened: a
    // round's launch then costs more than edges walked too early (the first
    // steps of any search are small, so one alone says nothing).  The far nodes are finite, so
    // the threshold reaches them; where adding delta no longer moves it,
    // nothing is far any more.
    s->small_steps = s->walked < kStepEntries ? s->small_steps + 1 : 0;
    if (s->small_steps > kSmallSteps) s->delta *= 2.0;
    s->walked = 0;
    double t = s->threshold + s->delta;
    // a refill that found nothing near has seen every far node: past a wide
    // gap, on to the nearest (one weight in a thousand 1, the others 1e-12, a
    // million nodes: 2.9 ms a call in steps of delta, 2.5 so)
    if (mode == kRefill) {
      const double nearest = __longlong_as_double((long long)__ldcg(&s->far_min));
      if (nearest - s->threshold > kGapSteps * s->delta) t = nearest + s->delta;
    }
    s->reached = s->threshold;
    if (t > s->threshold) {
      s->threshold = t;
    } else {
      s->delta = __longlong_as_double((long long)kInfBits);
      s->threshold = s->delta;
    }
  }
  s->far_min = ~0ull;
  s->mode = near ? kNear : fars ? kRefill : kSsspDone;
  s->entries[round & 1] = 0;
  s->round = round + 1;
  s->ticket = 0;
}

// Hop levels over tight edges (fl(dist[u] + w) == dist[v]) from the source;
// used to walk paths when zero-weight edges create equal-distance ties.
__global__ void tight_level_k(DirView d, const double* __restrict__ w0, const double* __restrict__ w1,
                              const uint32_t* __restrict__ F, uint64_t f,
                              const uint64_t* __restrict__ pos, uint64_t T,
                              const unsigned long long* __restrict__ dist, int32_t* level,
                              int32_t lvl, uint32_t* __restrict__ N, uint32_t* __restrict__ cnt) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t span = ((T + stride - 1) / stride) * stride;
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < span; e += stride) {
    bool take = false;
    uint32_t v = 0;
    if (e < T) {
      uint64_t i = owner_in_pos(pos, f, e);
      uint32_t u = F[i];
      uint32_t slot;
      bool second;
      v = dv_nbr(d, u, (uint32_t)(e - pos[i]), &slot, &second);
      double w = second ? w1[slot] : w0[slot];
      double nd = __dadd_rn(__longlong_as_double((long long)dist[u]), w);
      if ((unsigned long long)__double_as_longlong(nd) == dist[v] && dist[v] != kInfBits &&
          level[v] < 0)
        take = atomicCAS(&level[v], -1, lvl + 1) == -1;
    }
    append_w(N, cnt, take, v);
  }
}

__global__ void fill_u64_k(unsigned long long* p, uint64_t n, unsigned long long v) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

// One block walks the path back from the target: at node v it scans the
// reverse adjacency for tight predecessors and keeps the smallest
// (dist, id), restricted to (dist[u], u) < (dist[v], v) so a zero-weight
// cycle cannot loop -- or, when level is given, to predecessors one tight
// hop closer to the source.
__global__ void weighted_backtrack_k(DirView rev, const double* __restrict__ rw0,
                                     const double* __restrict__ rw1,
                                     const unsigned long long* __restrict__ dist,
                                     const int32_t* __restrict__ level, uint32_t source,
                                     uint32_t target, uint64_t cap, uint32_t* __restrict__ path,
                                     unsigned long long* __restrict__ out_len) {
  __shared__ unsigned long long best_d[kBlock / 32];
  __shared__ uint32_t best_u[kBlock / 32];
  __shared__ uint32_t s_cur;
  __shared__ uint64_t s_len;
  __shared__ int s_fail;
  if (threadIdx.x == 0) {
    s_cur = target;
    s_len = 0;
    s_fail = 0;
    path[0] = target;
    s_len = 1;
  }
  __syncthreads();
  while (true) {
    uint32_t v = s_cur;
    if (v == source || s_fail || s_len >= cap) break;
    unsigned long long dv = dist[v];
    double dvd = __longlong_as_double((long long)dv);
    unsigned long long bd = ~0ull;
    uint32_t bu = 0xFFFFFFFFu;
    uint32_t deg = dv_deg(rev, v);
    for (uint32_t j = threadIdx.x; j < deg; j += blockDim.x) {
      uint32_t slot;
      bool second;
      uint32_t u = dv_nbr(rev, v, j, &slot, &second);
      if (u == v) continue;
      unsigned long long du = dist[u];
      if (du == kInfBits) continue;
      double w = second ? rw1[slot] : rw0[slot];
      double nd = __dadd_rn(__longlong_as_double((long long)du), w);
      if ((unsigned long long)__double_as_longlong(nd) != dv || !(nd == dvd)) continue;
      bool before = level ? (level[u] >= 0 && level[u] + 1 == level[v])
                          : (du < dv || (du == dv && u < v));
      if (!before) continue;
      if (du < bd || (du == bd && u < bu)) {
        bd = du;
        bu = u;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long od = __shfl_down_sync(0xffffffffu, bd, o);
      uint32_t ou = __shfl_down_sync(0xffffffffu, bu, o);
      if (od < bd || (od == bd && ou < bu)) {
        bd = od;
        bu = ou;
      }
    }
    if ((threadIdx.x & 31) == 0) {
      best_d[threadIdx.x >> 5] = bd;
      best_u[threadIdx.x >> 5] = bu;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long fd = ~0ull;
      uint32_t fu = 0xFFFFFFFFu;
      for (int k = 0; k < (int)(blockDim.x / 32); k++)
        if (best_d[k] < fd || (best_d[k] == fd && best_u[k] < fu)) {
          fd = best_d[k];
          fu = best_u[k];
        }
      if (fu == 0xFFFFFFFFu) {
        s_fail = 1;
      } else {
        path[s_len] = fu;
        s_len = s_len + 1;
        s_cur = fu;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *out_len = s_fail ? 0ull : s_len;
}

__global__ void bits_to_costs_k(const uint32_t* __restrict__ path, uint64_t len,
                                const unsigned long long* __restrict__ dist,
                                double* __restrict__ cost) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len;
       i += (uint64_t)gridDim.x * blockDim.x)
    cost[i] = __longlong_as_double((long long)dist[path[i]]);
}

}  // namespace

// Distances from source over view d (m slots a CSR) with per-slot weights
// w0/w1 into dist (n u64 bit patterns of f64, +inf = unreachable).
void sssp_run(const DirView& d, const double* w0, const double* w1, uint64_t n, uint64_t m,
              uint32_t source, unsigned long long* dist, cudaStream_t s) {
  fill_u64_k<<<grid_for(n), kBlock, 0, s>>>(dist, n, kInfBits);
  UG_LAUNCH_CHECK();
  if ((uint64_t)source >= n) return;
  const uint64_t entries = n + (d.off1 ? 2 : 1) * m / kSpan + 1;
  Scratch<uint2> list(2 * entries, s);
  Scratch<uint32_t> marks(2 * n, s), fars(2 * n, s);
  Scratch<SsspState> st(1, s);
  UG_CUDA(cudaMemsetAsync(marks.get(), 0, 2 * n * sizeof(uint32_t), s));
  SsspArgs a;
  a.d = d;
  a.w0 = w0;
  a.w1 = w1;
  a.n = n;
  a.dist = dist;
  a.stamp = marks.get();
  a.far = marks.get() + n;
  a.list[0] = list.get();
  a.list[1] = list.get() + entries;
  a.far_list[0] = fars.get();
  a.far_list[1] = fars.get() + n;
  a.st = st.get();
  sssp_init_k<<<1, 1024, 0, s>>>(a, source, m);
  UG_LAUNCH_CHECK();
  int dev = 0;
  UG_CUDA(cudaGetDevice(&dev));
  const unsigned grid = grid_for(entries * kEntryLanes, kBlock, (unsigned)sm_count(dev) * kSsspBlocks);
  uint32_t mode = kNear;
  for (int run = 16; mode != kSsspDone; run = run < 64 ? 2 * run : run) {
    for (int i = 0; i < run; i++) {
      sssp_round_k<<<grid, kBlock, 0, s>>>(a);
      UG_LAUNCH_CHECK();
    }
    mode = read_u32(&st.get()->mode, s);
  }
}

void dijkstra_run(TopoImpl* t, const double* d_weights, uint32_t source, int dir, double* d_out,
                  cudaStream_t s) {
  DirView d = dir_view(t, dir, s);
  DirWeights w;
  gather_dir_weights(t, d, d_weights, w, s);
  sssp_run(d, w.w0.get(), w.w1.get(), t->n, t->m, source, (unsigned long long*)d_out, s);
}

int64_t weighted_path_run(TopoImpl* t, const double* d_weights, uint32_t source, uint32_t target,
                          int dir, uint32_t* path, double* costs, uint64_t cap, cudaStream_t s) {
  const uint64_t n = t->n;
  if ((uint64_t)source >= n || (uint64_t)target >= n) return -1;  // bfs.rs:208-210
  if (source == target) {                                          // bfs.rs:211-213
    UG_CHECK(cap >= 1, URSA_GPU_ETRUNC, "path buffer too small");
    path[0] = source;
    if (costs) costs[0] = 0.0;
    return 1;
  }
  DirView d = dir_view(t, dir, s);
  DirWeights w;
  gather_dir_weights(t, d, d_weights, w, s);
  Scratch<unsigned long long> dist(n, s);
  sssp_run(d, w.w0.get(), w.w1.get(), n, t->m, source, dist.get(), s);
  unsigned long long dt = 0;
  UG_CUDA(cudaMemcpyAsync(&dt, dist.get() + target, 8, cudaMemcpyDeviceToHost, s));
  UG_CUDA(cudaStreamSynchronize(s));
  if (dt == kInfBits) return -1;  // unreachable (bfs.rs:245-247)
  DirView rv = reverse_view(t, dir, s);
  DirWeights rw;
  gather_dir_weights(t, rv, d_weights, rw, s);
  Scratch<uint32_t> dpath(n, s);
  Scratch<unsigned long long> dlen(1, s);
  weighted_backtrack_k<<<1, kBlock, 0, s>>>(rv, rw.w0.get(), rw.w1.get(), dist.get(), nullptr,
                                            source, target, n, dpath.get(), dlen.get());
  UG_LAUNCH_CHECK();
  unsigned long long len = 0;
  UG_CUDA(cudaMemcpyAsync(&len, dlen.get(), 8, cudaMemcpyDeviceToHost, s));
  UG_CUDA(cudaStreamSynchronize(s));
  if (len == 0) {
    // Zero-weight ties: walk back along hop levels of the tight-edge graph.
    Scratch<int32_t> level(n, s);
    UG_CUDA(cudaMemsetAsync(level.get(), 0xFF, n * sizeof(int32_t), s));
    FrontierBufs b;
    b.alloc(n, s);
    UG_CUDA(cudaMemsetAsync(level.get() + source, 0, sizeof(int32_t), s));
    UG_CUDA(cudaMemcpyAsync(b.F.get(), &source, sizeof(uint32_t), cudaMemcpyHostToDevice, s));
    uint32_t f = 1;
    int32_t lvl = 0;
    while (f > 0) {
      uint64_t T = frontier_scan(d, b.F.get(), f, b.pos.get(), s);
      if (T == 0) break;
      UG_CUDA(cudaMemsetAsync(b.count.get(), 0, sizeof(uint32_t), s));
      tight_level_k<<<grid_for(T, kBlock, 148u * 64u), kBlock, 0, s>>>(
          d, w.w0.get(), w.w1.get(), b.F.get(), f, b.pos.get(), T, dist.get(), level.get(), lvl,
          b.N.get(), b.count.get());
      UG_LAUNCH_CHECK();
      uint32_t next = read_u32(b.count.get(), s);
      swap(b.F, b.N);
      f = next;
      lvl++;
    }
    weighted_backtrack_k<<<1, kBlock, 0, s>>>(rv, rw.w0.get(), rw.w1.get(), dist.get(), level.get(),
                                              source, target, n, dpath.get(), dlen.get());
    UG_LAUNCH_CHECK();
    UG_CUDA(cudaMemcpyAsync(&len, dlen.get(), 8, cudaMemcpyDeviceToHost, s));
    UG_CUDA(cudaStreamSynchronize(s));
  }
  UG_CHECK(len > 0, URSA_GPU_EINVAL, "weighted path walk found no predecessor");
  if (len > cap) return -(int64_t)len - 2;
  // reverse into forward order on the host copy
  std::vector<uint32_t> h(len);
  UG_CUDA(cudaMemcpyAsync(h.data(), dpath.get(), len * 4, cudaMemcpyDeviceToHost, s));
  Scratch<double> dcost(len, s);
  std::vector<double> hc(len);
  if (costs) {
    bits_to_costs_k<<<grid_for(len), kBlock, 0, s>>>(dpath.get(), len, dist.get(), dcost.get());
    UG_LAUNCH_CHECK();
    UG_CUDA(cudaMemcpyAsync(hc.data(), dcost.get(), len * 8, cudaMemcpyDeviceToHost, s));
  }
  UG_CUDA(cudaStreamSynchronize(s));
  for (uint64_t i = 0; i < len; i++) {
    path[i] = h[len - 1 - i];
    if (costs) costs[i] = hc[len - 1 - i];
  }
  return (int64_t)len;
}

}  // namespace ug

using namespace ug;

extern "C" {

int ursa_gpu_dijkstra_distances(ursa_gpu_topo* t, const double* weights, uint64_t n_weights,
                                uint32_t source, int dir, double* out) {
  return guard([&] {
    UG_CHECK(t, URSA_GPU_EINVAL, "topology is NULL");
    UG_CHECK(dir >= 0 && dir <= 2, URSA_GPU_EINVAL, "direction must be 0, 1 or 2");
    TopoImpl* ti = &t->impl;
    UG_CHECK(n_weights == ti->m, URSA_GPU_EINVAL, "weights length must equal the edge count");
    UG_CHECK(ti->m == 0 || weights, URSA_GPU_EINVAL, "weights is NULL");
    if (ti->n == 0) return;
    UG_CHECK(out, URSA_GPU_EINVAL, "out is NULL");
    cudaStream_t s = thread_stream(ti->device);
    Scratch<double> dw(ti->m ? ti->m : 1, s), dout(ti->n, s);
    if (ti->m) UG_CUDA(cudaMemcpyAsync(dw.get(), weights, ti->m * 8, cudaMemcpyHostToDevice, s));
    check_sssp_weights_device(dw.get(), ti->m, s);
    dijkstra_run(ti, dw.get(), source, dir, dout.get(), s);
    UG_CUDA(cudaMemcpyAsync(out, dout.get(), ti->n * 8, cudaMemcpyDeviceToHost, s));
    UG_CUDA(cudaStreamSynchronize(s));
  });
}

int ursa_gpu_shortest_path_weighted_with_cost(ursa_gpu_topo* t, const double* weights,
                                              uint64_t n_weights, uint32_t source,
                                              uint32_t target, int dir, uint32_t* path,
                                              double* costs, uint64_t cap, int64_t* len) {
  return guard([&] {
    UG_CHECK(t && len, URSA_GPU_EINVAL, "topology or len is NULL");
    UG_CHECK(dir >= 0 && dir <= 2, URSA_GPU_EINVAL, "direction must be 0, 1 or 2");
    *len = -1;
    TopoImpl* ti = &t->impl;
    UG_CHECK(n_weights == ti->m, URSA_GPU_EINVAL, "weights length must equal the edge count");
    UG_CHECK(ti->m == 0 || weights, URSA_GPU_EINVAL, "weights is NULL");
    cudaStream_t s = thread_stream(ti->device);
    Scratch<double> dw(ti->m ? ti->m : 1, s);
    if (ti->m) UG_CUDA(cudaMemcpyAsync(dw.get(), weights, ti->m * 8, cudaMemcpyHostToDevice, s));
    check_sssp_weights_device(dw.get(), ti->m, s);
    int64_t r = weighted_path_run(ti, dw.get(), source, target, dir, path, costs, cap, s);
    if (r < -1) {
      *len = -r - 2;
      throw Error(URSA_GPU_ETRUNC, "path buffer too small");
    }
    *len = r;
  });
}

}  // extern "C"
