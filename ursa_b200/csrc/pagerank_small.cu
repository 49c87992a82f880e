// pagerank_small.cu -- PageRank of graphs that fit one thread-block cluster
// (ursa-core/src/algo/pagerank.rs:44-124).
//
// On a graph of a thousand nodes the persistent kernel of pagerank.cu spends
// its time on what makes it fast on a large one: per iteration every block
// loads a 192 KB slice of shares and crosses two grid barriers (about 17 us),
// after an execution layout that costs a new topology 0.4 ms and more.  Here
// one cluster of eight CTAs runs the whole call straight from the in-CSR: each
// CTA owns a run of rows (equal rows + edges), keeps every node's share in its
// own shared memory, and writes a row's new share to all eight (distributed
// shared memory), so an iteration costs one cluster barrier and no trip to L2
// for the shares.  The rows' sources are kept in shared memory too, as 16-bit
// ids: those of long rows always, the others where they fit.
// The arithmetic is pagerank.cu's, operation for operation: f32 shares, a row
// of up to 64 in-edges summed by one lane in CSR order with a compensated f32
// pair, longer rows in pieces of 128 edges combined in that kernel's order;
// f64 ranks; residual and dangling mass summed exactly, in fixed point.  So
// both kernels give the same ranks bit for bit on the graphs compared.  A call
// on 1,000 nodes, 10,000 edges: 234 us before, 70 now; 30 iterations on R-MAT
// with 14,336 nodes and 140,000 edges, ranks to the host: 591 and 475; with
// 2,000 nodes and 200,000 edges 642 and 397.  What is left is the launch and,
// per iteration, the chain of one row's additions, the block-wide waits and the
// cluster barrier (about 4 us).
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "fixedpoint.cuh"
#include "topo.cuh"

namespace cg = cooperative_groups;

namespace ug {

namespace {

constexpr int kCtas = 8;  // the portable cluster size
constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
// What a CTA keeps in shared memory has to fit (small_bytes): two share
// buffers (8 bytes a node), its rows (18 bytes each, at most a quarter of all
// and one), and its rows of more than 64 edges with their pieces and sources.
// Those are the larger part of a skewed graph's edges, and a lane walks one
// piece: from global memory every lane would read a line of its own, so a graph
// whose pieces do not fit takes the large kernel.  (One hub of 100,000 edges:
// 2,170 us a call with its sources in global memory, 635 with the large kernel.)
constexpr uint64_t kMaxNodes = 14336;
constexpr uint64_t kMaxEdges = 1u << 18;  // R-MAT with 14,336 nodes and twice as many: the large kernel is faster
constexpr size_t kSmemBytes = 227u * 1024u - 3u * 1024u;  // under 2 KB are static
static_assert(kWarps == 32, "one warp sums the warps' sums");
constexpr uint32_t kShort = 8;     // rows up to this are kept together, so that lanes end together
constexpr uint32_t kDirect = 64;   // rows up to this: one lane
constexpr uint32_t kPiece = 128;   // longer ones: a lane per piece of this many edges,
constexpr uint32_t kPieceStride = kPiece + 2;  // u16 between two pieces' sources: an odd number of banks
constexpr uint32_t kWide = 32;     // combined by one lane up to this many pieces, else a warp

struct SmallArgs {
  const uint32_t* in_off;
  const uint32_t* in_src;
  const uint32_t* out_off;
  uint32_t n, m;
  double damping, tol;
  uint32_t max_iter;
  uint32_t row_cost;  // of a row, in edges: at least the mean in-degree
  double* out;
  double* delta_out;    // optional: the last residual
  uint32_t* iters_out;  // optional: iterations run
};

// First row of CTA c: rows are cut at equal (rows * row_cost + edges), so no
// CTA gets more than a quarter of the rows and one.
__device__ uint32_t first_row(const SmallArgs& a, uint32_t c) {
  const uint64_t want = (uint64_t)c * ((uint64_t)a.n * a.row_cost + a.m) / kCtas;
  uint32_t lo = 0, hi = a.n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if ((uint64_t)a.in_off[mid] + (uint64_t)mid * a.row_cost < want) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// (residual, dangling mass) in fixed point, as in pagerank.cu: exact, in any
// order.
struct Sums {
  u128 delta, dang;
};

// Sums over the warp, valid in every lane: limbs of 26 bits, whose 32-lane
// sums fit the 32 bits of a warp-wide add (shuffles of whole words: 20 us
// more for a call on 1,000 nodes).
__device__ __forceinline__ u128 warp_sum(u128 v) {
  constexpr int kBits = 26;
  if (!__any_sync(0xffffffffu, v != 0)) return 0;  // warps without rows, graphs without dangling nodes
  u128 t = 0;
#pragma unroll
  for (int i = 0; i * kBits < 128; i++) {
    const uint32_t limb = (uint32_t)(v >> (i * kBits)) & ((1u << kBits) - 1u);
    t += (u128)__reduce_add_sync(0xffffffffu, limb) << (i * kBits);
  }
  return t;
}

__device__ __forceinline__ Sums warp_sum(Sums v) { return Sums{warp_sum(v.delta), warp_sum(v.dang)}; }

// The CTA's sums, put into every CTA's table (lane c of warp 0 writes CTA c's).
__device__ __forceinline__ void publish(cg::cluster_group& cluster, FxPair* table, FxPair* warps, Sums v) {
  const uint32_t lane = threadIdx.x & 31;
  v = warp_sum(v);
  if (lane == 0) warps[threadIdx.x >> 5] = fx_pack(v.delta, v.dang);
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const FxPair w = warps[lane];
  v = warp_sum(Sums{fx_delta(w), fx_dang(w)});
  if (lane < kCtas) cluster.map_shared_rank(table, lane)[cluster.block_rank()] = fx_pack(v.delta, v.dang);
}

// The table's total, the same in every thread of the cluster.
__device__ __forceinline__ double2 total(const FxPair* table) {
  const uint32_t lane = threadIdx.x & 31;
  Sums t{0, 0};
  if (lane < kCtas) t = Sums{fx_delta(table[lane]), fx_dang(table[lane])};
  t = warp_sum(t);
  return make_double2(fx_value(t.delta), fx_value(t.dang));
}

__global__ void __cluster_dims__(kCtas, 1, 1) __launch_bounds__(kThreads, 1) pr_small_k(SmallArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ FxPair part[2][kCtas];  // every CTA's sums, by parity
  __shared__ FxPair warps[kWarps];   // this CTA's, per warp
  __shared__ uint32_t s_rows[kCtas + 1];
  __shared__ uint32_t s_warp[kWarps];
  cg::cluster_group cluster = cg::this_cluster();
  cluster.barrier_arrive();  // waited for before the first write to another CTA's shared memory
  const uint32_t me = cluster.block_rank();
  const int lane = threadIdx.x & 31;
  if (threadIdx.x <= kCtas) s_rows[threadIdx.x] = threadIdx.x == kCtas ? a.n : first_row(a, threadIdx.x);
  __syncthreads();
  const uint32_t r0 = s_rows[me], rows = s_rows[me + 1] - r0;
  const uint32_t e0 = a.in_off[r0], edges = a.in_off[r0 + rows] - e0;
  // layout: two share buffers [n], this CTA's ranks, offsets, divisors and
  // its rows by length (short, mid, long), the long rows' pieces, then the
  // sources if they fit
  float* x0 = reinterpret_cast<float*>(smem);
  float* x1 = x0 + a.n;
  double* rank = reinterpret_cast<double*>(x1 + a.n);  // 8 n bytes in: aligned
  uint32_t* off = reinterpret_cast<uint32_t*>(rank + rows);
  uint32_t* div = off + rows + 1;
  uint16_t* by_len = reinterpret_cast<uint16_t*>(div + rows);
  const double nf = (double)a.n;
  const double first = 1.0 / nf;
  if (threadIdx.x == 0) off[rows] = edges;
  Sums acc{0, 0};
  for (uint32_t r = threadIdx.x; r < rows; r += kThreads) {
    const uint32_t u = r0 + r;
    const uint32_t b = a.in_off[u];
    off[r] = b - e0;
    const uint32_t d = a.out_off[u + 1] - a.out_off[u];
    div[r] = d;
    rank[r] = first;
    if (d == 0) acc.dang += fx_of(first);
  }
  for (uint32_t u = threadIdx.x; u < a.n; u += kThreads) {  // every CTA fills its own copy
    const uint32_t d = a.out_off[u + 1] - a.out_off[u];
    x0[u] = d ? (float)(first / (double)d) : 0.f;
  }
  // A CTA's shared memory may be written from another only once it has
  // started; the arrival was at the kernel's entry, so the loads above hide
  // the wait.
  cluster.barrier_wait();
  publish(cluster, part[0], warps, acc);
  __syncthreads();
  // rows by length, in row order within a length: a lane's rows, and so the
  // order of the sums below, are the same in every run
  uint32_t ends[3], filled = 0;
  for (int k = 0; k < 3; k++) {
    for (uint32_t rb = 0; rb < rows; rb += kThreads) {
      const uint32_t r = rb + threadIdx.x;
      bool in = false;
      if (r < rows) {
        const uint32_t len = off[r + 1] - off[r];
        in = k == (len <= kShort ? 0 : len <= kDirect ? 1 : 2);
      }
      const uint32_t b = __ballot_sync(0xffffffffu, in);
      if (lane == 0) s_warp[threadIdx.x >> 5] = __popc(b);
      __syncthreads();
      uint32_t at = filled, total = 0;
      for (uint32_t w = 0; w < kWarps; w++) {
        if (w < threadIdx.x >> 5) at += s_warp[w];
        total += s_warp[w];
      }
      if (in) by_len[at + __popc(b & ((1u << lane) - 1u))] = (uint16_t)r;
      filled += total;
      __syncthreads();
    }
    ends[k] = filled;
  }
  // the long rows: edges before each (those of long rows alone), first edge,
  // first piece (one past the last closes both lists); and each piece's row
  const uint32_t n_long = ends[2] - ends[1];
  const uint16_t* longs = by_len + ends[1];
  const size_t used = reinterpret_cast<unsigned char*>(by_len + rows) - smem;
  F2* partial = reinterpret_cast<F2*>(smem + (used + 7) / 8 * 8);
  if (threadIdx.x < 32) {
    uint32_t sum = 0;
    for (uint32_t i = lane; i < n_long; i += 32) sum += (off[longs[i] + 1] - off[longs[i]] + kPiece - 1) / kPiece;
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) s_warp[0] = sum;
  }
  __syncthreads();
  const uint32_t n_pieces = s_warp[0];
  uint32_t* before = reinterpret_cast<uint32_t*>(partial + n_pieces);
  uint32_t* begin = before + n_long + 1;
  uint16_t* piece_row = reinterpret_cast<uint16_t*>(begin + n_long);
  uint16_t* first_piece = piece_row + n_pieces;
  if (threadIdx.x < 32) {
    uint32_t at = 0, ate = 0;
    for (uint32_t ib = 0; ib < n_long; ib += 32) {
      const uint32_t i = ib + lane;
      const uint32_t b = i < n_long ? off[longs[i]] : 0u;
      const uint32_t len = i < n_long ? off[longs[i] + 1] - b : 0u;
      const uint32_t c = (len + kPiece - 1) / kPiece;
      uint32_t incl = c, incle = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o), te = __shfl_up_sync(0xffffffffu, incle, o);
        if (lane >= o) {
          incl += t;
          incle += te;
        }
      }
      if (i < n_long) {
        first_piece[i] = (uint16_t)(at + incl - c);
        before[i] = ate + incle - len;
        begin[i] = b;
      }
      at += __shfl_sync(0xffffffffu, incl, 31);
      ate += __shfl_sync(0xffffffffu, incle, 31);
    }
    if (lane == 0) {
      first_piece[n_long] = (uint16_t)at;
      before[n_long] = ate;
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < n_long; i += kThreads)
    for (uint32_t q = first_piece[i]; q < first_piece[i + 1]; q++) piece_row[q] = (uint16_t)i;
  // from here on off[] counts the edges of the other rows alone
  if (n_long)
    for (uint32_t r = threadIdx.x; r <= rows; r += kThreads) {
      uint32_t lo = 0, hi = n_long;  // long rows before r
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (longs[mid] < r) lo = mid + 1; else hi = mid;
      }
      off[r] -= before[lo];
    }
  __syncthreads();
  auto piece_end = [&](uint32_t i, uint32_t b) { return min(b + kPiece, begin[i] + before[i + 1] - before[i]); };
  // sources: of the pieces first, kPieceStride apart, then of the other rows
  uint16_t* psrc = first_piece + n_long + 1;
  const bool pcached = reinterpret_cast<unsigned char*>(psrc + n_pieces * kPieceStride) <= smem + kSmemBytes;
  uint16_t* src = psrc + (pcached ? n_pieces * kPieceStride : 0u);
  const bool cached = reinterpret_cast<unsigned char*>(src + off[rows]) <= smem + kSmemBytes;
  if (pcached)
    for (uint32_t q = threadIdx.x >> 5; q < n_pieces; q += kWarps) {
      const uint32_t i = piece_row[q], b = begin[i] + (q - first_piece[i]) * kPiece, e = piece_end(i, b);
      for (uint32_t k = b + lane; k < e; k += 32) psrc[q * kPieceStride + k - b] = (uint16_t)a.in_src[e0 + k];
    }
  if (cached && !n_long)
    for (uint32_t k = threadIdx.x; k < edges; k += kThreads) src[k] = (uint16_t)a.in_src[e0 + k];
  else if (cached)
    for (uint32_t r = threadIdx.x; r < rows; r += kThreads)
      for (uint32_t b = off[r], k = 0, g = a.in_off[r0 + r]; k < off[r + 1] - b; k++)
        src[b + k] = (uint16_t)a.in_src[g + k];
  cluster.sync();
  uint32_t it = 0;
  double2 sums = total(part[0]);
  double delta = 0.0;
  float* cur = x0;
  float* nxt = x1;
  for (; it < a.max_iter;) {
    const double dm = sums.y;
    // base = (1-d)/n + d*dangling_mass/n   (pagerank.rs:79)
    const double base = __dadd_rn(__ddiv_rn(1.0 - a.damping, nf), __ddiv_rn(__dmul_rn(a.damping, dm), nf));
    acc = Sums{0, 0};
    auto finish = [&](uint32_t r, double sum) {  // next[u] = base + d * contrib(u)  (:81-83)
      const double nx = __dadd_rn(base, __dmul_rn(a.damping, sum));
      acc.delta += fx_of(fabs(__dsub_rn(nx, rank[r])));
      rank[r] = nx;
      const uint32_t d = div[r];
      if (d == 0) acc.dang += fx_of(nx);
      const float share = d ? (float)(nx / (double)d) : 0.f;
#pragma unroll
      for (int c = 0; c < kCtas; c++) cluster.map_shared_rank(nxt, c)[r0 + r] = share;
    };
    auto sum = [&](const uint16_t* kept, const uint32_t* far, uint32_t len) {  // Kahan, in CSR order
      float v = 0.f, c = 0.f;
      for (uint32_t k = 0; k < len; k++) {
        const float y = __fsub_rn(cur[kept ? (uint32_t)kept[k] : far[k]], c);
        const float t = __fadd_rn(v, y);
        c = __fsub_rn(__fsub_rn(t, v), y);
        v = t;
      }
      return F2{v, -c};
    };
    auto row_sum = [&](uint32_t r) {
      return f2_value(sum(cached ? src + off[r] : nullptr, cached ? nullptr : a.in_src + a.in_off[r0 + r],
                          off[r + 1] - off[r]));
    };
    for (uint32_t i = threadIdx.x; i < ends[0]; i += kThreads) finish(by_len[i], row_sum(by_len[i]));
    for (uint32_t i = ends[0] + threadIdx.x; i < ends[1]; i += kThreads) finish(by_len[i], row_sum(by_len[i]));
    for (uint32_t q = threadIdx.x; q < n_pieces; q += kThreads) {
      const uint32_t i = piece_row[q], b = begin[i] + (q - first_piece[i]) * kPiece;
      partial[q] = sum(pcached ? psrc + q * kPieceStride : nullptr, a.in_src + e0 + b, piece_end(i, b) - b);
    }
    if (n_long) {
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < n_long; i += kThreads) {
        const uint32_t q0 = first_piece[i], q1 = first_piece[i + 1];
        if (q1 - q0 > kWide) continue;
        F2 t = f2_zero();
        for (uint32_t q = q0; q < q1; q++) t = f2_combine(t, partial[q]);
        finish(longs[i], f2_value(t));
      }
      for (uint32_t i = threadIdx.x >> 5; i < n_long; i += kWarps) {
        const uint32_t q0 = first_piece[i], q1 = first_piece[i + 1];
        if (q1 - q0 <= kWide) continue;
        F2 t[4] = {f2_zero(), f2_zero(), f2_zero(), f2_zero()};  // four streams per lane, then a fixed tree
        uint32_t q = q0 + lane;
        for (; q + 96 < q1; q += 128)
#pragma unroll
          for (int j = 0; j < 4; j++) t[j] = f2_combine(t[j], partial[q + 32 * j]);
#pragma unroll
        for (int j = 0; j < 4; j++, q += 32)
          if (q < q1) t[j] = f2_combine(t[j], partial[q]);
        F2 v = f2_combine(f2_combine(t[0], t[1]), f2_combine(t[2], t[3]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
          v = f2_combine(v, F2{__shfl_down_sync(0xffffffffu, v.hi, o), __shfl_down_sync(0xffffffffu, v.lo, o)});
        if (lane == 0) finish(longs[i], f2_value(v));
      }
    }
    publish(cluster, part[(it + 1) & 1], warps, acc);
    cluster.sync();  // new shares and partial sums are in place everywhere
    sums = total(part[(it + 1) & 1]);
    delta = sums.x;
    float* t = cur;
    cur = nxt;
    nxt = t;
    it++;
    if (delta < a.tol) break;  // the same sum in every CTA
  }
  for (uint32_t r = threadIdx.x; r < rows; r += kThreads) a.out[r0 + r] = rank[r];
  if (me == 0 && threadIdx.x == 0) {
    if (a.delta_out) *a.delta_out = delta;
    if (a.iters_out) *a.iters_out = it;
  }
  cluster.sync();  // no CTA leaves while another may still write its shared memory
}

}  // namespace

// Shared memory of a CTA up to its pieces' sources.
static __host__ __device__ uint64_t small_bytes(uint64_t n, uint64_t rows, uint64_t longs, uint64_t pieces) {
  return (8 * n + 18 * rows + 4 + 7) / 8 * 8 + 10 * pieces + 10 * (longs + 1) + 2 * kPieceStride * pieces;
}

// Whether every CTA's rows and pieces fit.
__global__ void __launch_bounds__(kThreads) pr_small_check_k(SmallArgs a, uint32_t* fits) {
  __shared__ uint32_t s_rows[kCtas + 1], pieces[kCtas], longs[kCtas];
  if (threadIdx.x <= kCtas) s_rows[threadIdx.x] = threadIdx.x == kCtas ? a.n : first_row(a, threadIdx.x);
  if (threadIdx.x < kCtas) pieces[threadIdx.x] = longs[threadIdx.x] = 0;
  __syncthreads();
  for (uint32_t r = threadIdx.x; r < a.n; r += kThreads) {
    const uint32_t len = a.in_off[r + 1] - a.in_off[r];
    if (len <= kDirect) continue;
    uint32_t c = 0;
    while (r >= s_rows[c + 1]) c++;
    atomicAdd(&pieces[c], (len + kPiece - 1) / kPiece);
    atomicAdd(&longs[c], 1u);
  }
  __syncthreads();
  if (threadIdx.x) return;
  bool all = true;
  for (int c = 0; c < kCtas; c++)
    all = all && small_bytes(a.n, s_rows[c + 1] - s_rows[c], longs[c], pieces[c]) <= kSmemBytes;
  *fits = all;
}

static SmallArgs small_args(TopoImpl* t) {
  SmallArgs a{};
  a.in_off = t->in.off.get();
  a.in_src = t->in.tgt.get();
  a.out_off = t->out.off.get();
  a.n = (uint32_t)t->n;
  a.m = (uint32_t)t->m;
  a.row_cost = (uint32_t)std::max<uint64_t>(1, (t->m + t->n - 1) / t->n);
  return a;
}

// Looked at once per topology, and not where any graph of its size fits.
bool pagerank_small_fits(TopoImpl* t, cudaStream_t s) {
  if (t->n > kMaxNodes || t->m > kMaxEdges) return false;
  const uint64_t longs = t->m / (kDirect + 1), pieces = longs + t->m / kPiece;  // at most
  if (small_bytes(t->n, t->n / 4 + 2, longs, pieces) <= kSmemBytes) return true;
  ensure_in(t, s);
  std::lock_guard<std::mutex> g(t->mu);
  if (t->pr_small < 0) {
    Scratch<uint32_t> fits(1, s);
    pr_small_check_k<<<1, kThreads, 0, s>>>(small_args(t), fits.get());
    UG_LAUNCH_CHECK();
    uint32_t f = 0;
    UG_CUDA(cudaMemcpyAsync(&f, fits.get(), sizeof(f), cudaMemcpyDeviceToHost, s));
    UG_CUDA(cudaStreamSynchronize(s));
    t->pr_small = (int)f;
  }
  return t->pr_small != 0;
}

void pagerank_small_run(TopoImpl* t, const ursa_gpu_pagerank_params& p, double* d_out, cudaStream_t s,
                        ursa_gpu_pagerank_stats* stats) {
  ensure_in(t, s);
  {
    static std::mutex mu;
    static bool ready[64] = {false};
    std::lock_guard<std::mutex> g(mu);
    UG_CHECK(t->device >= 0 && t->device < 64, URSA_GPU_EINVAL, "device index out of range");
    if (!ready[t->device]) {
      UG_CUDA(cudaFuncSetAttribute(pr_small_k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
      ready[t->device] = true;
    }
  }
  SmallArgs a = small_args(t);
  a.damping = p.damping;
  a.tol = p.tol;
  a.max_iter = p.max_iter;
  a.out = d_out;
  Scratch<double> info;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (stats) {
    info.alloc(2, s);
    a.delta_out = info.get();
    a.iters_out = reinterpret_cast<uint32_t*>(info.get() + 1);
    UG_CUDA(cudaEventCreate(&e0));
    UG_CUDA(cudaEventCreate(&e1));
    UG_CUDA(cudaEventRecord(e0, s));
  }
  pr_small_k<<<kCtas, kThreads, kSmemBytes, s>>>(a);
  UG_LAUNCH_CHECK();
  if (stats) {
    double h[2];
    UG_CUDA(cudaEventRecord(e1, s));
    UG_CUDA(cudaMemcpyAsync(h, info.get(), sizeof(h), cudaMemcpyDeviceToHost, s));
    UG_CUDA(cudaStreamSynchronize(s));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    stats->iterations = *reinterpret_cast<uint32_t*>(h + 1);
    stats->last_delta = h[0];
    stats->device_ms = ms;
  }
}

}  // namespace ug
