// primitives.cu -- reduce-then-scan prefix sums and a stable LSD radix sort.
//
// The radix sort is the core of the byte-exact CSR build: a stable sort of
// edge rows by their grouping endpoint reproduces ursa-core's counting sort
// exactly (rows keep their original order inside each node's segment,
// ursa-core/src/topology.rs:109-114).  Each 8-bit pass is
//   upsweep:   per-tile digit histograms, written digit-major,
//   scan:      one exclusive scan over the digit-major histogram,
//   downsweep: per-tile stable ranking (warp match_any + per-warp digit
//              counters, warps own contiguous sub-tiles) and scatter.
#include "primitives.cuh"

namespace ug {

namespace {

constexpr int kScanTile = 2048;  // 256 threads x 8 items
constexpr int kRadixItems = 16;  // per thread
constexpr int kRadixTile = kBlock * kRadixItems;  // 4096
constexpr int kWarps = kBlock / 32;
constexpr int kDownBlock = 512;  // threads of a tile's block in radix_carry_k
constexpr int kDownItems = kRadixTile / kDownBlock;
constexpr int kDownWarps = kDownBlock / 32;
// From 3 * 2^24 rows (a 200 MB column: its gather leaves L2) to 2^30 (above,
// two buffers more would count) the gathered column travels with the pairs: at
// 65M rows three passes take 600 + 620 + 535 us against 460 + 466 + 1,187 with
// the gather in the last one (a build and a PageRank 9.07 -> 8.07 ms).  Where
// the rows come sorted by source the out-CSR's gather is a stream: there the
// two are even at 67M rows, and the gather is 1% faster at 48M, 2% at 36M.
constexpr uint64_t kCarryMin = 3ull << 24, kCarryMax = 1ull << 30;

__device__ __forceinline__ int pad(int i) { return i + (i >> 5); }

template <class T>
__device__ T block_exclusive_scan(T v, T* block_total) {
  __shared__ T warp_tot[kWarps];
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[w] = x;
  __syncthreads();
  if (w == 0) {
    T t = lane < kWarps ? warp_tot[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    if (lane < kWarps) warp_tot[lane] = t;  // inclusive
  }
  __syncthreads();
  T warp_excl = w ? warp_tot[w - 1] : T(0);
  if (block_total) *block_total = warp_tot[kWarps - 1];
  __syncthreads();
  return warp_excl + x - v;
}

template <class T>
__global__ void scan_reduce_k(const T* __restrict__ in, uint64_t n, T* __restrict__ sums) {
  uint64_t base = (uint64_t)blockIdx.x * kScanTile;
  T acc = 0;
  for (int i = threadIdx.x; i < kScanTile; i += kBlock) {
    uint64_t idx = base + i;
    if (idx < n) acc += in[idx];
  }
  T tot;
  block_exclusive_scan<T>(acc, &tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

template <class T>
__global__ void scan_tile_k(const T* in, T* out, uint64_t n, const T* __restrict__ block_offsets,
                            T* total) {
  __shared__ T s[kScanTile + kScanTile / 32];
  uint64_t base = (uint64_t)blockIdx.x * kScanTile;
  for (int i = threadIdx.x; i < kScanTile; i += kBlock) {
    uint64_t idx = base + i;
    s[pad(i)] = idx < n ? in[idx] : T(0);
  }
  __syncthreads();
  T v[8];
  T tsum = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    v[j] = s[pad(threadIdx.x * 8 + j)];
    tsum += v[j];
  }
  T btot;
  T run = block_exclusive_scan<T>(tsum, &btot);
  if (block_offsets) run += block_offsets[blockIdx.x];
#pragma unroll
  for (int j = 0; j < 8; j++) {
    s[pad(threadIdx.x * 8 + j)] = run;
    run += v[j];
  }
  if (total && threadIdx.x == 0) *total = (block_offsets ? block_offsets[blockIdx.x] : T(0)) + btot;
  __syncthreads();
  for (int i = threadIdx.x; i < kScanTile; i += kBlock) {
    uint64_t idx = base + i;
    if (idx < n) out[idx] = s[pad(i)];
  }
}

template <class T>
void scan_impl(const T* in, T* out, uint64_t n, T* total, cudaStream_t s) {
  if (n == 0) {
    if (total) UG_CUDA(cudaMemsetAsync(total, 0, sizeof(T), s));
    return;
  }
  uint64_t nb = (n + kScanTile - 1) / kScanTile;
  if (nb == 1) {
    scan_tile_k<T><<<1, kBlock, 0, s>>>(in, out, n, nullptr, total);
    UG_LAUNCH_CHECK();
    return;
  }
  Scratch<T> sums(nb, s);
  scan_reduce_k<T><<<(unsigned)nb, kBlock, 0, s>>>(in, n, sums.get());
  UG_LAUNCH_CHECK();
  // The last block's total must include its own offset, so the recursive call
  // produces both the block offsets and the grand total.
  scan_impl<T>(sums.get(), sums.get(), nb, total, s);
  scan_tile_k<T><<<(unsigned)nb, kBlock, 0, s>>>(in, out, n, sums.get(), nullptr);
  UG_LAUNCH_CHECK();
}

// ---------------------------------------------------------------- radix sort
// bad != nullptr: every key >= limit sets *bad (the caller's range check,
// folded into the pass that reads the keys anyway).
__global__ void __launch_bounds__(kBlock) radix_upsweep_k(const uint32_t* __restrict__ keys,
                                                          uint64_t n, int shift, uint32_t mask,
                                                          uint32_t* __restrict__ hist,
                                                          uint32_t num_tiles,
                                                          unsigned* __restrict__ bad,
                                                          uint64_t limit) {
  __shared__ uint32_t cnt[kWarps][256];
  for (int i = threadIdx.x; i < kWarps * 256; i += kBlock) (&cnt[0][0])[i] = 0;
  __syncthreads();
  uint32_t tile = blockIdx.x;
  uint64_t base = (uint64_t)tile * kRadixTile;
  int w = threadIdx.x >> 5;
  uint32_t k[kRadixItems];
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) {
    const uint64_t idx = base + (uint64_t)i * kBlock + threadIdx.x;
    k[i] = idx < n ? __ldg(&keys[idx]) : 0u;
  }
  bool out_of_range = false;
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) {
    const uint64_t idx = base + (uint64_t)i * kBlock + threadIdx.x;
    if (idx < n) {
      atomicAdd(&cnt[w][(k[i] >> shift) & mask], 1u);
      out_of_range |= (uint64_t)k[i] >= limit;
    }
  }
  if (bad && __any_sync(0xffffffffu, out_of_range) && (threadIdx.x & 31) == 0) atomicOr(bad, 1u);
  __syncthreads();
  for (int d = threadIdx.x; d < 256; d += kBlock) {
    uint32_t s = 0;
#pragma unroll
    for (int ww = 0; ww < kWarps; ww++) s += cnt[ww][d];
    hist[(uint64_t)d * num_tiles + tile] = s;
  }
}

__global__ void __launch_bounds__(kBlock) radix_downsweep_k(
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, uint64_t n,
    int shift, uint32_t mask, const uint32_t* __restrict__ hist_scanned, uint32_t num_tiles,
    uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
    const uint32_t* __restrict__ gather_src, uint32_t* __restrict__ gather_out) {
  __shared__ uint32_t wcnt[kWarps][256];
  __shared__ uint32_t gofs[256];
  uint32_t tile = blockIdx.x;
  for (int i = threadIdx.x; i < kWarps * 256; i += kBlock) (&wcnt[0][0])[i] = 0;
  for (int d = threadIdx.x; d < 256; d += kBlock) gofs[d] = hist_scanned[(uint64_t)d * num_tiles + tile];
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  // Warp w owns the contiguous sub-tile [w*512, (w+1)*512); round i covers
  // items w*512 + i*32 + lane, so (round, lane) order is input order.
  const uint64_t wbase = (uint64_t)tile * kRadixTile + (uint64_t)w * (32 * kRadixItems);
  uint32_t k[kRadixItems], v[kRadixItems], dr[kRadixItems];
  // all of the warp's loads in flight before the first ranking step
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) {
    const uint64_t idx = wbase + (uint64_t)i * 32 + lane;
    const bool valid = idx < n;
    k[i] = valid ? __ldg(&keys_in[idx]) : 0u;
    v[i] = valid ? (vals_in ? __ldg(&vals_in[idx]) : (uint32_t)idx) : 0u;
  }
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) {
    uint64_t idx = wbase + (uint64_t)i * 32 + lane;
    bool valid = idx < n;
    uint32_t key = k[i];
    uint32_t d = valid ? ((key >> shift) & mask) : 256u;
    uint32_t peers = __match_any_sync(0xffffffffu, d);
    uint32_t rank_in = __popc(peers & lt);
    uint32_t before = d < 256u ? wcnt[w][d] : 0u;
    __syncwarp();
    if (d < 256u && rank_in == 0) wcnt[w][d] = before + __popc(peers);
    __syncwarp();
    dr[i] = (d << 16) | (before + rank_in);
  }
  __syncthreads();
  // Per digit: each warp's exclusive start, and the tile's digit total.
  static_assert(kBlock == 256, "one thread per digit");
  uint32_t run = 0;
  {
    const int d = threadIdx.x;
#pragma unroll
    for (int ww = 0; ww < kWarps; ww++) {
      uint32_t x = wcnt[ww][d];
      wcnt[ww][d] = run;
      run += x;
    }
  }
  // Tile-local digit starts, so the tile can be ordered in shared memory and
  // written out in coalesced runs (one run per digit).
  __shared__ uint32_t toff[256];
  __shared__ uint32_t sk[kRadixTile];
  __shared__ uint32_t sv[kRadixTile];
  toff[threadIdx.x] = block_exclusive_scan<uint32_t>(run, nullptr);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) {
    uint32_t d = dr[i] >> 16;
    if (d < 256u) {
      uint32_t p = toff[d] + wcnt[w][d] + (dr[i] & 0xffffu);
      sk[p] = k[i];
      sv[p] = v[i];
    }
  }
  __syncthreads();
  const uint64_t tile0 = (uint64_t)tile * kRadixTile;
  const uint32_t tile_n = (uint32_t)(n - tile0 < (uint64_t)kRadixTile ? n - tile0 : kRadixTile);
  for (uint32_t i = threadIdx.x; i < tile_n; i += kBlock) {
    const uint32_t key = sk[i], val = sv[i];
    const uint32_t d = (key >> shift) & mask;
    const uint32_t dest = gofs[d] + (i - toff[d]);
    keys_out[dest] = key;
    vals_out[dest] = val;
    if (gather_src) gather_out[dest] = gather_src[val];
  }
}

// A word from global to shared memory without a register (any 4-byte
// alignment); waited for with tile_wait().
__device__ __forceinline__ void tile_copy(uint32_t* dst, const uint32_t* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void tile_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The downsweep of triples: key, value (vals_in == nullptr: the input
// position) and a third word.  A pass is bound by shared memory (ranking and
// staging, some 40 accesses of a warp per 32 items) and by the loads'
// latency, not by the 24 bytes an item moves.  So the values and the third
// words cross to shared memory while the keys are ranked, and only the keys'
// ranks are held in registers.
struct CarrySmem {
  uint32_t stage[kRadixTile];
  uint32_t vals[kRadixTile];
  uint32_t other[kRadixTile];
  uint32_t gofs[256];  // global start of the digit, less its start in the tile
  uint16_t wcnt[kDownWarps][256];
  uint32_t warp_sum[8];
};

__global__ void __launch_bounds__(kDownBlock, 3) radix_carry_k(
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
    const uint32_t* __restrict__ other_in, uint64_t n, int shift, uint32_t mask,
    const uint32_t* __restrict__ hist_scanned, uint32_t num_tiles, uint32_t* __restrict__ keys_out,
    uint32_t* __restrict__ vals_out, uint32_t* __restrict__ other_out) {
  extern __shared__ __align__(16) unsigned char carry_sm[];
  CarrySmem& sm = *reinterpret_cast<CarrySmem*>(carry_sm);
  const uint32_t tile = blockIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  // Warp w owns the contiguous sub-tile [w*256, (w+1)*256); round i covers
  // items w*256 + i*32 + lane, so (round, lane) order is input order.
  const uint64_t tile0 = (uint64_t)tile * kRadixTile;
  const uint32_t item0 = w * (32 * kDownItems) + lane;
  const uint32_t tile_n = (uint32_t)(n - tile0 < (uint64_t)kRadixTile ? n - tile0 : kRadixTile);
  uint32_t k[kDownItems], p[kDownItems];
#pragma unroll
  for (int i = 0; i < kDownItems; i++) {
    const uint32_t it = item0 + i * 32;
    k[i] = it < tile_n ? __ldg(&keys_in[tile0 + it]) : 0u;
  }
#pragma unroll
  for (int i = 0; i < kDownItems; i++) {
    const uint32_t it = item0 + i * 32;
    if (it < tile_n) {
      if (vals_in) tile_copy(&sm.vals[it], &vals_in[tile0 + it]);
      tile_copy(&sm.other[it], &other_in[tile0 + it]);
    }
  }
  const uint32_t digit = threadIdx.x;  // of the first 256 threads
  const uint32_t g = digit < 256 ? hist_scanned[(uint64_t)digit * num_tiles + tile] : 0u;
  for (int i = lane; i < 256; i += 32) sm.wcnt[w][i] = 0;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < kDownItems; i++) {
    const uint32_t d = (k[i] >> shift) & mask;
    const bool valid = item0 + i * 32 < tile_n;
    const uint32_t peers = __match_any_sync(0xffffffffu, valid ? d : 256u);
    const uint32_t before = valid ? sm.wcnt[w][d] : 0u;
    __syncwarp();
    const uint32_t rank = __popc(peers & lt);
    if (valid && rank == 0) sm.wcnt[w][d] = (uint16_t)(before + __popc(peers));
    __syncwarp();
    p[i] = before + rank;
  }
  __syncthreads();
  // Per digit: the tile's total, and each warp's start in the ordered tile.
  uint32_t sum = 0, incl = 0;
  if (digit < 256) {
#pragma unroll
    for (int ww = 0; ww < kDownWarps; ww++) sum += sm.wcnt[ww][digit];
    incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    if (lane == 31) sm.warp_sum[w] = incl;
  }
  __syncthreads();
  if (digit < 256) {
    uint32_t run = incl - sum;
    for (int ww = 0; ww < w; ww++) run += sm.warp_sum[ww];
    sm.gofs[digit] = g - run;
#pragma unroll
    for (int ww = 0; ww < kDownWarps; ww++) {
      const uint32_t x = sm.wcnt[ww][digit];
      sm.wcnt[ww][digit] = (uint16_t)run;
      run += x;
    }
  }
  __syncthreads();
  // the tile in digit order, so that it is written in one run per digit
#pragma unroll
  for (int i = 0; i < kDownItems; i++) {
    p[i] += sm.wcnt[w][(k[i] >> shift) & mask];
    if (item0 + i * 32 < tile_n) sm.stage[p[i]] = k[i];
  }
  __syncthreads();
  uint32_t dest[kDownItems];
#pragma unroll
  for (int j = 0; j < kDownItems; j++) {
    const uint32_t i = j * kDownBlock + threadIdx.x;
    if (i < tile_n) {
      const uint32_t key = sm.stage[i];
      dest[j] = sm.gofs[(key >> shift) & mask] + i;
      keys_out[dest[j]] = key;
    }
  }
  tile_wait();
  __syncthreads();  // every copy has landed, and the keys have been read
#pragma unroll
  for (int i = 0; i < kDownItems; i++) {
    const uint32_t it = item0 + i * 32;
    if (it < tile_n) sm.stage[p[i]] = vals_in ? sm.vals[it] : (uint32_t)(tile0 + it);
  }
  __syncthreads();  // the values have been read from sm.vals, too
#pragma unroll
  for (int j = 0; j < kDownItems; j++) {
    const uint32_t i = j * kDownBlock + threadIdx.x;
    if (i < tile_n) vals_out[dest[j]] = sm.stage[i];
  }
#pragma unroll
  for (int i = 0; i < kDownItems; i++) {
    const uint32_t it = item0 + i * 32;
    if (it < tile_n) sm.vals[p[i]] = sm.other[it];
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kDownItems; j++) {
    const uint32_t i = j * kDownBlock + threadIdx.x;
    if (i < tile_n) other_out[dest[j]] = sm.vals[i];
  }
}

__global__ void offsets_k(const uint32_t* __restrict__ keys, uint64_t m, uint64_t n,
                          uint32_t* __restrict__ off) {
  for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u <= n;
       u += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t lo = 0, hi = m;
    while (lo < hi) {
      uint64_t mid = (lo + hi) >> 1;
      if ((uint64_t)keys[mid] < u)
        lo = mid + 1;
      else
        hi = mid;
    }
    off[u] = (uint32_t)lo;
  }
}

// radix_carry_k's shared memory is above the default limit: raised once per
// device.
void carry_allow_smem() {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  UG_CUDA(cudaGetDevice(&dev));
  UG_CHECK(dev >= 0 && dev < 64, URSA_GPU_EINVAL, "device index out of range");
  std::lock_guard<std::mutex> g(mu);
  if (done[dev]) return;
  UG_CUDA(cudaFuncSetAttribute(radix_carry_k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sizeof(CarrySmem)));
  done[dev] = true;
}

}  // namespace

void exclusive_scan_u32(const uint32_t* in, uint32_t* out, uint64_t n, uint32_t* total,
                        cudaStream_t s) {
  scan_impl<uint32_t>(in, out, n, total, s);
}
void exclusive_scan_u64(const uint64_t* in, uint64_t* out, uint64_t n, uint64_t* total,
                        cudaStream_t s) {
  scan_impl<uint64_t>(in, out, n, total, s);
}

void radix_sort_pairs(const uint32_t* keys_in, const uint32_t* vals_in, uint64_t n, int key_bits,
                      uint32_t* keys_out, uint32_t* vals_out, const uint32_t* gather_src,
                      uint32_t* gather_out, cudaStream_t s, cudaEvent_t gather_ready,
                      unsigned* bad, uint64_t limit) {
  UG_CHECK(n < (1ull << 32), URSA_GPU_EINVAL, "radix sort: more than 2^32-1 items");
  if (n == 0) return;
  int passes = key_bits <= 8 ? 1 : (key_bits + 7) / 8;
  uint32_t num_tiles = (uint32_t)((n + kRadixTile - 1) / kRadixTile);
  Scratch<uint32_t> hist((size_t)256 * num_tiles, s);
  // a column that still arrives is gathered in the last pass
  const bool carry = gather_src && !gather_ready && n >= kCarryMin && n <= kCarryMax;
  if (carry) carry_allow_smem();
  Scratch<uint32_t> kb[2], vb[2], ob[2];
  for (int i = 0; i < 2 && i < passes - 1; i++) {
    kb[i].alloc(n, s);
    vb[i].alloc(n, s);
    if (carry) ob[i].alloc(n, s);
  }
  const uint32_t* kin = keys_in;
  const uint32_t* vin = vals_in;
  const uint32_t* oin = gather_src;
  for (int p = 0; p < passes; p++) {
    int shift = 8 * p;
    int bits = key_bits - shift;
    if (bits > 8) bits = 8;
    if (bits < 0) bits = 0;
    uint32_t mask = bits == 0 ? 0u : ((1u << bits) - 1u);
    bool last = p == passes - 1;
    uint32_t* kout = last ? keys_out : kb[p & 1].get();
    uint32_t* vout = last ? vals_out : vb[p & 1].get();
    radix_upsweep_k<<<num_tiles, kBlock, 0, s>>>(kin, n, shift, mask, hist.get(), num_tiles,
                                                 p == 0 ? bad : nullptr, limit);
    UG_LAUNCH_CHECK();
    exclusive_scan_u32(hist.get(), hist.get(), (uint64_t)256 * num_tiles, nullptr, s);
    if (last && gather_ready) UG_CUDA(cudaStreamWaitEvent(s, gather_ready, 0));
    if (carry) {
      uint32_t* oout = last ? gather_out : ob[p & 1].get();
      radix_carry_k<<<num_tiles, kDownBlock, sizeof(CarrySmem), s>>>(
          kin, vin, oin, n, shift, mask, hist.get(), num_tiles, kout, vout, oout);
      oin = oout;
    } else {
      radix_downsweep_k<<<num_tiles, kBlock, 0, s>>>(kin, vin, n, shift, mask, hist.get(), num_tiles,
                                                     kout, vout, last ? gather_src : nullptr,
                                                     gather_out);
    }
    UG_LAUNCH_CHECK();
    kin = kout;
    vin = vout;
  }
}

void offsets_from_sorted(const uint32_t* sorted_keys, uint64_t m, uint64_t n, uint32_t* offsets,
                         cudaStream_t s) {
  offsets_k<<<grid_for(n + 1), kBlock, 0, s>>>(sorted_keys, m, n, offsets);
  UG_LAUNCH_CHECK();
}

namespace {
__global__ void any_negative_k(const double* __restrict__ w, uint64_t m, unsigned* __restrict__ bad) {
  bool neg = false;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (uint64_t)gridDim.x * blockDim.x)
    neg |= __ldg(&w[i]) < 0.0;
  if (__any_sync(0xffffffffu, neg) && (threadIdx.x & 31) == 0) *bad = 1u;
}
}  // namespace

void check_sssp_weights_device(const double* d_w, uint64_t m, cudaStream_t s) {
  if (m == 0) return;
  Scratch<unsigned> bad(1, s);
  UG_CUDA(cudaMemsetAsync(bad.get(), 0, 4, s));
  any_negative_k<<<grid_for(m, kBlock, 148u * 16u), kBlock, 0, s>>>(d_w, m, bad.get());
  UG_LAUNCH_CHECK();
  unsigned h = 0;
  UG_CUDA(cudaMemcpyAsync(&h, bad.get(), 4, cudaMemcpyDeviceToHost, s));
  UG_CUDA(cudaStreamSynchronize(s));
  UG_CHECK(h == 0, URSA_GPU_EINVAL, "weights must be non-negative");
}

}  // namespace ug
