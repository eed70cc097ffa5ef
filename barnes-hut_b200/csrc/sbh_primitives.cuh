// Device-wide primitives written for this library: exclusive scans (u32,
// double and small double vectors) and a stable LSD radix sort of u32/u64
// keys with u32 payloads. All of them are deterministic (no floating-point
// atomics; fixed reduction trees), allocate nothing (temporaries come from
// the caller's workspace) and launch a fixed number of kernels, so they can
// be captured in CUDA graphs.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

namespace sbh {

constexpr int kScanThreads = 256;

// Items per thread: 8 for 4-8 byte elements, fewer for the FP64 moment
// vectors so a tile stays in registers without spilling.
template <typename T>
struct ScanCfg {
  static constexpr int kItems = sizeof(T) <= 8 ? 8 : (sizeof(T) <= 32 ? 4 : 2);
  static constexpr int kTile = kScanThreads * kItems;
};

// K doubles summed component-wise.
template <int K>
struct DVec {
  double v[K];
  __host__ __device__ DVec() {
    for (int i = 0; i < K; i++) v[i] = 0.0;
  }
  __host__ __device__ DVec operator+(const DVec& o) const {
    DVec r;
    for (int i = 0; i < K; i++) r.v[i] = v[i] + o.v[i];
    return r;
  }
};

__device__ __forceinline__ uint32_t shfl_up_t(uint32_t x, int d) {
  return __shfl_up_sync(0xffffffffu, x, d);
}
__device__ __forceinline__ uint64_t shfl_up_t(uint64_t x, int d) {
  return __shfl_up_sync(0xffffffffu, x, d);
}
__device__ __forceinline__ double shfl_up_t(double x, int d) {
  return __shfl_up_sync(0xffffffffu, x, d);
}
template <int K>
__device__ __forceinline__ DVec<K> shfl_up_t(const DVec<K>& x, int d) {
  DVec<K> r;
  for (int i = 0; i < K; i++) r.v[i] = __shfl_up_sync(0xffffffffu, x.v[i], d);
  return r;
}

template <typename T>
__device__ __forceinline__ T zero_t() {
  return T();
}
template <>
__device__ __forceinline__ uint32_t zero_t<uint32_t>() {
  return 0u;
}
template <>
__device__ __forceinline__ uint64_t zero_t<uint64_t>() {
  return 0ull;
}
template <>
__device__ __forceinline__ double zero_t<double>() {
  return 0.0;
}

// Inclusive warp scan.
template <typename T>
__device__ __forceinline__ T warp_inclusive(T x) {
  int lane = threadIdx.x & 31;
  for (int d = 1; d < 32; d <<= 1) {
    T y = shfl_up_t(x, d);
    if (lane >= d) x = x + y;
  }
  return x;
}

// Exclusive block scan of one value per thread; returns the exclusive prefix
// and writes the block total to *total. blockDim.x == kScanThreads.
template <typename T>
__device__ T block_exclusive(T x, T* total) {
  __shared__ T warp_tot[kScanThreads / 32];
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T inc = warp_inclusive(x);
  if (lane == 31) warp_tot[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    T w = lane < kScanThreads / 32 ? warp_tot[lane] : zero_t<T>();
    T wi = warp_inclusive(w);
    if (lane < kScanThreads / 32) warp_tot[lane] = wi;
  }
  __syncthreads();
  T base = warp == 0 ? zero_t<T>() : warp_tot[warp - 1];
  T t = warp_tot[kScanThreads / 32 - 1];
  __syncthreads();
  if (total) *total = t;
  // exclusive = inclusive - x, computed as base + (inc - x) without subtraction:
  T prev = shfl_up_t(inc, 1);
  if (lane == 0) prev = zero_t<T>();
  return base + prev;
}

// Phase 1: per-tile totals.
template <typename T, typename Load>
__global__ void __launch_bounds__(kScanThreads) scan_tile_totals(Load load, int64_t n, T* tile_tot) {
  constexpr int kItems = ScanCfg<T>::kItems;
  int64_t tile0 = static_cast<int64_t>(blockIdx.x) * ScanCfg<T>::kTile;
  T acc = zero_t<T>();
  for (int k = 0; k < kItems; k++) {
    int64_t i = tile0 + static_cast<int64_t>(threadIdx.x) * kItems + k;
    if (i < n) acc = acc + load(i);
  }
  T tot;
  block_exclusive(acc, &tot);
  if (threadIdx.x == 0) tile_tot[blockIdx.x] = tot;
}

// Phase 2: exclusive scan of the tile totals in one block (any count).
template <typename T>
__global__ void __launch_bounds__(kScanThreads) scan_tile_offsets(T* tile_tot, int64_t ntiles) {
  __shared__ T carry_s;
  if (threadIdx.x == 0) carry_s = zero_t<T>();
  __syncthreads();
  for (int64_t c0 = 0; c0 < ntiles; c0 += kScanThreads) {
    int64_t i = c0 + threadIdx.x;
    T x = i < ntiles ? tile_tot[i] : zero_t<T>();
    T tot;
    T ex = block_exclusive(x, &tot);
    T carry = carry_s;
    if (i < ntiles) tile_tot[i] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry_s = carry + tot;
    __syncthreads();
  }
}

// Phase 3: exclusive scan within tiles plus the tile offset; out[n] = total
// when write_total.
template <typename T, typename Load>
__global__ void __launch_bounds__(kScanThreads) scan_tile_apply(Load load, int64_t n,
                                                               const T* tile_off, T* out,
                                                               int write_total, T* total_out) {
  constexpr int kItems = ScanCfg<T>::kItems;
  int64_t tile0 = static_cast<int64_t>(blockIdx.x) * ScanCfg<T>::kTile;
  T items[kItems];
  T acc = zero_t<T>();
  for (int k = 0; k < kItems; k++) {
    int64_t i = tile0 + static_cast<int64_t>(threadIdx.x) * kItems + k;
    items[k] = i < n ? load(i) : zero_t<T>();
    acc = acc + items[k];
  }
  T tot;
  T run = tile_off[blockIdx.x] + block_exclusive(acc, &tot);
  for (int k = 0; k < kItems; k++) {
    int64_t i = tile0 + static_cast<int64_t>(threadIdx.x) * kItems + k;
    if (i < n) out[i] = run;
    run = run + items[k];
  }
  if (write_total && blockIdx.x == gridDim.x - 1 && threadIdx.x == kScanThreads - 1) {
    T t = tile_off[blockIdx.x] + tot;
    if (total_out) *total_out = t;
    out[n] = t;
  }
}

// A few tiles in one block and one launch, the running total carried along: for
// the moment vectors two, a tile of which takes about 8 us there, as long as the
// two launches saved (8 tiles of 14 doubles: force + adjoint of 4,000 particles 179
// us, 138 by three launches; build 138 and 115), for words eight.
template <typename T>
constexpr int64_t kScanFewTiles = sizeof(T) <= 8 ? 8 : 2;
template <typename T, typename Load>
__global__ void __launch_bounds__(kScanThreads) scan_few_tiles(Load load, int64_t n, T* out, int write_total) {
  constexpr int kItems = ScanCfg<T>::kItems;
  T carry = zero_t<T>();
  for (int64_t tile0 = 0; tile0 < n || tile0 == 0; tile0 += ScanCfg<T>::kTile) {
    T items[kItems];
    T acc = zero_t<T>();
    for (int k = 0; k < kItems; k++) {
      const int64_t i = tile0 + static_cast<int64_t>(threadIdx.x) * kItems + k;
      items[k] = i < n ? load(i) : zero_t<T>();
      acc = acc + items[k];
    }
    T tot;
    T run = carry + block_exclusive(acc, &tot);
    for (int k = 0; k < kItems; k++) {
      const int64_t i = tile0 + static_cast<int64_t>(threadIdx.x) * kItems + k;
      if (i < n) out[i] = run;
      run = run + items[k];
    }
    carry = carry + tot;
  }
  if (write_total && threadIdx.x == 0) out[n] = carry;
}

// Number of tiles (= temporaries of type T) of a scan over n elements of T.
template <typename T = uint32_t>
inline int64_t scan_tiles(int64_t n) {
  return n <= 0 ? 1 : (n + ScanCfg<T>::kTile - 1) / ScanCfg<T>::kTile;
}

// Exclusive scan of load(0..n-1) into out[0..n-1] (and out[n] = total when
// write_total). tmp: scan_tiles<T>(n) elements of T.
template <typename T, typename Load>
cudaError_t exclusive_scan(cudaStream_t s, Load load, int64_t n, T* out, T* tmp,
                           bool write_total) {
  int64_t nt = scan_tiles<T>(n);
  if (nt <= kScanFewTiles<T>) {
    scan_few_tiles<T, Load><<<1, kScanThreads, 0, s>>>(load, n, out, write_total ? 1 : 0);
    return cudaGetLastError();
  }
  scan_tile_totals<T, Load><<<static_cast<unsigned>(nt), kScanThreads, 0, s>>>(load, n, tmp);
  scan_tile_offsets<T><<<1, kScanThreads, 0, s>>>(tmp, nt);
  scan_tile_apply<T, Load><<<static_cast<unsigned>(nt), kScanThreads, 0, s>>>(
      load, n, tmp, out, write_total ? 1 : 0, static_cast<T*>(nullptr));
  return cudaGetLastError();
}

template <typename T>
struct ArrayLoad {
  const T* p;
  __device__ T operator()(int64_t i) const { return p[i]; }
};

// --------------------------------------------------------------------------
// Stable LSD radix sort, 8-bit digits.
// --------------------------------------------------------------------------
constexpr int kSortThreads = 256;
constexpr int kSortRounds = 8;
constexpr int kSortTile = kSortThreads * kSortRounds;  // 2048 keys per block

// The lanes whose 8-bit digit equals this lane's, among the valid ones: eight
// ballots. (__match_any_sync runs once per distinct value, some thirty times for
// random digits: radix_scatter's rounds took about 2 us each with it.)
__device__ __forceinline__ uint32_t match_digit(uint32_t d, bool valid) {
  uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
  for (int b = 0; b < 8; b++) {
    const bool one = (d >> b) & 1u;
    const uint32_t v = __ballot_sync(0xffffffffu, one);
    peers &= one ? v : ~v;
  }
  return peers;
}

template <typename K>
__global__ void __launch_bounds__(kSortThreads) radix_count(const K* keys, int64_t n, int shift,
                                                            uint32_t* hist, int64_t nblocks) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  int64_t t0 = static_cast<int64_t>(blockIdx.x) * kSortTile;
  for (int r = 0; r < kSortRounds; r++) {
    int64_t i = t0 + r * kSortThreads + threadIdx.x;
    if (i < n) atomicAdd(&h[static_cast<uint32_t>(keys[i] >> shift) & 255u], 1u);
  }
  __syncthreads();
  hist[static_cast<int64_t>(threadIdx.x) * nblocks + blockIdx.x] = h[threadIdx.x];
}

// Each warp ranks its contiguous run of 256 keys, 32 at a time, against its own
// digit counters without waiting for the others; one scan over the warps'
// counters then places them. (Ranking 256 keys per round across the block took
// five barriers a round, about 40 per tile.)
template <typename K>
__global__ void __launch_bounds__(kSortThreads) radix_scatter(const K* keys_in, const uint32_t* vals_in,
                                                              K* keys_out, uint32_t* vals_out,
                                                              int64_t n, int shift,
                                                              const uint32_t* hist_off,
                                                              int64_t nblocks) {
  constexpr int kWarps = kSortThreads / 32;
  __shared__ uint32_t cnt[kWarps][256];
  __shared__ uint32_t to[256];  // digit's first position in the output, less its first in the tile
  __shared__ K skey[kSortTile];
  __shared__ uint32_t sval[kSortTile];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t goff = hist_off[static_cast<int64_t>(threadIdx.x) * nblocks + blockIdx.x];
  for (int d = lane; d < 256; d += 32) cnt[warp][d] = 0;
  __syncwarp();
  const int64_t first = static_cast<int64_t>(blockIdx.x) * kSortTile + warp * (32 * kSortRounds) + lane;
  const uint32_t lt = (1u << lane) - 1u;
  K key[kSortRounds];
  uint32_t val[kSortRounds], rank[kSortRounds];
#pragma unroll
  for (int r = 0; r < kSortRounds; r++) {
    const int64_t i = first + 32 * r;
    key[r] = i < n ? keys_in[i] : K(0);
    val[r] = i < n ? (vals_in ? vals_in[i] : static_cast<uint32_t>(i)) : 0u;
  }
#pragma unroll
  for (int r = 0; r < kSortRounds; r++) {
    const bool valid = first + 32 * r < n;
    const uint32_t d = static_cast<uint32_t>(key[r] >> shift) & 255u;
    const uint32_t peers = match_digit(d, valid);
    const uint32_t before = cnt[warp][d];
    rank[r] = before + __popc(peers & lt);
    __syncwarp();
    if (valid && (peers & lt) == 0) cnt[warp][d] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  uint32_t sum = 0;
#pragma unroll
  for (int w = 0; w < kWarps; w++) sum += cnt[w][threadIdx.x];
  uint32_t at = block_exclusive(sum, static_cast<uint32_t*>(nullptr));  // thread d: digit d's place in the tile
  to[threadIdx.x] = goff - at;
#pragma unroll
  for (int w = 0; w < kWarps; w++) {
    const uint32_t c = cnt[w][threadIdx.x];
    cnt[w][threadIdx.x] = at;
    at += c;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortRounds; r++) {
    if (first + 32 * r < n) {
      const uint32_t p = cnt[warp][static_cast<uint32_t>(key[r] >> shift) & 255u] + rank[r];
      skey[p] = key[r];
      sval[p] = val[r];
    }
  }
  __syncthreads();
  // neighbours in the tile's order mostly go to neighbouring places
  const int64_t left = n - static_cast<int64_t>(blockIdx.x) * kSortTile;
  const int m = left < kSortTile ? static_cast<int>(left) : kSortTile;
#pragma unroll
  for (int r = 0; r < kSortRounds; r++) {
    const int i = r * kSortThreads + static_cast<int>(threadIdx.x);
    if (i < m) {
      const K k = skey[i];
      const uint32_t dst = to[static_cast<uint32_t>(k >> shift) & 255u] + static_cast<uint32_t>(i);
      keys_out[dst] = k;
      vals_out[dst] = sval[i];
    }
  }
}

// Small sorts run in one block: the keys and their input indices stay in
// registers and shared memory through all the passes, so a sort is one launch
// where the device-wide passes take five each (10,000 63-bit keys: 40 launches,
// about 200 us of kernels of 3 to 16 us, bound by launches and by the few blocks'
// barriers). Each warp holds a contiguous run of the keys, ranks it 32 at a
// time with ballots against its own digit counters, and one scan over the
// warps' counters turns ranks into positions; the order of equal digits is kept
// throughout.
constexpr int kSmallSortThreads = 1024;
constexpr int kSmallSortItems = 16;
constexpr int kSmallSortRun = 8;
constexpr int64_t kSmallSortMax = kSmallSortThreads * kSmallSortItems;  // payloads are 16-bit there

template <typename K>
struct SmallSortShared {
  K key[kSmallSortMax];
  uint16_t val[kSmallSortMax];
  uint16_t cnt[32][256];
  uint32_t warp_tot[8];
};

template <typename K>
__global__ void __launch_bounds__(kSmallSortThreads, 1)
    radix_small(K* __restrict__ keys, uint32_t* __restrict__ vals, int n, int bits, int vals_given) {
  extern __shared__ uint4 small_sort_smem[];
  SmallSortShared<K>& S = *reinterpret_cast<SmallSortShared<K>*>(small_sort_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (n + 1023) / 1024;  // rounds of 32 keys per warp
  const int first = warp * 32 * per;
  const uint32_t lt = (1u << lane) - 1u;
  K key[kSmallSortItems];
  uint32_t val[kSmallSortItems];  // input index, and above it the rank within the pass
  // Keys of more than 32 bits are first sorted by their top 32 alone, half the
  // passes. Few keys of so small a set agree in those, and their runs are then
  // ordered in place; a run of more than kSmallSortRun keys (coincident points)
  // sends the sort back to all bits.
  for (int low = sizeof(K) > 4 && bits > 32 ? bits - 32 : 0;; low = 0) {
#pragma unroll
    for (int r = 0; r < kSmallSortItems; r++) {
      const int i = first + 32 * r + lane;
      key[r] = r < per && i < n ? keys[i] : K(0);
      val[r] = static_cast<uint32_t>(i) & 0xFFFFu;
    }
    for (int shift = low; shift < bits; shift += 8) {
      for (int d = lane; d < 128; d += 32) reinterpret_cast<uint32_t*>(S.cnt[warp])[d] = 0u;
      __syncwarp();
#pragma unroll
      for (int r = 0; r < kSmallSortItems; r++) {
        if (r < per) {  // uniform
          const bool in = first + 32 * r + lane < n;
          const uint32_t d = static_cast<uint32_t>(key[r] >> shift) & 255u;
          const uint32_t peers = match_digit(d, in);
          const uint32_t before = in ? S.cnt[warp][d] : 0u;
          val[r] |= (before + __popc(peers & lt)) << 16;
          __syncwarp();
          if (in && (peers & lt) == 0) S.cnt[warp][d] = static_cast<uint16_t>(before + __popc(peers));
          __syncwarp();
        }
      }
      __syncthreads();
      // thread d < 256: digit d's count per warp -> first position per warp
      uint32_t run = 0, inc = 0;
      if (threadIdx.x < 256) {
        for (int w = 0; w < 32; w++) run += S.cnt[w][threadIdx.x];
        inc = run;
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += v;
        }
        if (lane == 31) S.warp_tot[warp] = inc;
      }
      __syncthreads();
      if (threadIdx.x < 256) {
        uint32_t at = inc - run;
        for (int w = 0; w < warp; w++) at += S.warp_tot[w];
        for (int w = 0; w < 32; w++) {
          const uint32_t c = S.cnt[w][threadIdx.x];
          S.cnt[w][threadIdx.x] = static_cast<uint16_t>(at);
          at += c;
        }
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < kSmallSortItems; r++) {
        if (r < per && first + 32 * r + lane < n) {
          const uint32_t d = static_cast<uint32_t>(key[r] >> shift) & 255u;
          const int p = static_cast<int>(S.cnt[warp][d] + (val[r] >> 16));
          S.key[p] = key[r];
          S.val[p] = static_cast<uint16_t>(val[r]);
        }
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < kSmallSortItems; r++) {
        const int i = first + 32 * r + lane;
        if (r < per && i < n) {
          key[r] = S.key[i];
          val[r] = S.val[i];
        }
      }
      __syncthreads();
    }
    if (low == 0) break;
    bool again = false;
    for (int i = static_cast<int>(threadIdx.x); i < n; i += kSmallSortThreads) {
      const K top = S.key[i] >> low;
      if (i > 0 && S.key[i - 1] >> low == top) continue;  // not the head of a run
      int end = i + 1;
      while (end < n && end - i <= kSmallSortRun && S.key[end] >> low == top) end++;
      if (end - i > kSmallSortRun) again = true;
    }
    if (__syncthreads_or(again)) continue;
    for (int i = static_cast<int>(threadIdx.x); i < n; i += kSmallSortThreads) {
      const K top = S.key[i] >> low;
      if ((i > 0 && S.key[i - 1] >> low == top) || i + 1 >= n || S.key[i + 1] >> low != top) continue;
      for (int e = i + 1; e < n && S.key[e] >> low == top; e++) {  // stable insertion
        const K k = S.key[e];
        const uint16_t v = S.val[e];
        int at = e;
        for (; at > i && S.key[at - 1] > k; at--) {
          S.key[at] = S.key[at - 1];
          S.val[at] = S.val[at - 1];
        }
        S.key[at] = k;
        S.val[at] = v;
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSmallSortItems; r++) {
      const int i = first + 32 * r + lane;
      if (r < per && i < n) {
        key[r] = S.key[i];
        val[r] = S.val[i];
      }
    }
    break;
  }
  uint32_t out[kSmallSortItems];
#pragma unroll
  for (int r = 0; r < kSmallSortItems; r++) {
    const int i = first + 32 * r + lane;
    if (r < per && i < n) out[r] = vals_given ? vals[val[r] & 0xFFFFu] : val[r] & 0xFFFFu;
  }
  __syncthreads();  // the given payloads are read before any is overwritten
#pragma unroll
  for (int r = 0; r < kSmallSortItems; r++) {
    const int i = first + 32 * r + lane;
    if (r < per && i < n) {
      keys[i] = key[r];
      vals[i] = out[r];
    }
  }
}

template <typename K>
cudaError_t radix_sort_small(cudaStream_t s, K* keys, uint32_t* vals, int64_t n, int bits, bool vals_given) {
  static std::atomic<uint64_t> ready[2];  // devices whose copy of the kernel may take this much shared memory
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = 1ull << (dev & 63);
  std::atomic<uint64_t>& r = ready[(dev >> 6) & 1];
  if (!(r.load() & bit)) {
    e = cudaFuncSetAttribute(radix_small<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(sizeof(SmallSortShared<K>)));
    if (e != cudaSuccess) return e;
    r.fetch_or(bit);
  }
  radix_small<K><<<1, kSmallSortThreads, sizeof(SmallSortShared<K>), s>>>(keys, vals, static_cast<int>(n), bits,
                                                                         vals_given ? 1 : 0);
  return cudaGetLastError();
}

inline int64_t radix_blocks(int64_t n) { return n <= 0 ? 1 : (n + kSortTile - 1) / kSortTile; }

// Workspace elements (u32) for radix_sort's histogram + scan temporaries.
inline int64_t radix_hist_elems(int64_t n) { return 256 * radix_blocks(n); }

// Sorts (keys, vals) stably by the low `bits` bits of the key. vals_in may be
// null (payload = input index). Ping-pongs between (k0, v0) and (k1, v1);
// returns 0 if the sorted data ends in (k0, v0), 1 if in (k1, v1). The input
// must be in k0 (and v0 when given).
template <typename K>
cudaError_t radix_sort(cudaStream_t s, K* k0, uint32_t* v0, K* k1, uint32_t* v1, int64_t n,
                       int bits, bool vals_given, uint32_t* hist, uint32_t* scan_tmp,
                       int* which) {
  int64_t nb = radix_blocks(n);
  int cur = 0;
  bool first = true;
  if (n <= 0) {
    *which = 0;
    return cudaSuccess;
  }
  if (n <= kSmallSortMax && bits > 0) {
    *which = 0;
    return radix_sort_small<K>(s, k0, v0, n, bits, vals_given);
  }
  for (int shift = 0; shift < bits; shift += 8) {
    K* kin = cur == 0 ? k0 : k1;
    uint32_t* vin = cur == 0 ? v0 : v1;
    K* kout = cur == 0 ? k1 : k0;
    uint32_t* vout = cur == 0 ? v1 : v0;
    radix_count<K><<<static_cast<unsigned>(nb), kSortThreads, 0, s>>>(kin, n, shift, hist, nb);
    cudaError_t e = exclusive_scan<uint32_t>(s, ArrayLoad<uint32_t>{hist}, 256 * nb, hist,
                                             scan_tmp, false);
    if (e != cudaSuccess) return e;
    radix_scatter<K><<<static_cast<unsigned>(nb), kSortThreads, 0, s>>>(
        kin, (first && !vals_given) ? nullptr : vin, kout, vout, n, shift, hist, nb);
    first = false;
    cur ^= 1;
  }
  if (first) {
    // zero passes requested: payload = identity
    *which = 0;
    return cudaGetLastError();
  }
  *which = cur;
  return cudaGetLastError();
}

}  // namespace sbh
