// Device-wide exclusive scan and stable LSD radix sort (uint32 keys, int32
// values), written for the cell-list build of the neighbour search.
// Both are deterministic: equal keys keep their input order, so the particle
// order -- and with it every summation order downstream -- is reproducible.
#include "sort.cuh"

#include <algorithm>

namespace sph {

namespace {
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

template <typename T>
__device__ __forceinline__ T blockExclusiveScan(T v, T* smem, T* total) {
  // Warp-level inclusive scan then a scan over warp totals.
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    T w = lane < nw ? smem[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < nw) smem[lane] = w;   // inclusive warp totals
  }
  __syncthreads();
  const T warpPrefix = warp > 0 ? smem[warp - 1] : T(0);
  const T result = warpPrefix + x - v;
  if (total) *total = smem[(blockDim.x >> 5) - 1];
  __syncthreads();
  return result;
}

template <typename Tin>
__global__ void scanReduceKernel(const Tin* __restrict__ in, long n, long long* __restrict__ blockSums) {
  __shared__ long long smem[32];
  const long base = (long)blockIdx.x * kScanTile;
  long long s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const long idx = base + (long)threadIdx.x * kScanItems + k;
    if (idx < n) s += (long long)in[idx];
  }
  long long tot;
  blockExclusiveScan<long long>(s, smem, &tot);
  if (threadIdx.x == 0) blockSums[blockIdx.x] = tot;
}

__global__ void scanBlockSumsKernel(long long* __restrict__ sums, int nb, long long* __restrict__ grandTotal) {
  __shared__ long long smem[32];
  const int per = (nb + blockDim.x - 1) / blockDim.x;
  const int beg = threadIdx.x * per;
  long long local = 0;
  for (int k = 0; k < per; ++k) if (beg + k < nb) local += sums[beg + k];
  long long tot;
  long long run = blockExclusiveScan<long long>(local, smem, &tot);
  for (int k = 0; k < per; ++k) {
    if (beg + k < nb) { const long long v = sums[beg + k]; sums[beg + k] = run; run += v; }
  }
  if (threadIdx.x == 0 && grandTotal) *grandTotal = tot;
}

template <typename Tin>
__global__ void scanDownsweepKernel(const Tin* __restrict__ in, long n, const long long* __restrict__ blockSums,
                                    long long* __restrict__ out) {
  __shared__ long long smem[32];
  const long base = (long)blockIdx.x * kScanTile;
  long long vals[kScanItems];
  long long s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const long idx = base + (long)threadIdx.x * kScanItems + k;
    vals[k] = idx < n ? (long long)in[idx] : 0;
    s += vals[k];
  }
  long long run = blockExclusiveScan<long long>(s, smem, nullptr) + blockSums[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const long idx = base + (long)threadIdx.x * kScanItems + k;
    if (idx < n) out[idx] = run;
    run += vals[k];
  }
}
}  // namespace

size_t scanWorkspaceBytes(long n) {
  const long nb = (n + kScanTile - 1) / kScanTile;
  return (size_t)(nb + 2) * sizeof(long long);
}

template <typename Tin>
void scanExclusive(const Tin* in, long long* out, long n, void* workspace, long long* dTotal, cudaStream_t s,
                   LaunchCounter* lc) {
  const long nb = (n + kScanTile - 1) / kScanTile;
  long long* sums = static_cast<long long*>(workspace);
  if (n == 0) {
    cudaMemsetAsync(dTotal, 0, sizeof(long long), s);
    return;
  }
  scanReduceKernel<Tin><<<(unsigned)nb, kScanThreads, 0, s>>>(in, n, sums);
  scanBlockSumsKernel<<<1, 1024, 0, s>>>(sums, (int)nb, dTotal);
  scanDownsweepKernel<Tin><<<(unsigned)nb, kScanThreads, 0, s>>>(in, n, sums, out);
  if (lc) lc->add(3);
}
template void scanExclusive<int>(const int*, long long*, long, void*, long long*, cudaStream_t, LaunchCounter*);

//------------------------------------------------------------------------------
// Stable LSD radix sort, 8-bit digits, one kernel per digit.
//
// One pass over the keys counts the digits of every place; each digit's kernel
// then ranks its tile, obtains the number of equal digits in the tiles before
// it from their published counts (decoupled look-back) and scatters.  Tiles
// take their numbers from a counter, so every tile a block waits for has
// already started; the wait is bounded all the same and reports through
// `timeout` (the scatter is then skipped, so the output keeps what it held).
// A sort is 2 + digits launches (a clear, the count, one per digit; the node
// sort, whose key kernel counts, only the last) where the count / scan / scatter
// form took 5 per digit, which bound the neighbour build of small problems: 3375
// nodes 52 -> 14 us, 2.1 M nodes 119 -> 88 us.
//------------------------------------------------------------------------------
namespace {
constexpr int kSortThreads = 256;
constexpr int kSortRounds = 8;
constexpr int kSortTile = kSortThreads * kSortRounds;
constexpr int kWarps = kSortThreads / 32;
constexpr int kMaxDigits = 8;
constexpr unsigned kAggregate = 1u << 30, kInclusive = 2u << 30, kCountMask = (1u << 30) - 1u;
constexpr int kLookbackLimit = 1 << 24;   // polls before a wait gives up

// Workspace: digit counts [kMaxDigits][256] | tile counters [kMaxDigits] | tile status [digits][tiles][256]
struct SortWs {
  unsigned *hist, *ticket, *status;
};
SortWs sortWs(void* ws) {
  unsigned* u = static_cast<unsigned*>(ws);
  return SortWs{u, u + kMaxDigits * 256, u + kMaxDigits * 256 + 64};
}

template <typename K>
__global__ void __launch_bounds__(kSortThreads) radixCountKernel(const K* __restrict__ keys, long n, int digits,
                                                                 unsigned* __restrict__ hist) {
  __shared__ unsigned h[kMaxDigits][256];
  for (int d = 0; d < digits; ++d) h[d][threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (long b = blockIdx.x * (long)blockDim.x + threadIdx.x - lane; b < n; b += (long)gridDim.x * blockDim.x) {
    const bool valid = b + lane < n;
    const K k = valid ? keys[b + lane] : 0;
    for (int d = 0; d < digits; ++d) {
      const unsigned digit = valid ? (unsigned)(k >> (8 * d)) & 0xffu : 256u;
      int all;   // nearly sorted input: the high digits of a warp are mostly equal
      __match_all_sync(0xffffffffu, digit, &all);
      if (all) {
        if (lane == 0) atomicAdd(&h[d][digit], 32u);
      } else if (valid) {
        atomicAdd(&h[d][digit], 1u);
      }
    }
  }
  __syncthreads();
  for (int d = 0; d < digits; ++d)
    if (const unsigned c = h[d][threadIdx.x]) atomicAdd(&hist[d * 256 + threadIdx.x], c);
}

template <typename K>
__global__ void __launch_bounds__(kSortThreads) radixPassKernel(const K* __restrict__ keysIn,
                                                                const int* __restrict__ valsIn, long n, int shift,
                                                                const unsigned* __restrict__ hist,
                                                                unsigned* __restrict__ ticket,
                                                                unsigned* __restrict__ status, K* __restrict__ keysOut,
                                                                int* __restrict__ valsOut, int* __restrict__ timeout) {
  __shared__ unsigned warpHist[kWarps][256];
  __shared__ unsigned base[256];
  __shared__ unsigned scanWs[32];
  __shared__ unsigned sTile;
  __shared__ int sFail;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (t == 0) { sTile = atomicAdd(ticket, 1u); sFail = 0; }
#pragma unroll
  for (int w = 0; w < kWarps; ++w) warpHist[w][t] = 0;
  __syncthreads();
  const unsigned tile = sTile;
  // each warp takes a contiguous segment, so (warp, round, lane) is input order
  const long first = (long)tile * kSortTile + warp * (32 * kSortRounds) + lane;
  K key[kSortRounds];
  int val[kSortRounds];
  unsigned rank[kSortRounds];
  const unsigned below = (1u << lane) - 1u;
#pragma unroll
  for (int r = 0; r < kSortRounds; ++r) {
    const long idx = first + 32 * r;
    key[r] = 0;
    val[r] = 0;
    if (idx < n) { key[r] = keysIn[idx]; val[r] = valsIn[idx]; }
  }
#pragma unroll
  for (int r = 0; r < kSortRounds; ++r) {
    const bool valid = first + 32 * r < n;
    const unsigned digit = valid ? (unsigned)(key[r] >> shift) & 0xffu : 256u + lane;   // idle lanes stand alone
    const unsigned peers = __match_any_sync(0xffffffffu, digit);
    unsigned old = 0;
    if (valid && lane == __ffs(peers) - 1) {
      old = warpHist[warp][digit];
      warpHist[warp][digit] = old + __popc(peers);
    }
    old = __shfl_sync(0xffffffffu, old, __ffs(peers) - 1);
    rank[r] = old + __popc(peers & below);
    __syncwarp();
  }
  __syncthreads();
  // digit t: counts before each warp, the tile's count
  unsigned count = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const unsigned c = warpHist[w][t];
    warpHist[w][t] = count;
    count += c;
  }
  volatile unsigned* st = status;
  st[(size_t)tile * 256 + t] = (tile == 0 ? kInclusive : kAggregate) | count;
  const unsigned digitStart = blockExclusiveScan<unsigned>(hist[t], scanWs, nullptr);
  unsigned before = 0;
  if (tile > 0) {
    long p = (long)tile - 1;
    int polls = 0;
    while (true) {
      const unsigned v = st[(size_t)p * 256 + t];
      if (v & (kAggregate | kInclusive)) {
        before += v & kCountMask;
        if (v & kInclusive) break;
        --p;
      } else if (++polls > kLookbackLimit) {
        sFail = 1;
        break;
      }
    }
    st[(size_t)tile * 256 + t] = kInclusive | (before + count);
  }
  base[t] = digitStart + before;
  __syncthreads();
  if (sFail) {
    if (t == 0) atomicExch(timeout, 1);
    return;
  }
#pragma unroll
  for (int r = 0; r < kSortRounds; ++r)
    if (first + 32 * r < n) {
      const unsigned digit = (unsigned)(key[r] >> shift) & 0xffu;
      const unsigned pos = base[digit] + warpHist[warp][digit] + rank[r];
      keysOut[pos] = key[r];
      valsOut[pos] = val[r];
    }
}
}  // namespace

size_t radixSortWorkspaceBytes(long n) {
  const long nb = (n + kSortTile - 1) / kSortTile;
  return ((size_t)kMaxDigits * 256 + 64 + (size_t)kMaxDigits * nb * 256) * sizeof(unsigned);
}

SortPrep radixSortPrep(void* workspace, long n, int bits) {
  const long nb = (n + kSortTile - 1) / kSortTile;
  const SortWs w = sortWs(workspace);
  const int digits = (bits + 7) / 8;
  return SortPrep{w.hist, digits, w.ticket, 64 + (long long)digits * nb * 256};
}

template <typename K>
void radixSortPairs(K*& keys, int*& vals, K*& keysAlt, int*& valsAlt, long n, int bits, void* workspace, int* timeout,
                    bool counted, cudaStream_t s, LaunchCounter* lc) {
  if (n <= 1) return;
  const long nb = (n + kSortTile - 1) / kSortTile;
  const int digits = (bits + 7) / 8;
  const SortWs w = sortWs(workspace);
  if (!counted) {
    cudaMemsetAsync(workspace, 0, ((size_t)kMaxDigits * 256 + radixSortPrep(workspace, n, bits).nclear) * sizeof(unsigned), s);
    radixCountKernel<K><<<(unsigned)std::min<long>(nb, 1216), kSortThreads, 0, s>>>(keys, n, digits, w.hist);
  }
  for (int d = 0; d < digits; ++d) {
    radixPassKernel<K><<<(unsigned)nb, kSortThreads, 0, s>>>(keys, vals, n, 8 * d, w.hist + 256 * d, w.ticket + d,
                                                             w.status + (size_t)d * nb * 256, keysAlt, valsAlt, timeout);
    std::swap(keys, keysAlt);
    std::swap(vals, valsAlt);
  }
  if (lc) lc->add((counted ? 0 : 1) + digits);
}
template void radixSortPairs<uint32_t>(uint32_t*&, int*&, uint32_t*&, int*&, long, int, void*, int*, bool,
                                       cudaStream_t, LaunchCounter*);
template void radixSortPairs<uint64_t>(uint64_t*&, int*&, uint64_t*&, int*&, long, int, void*, int*, bool,
                                       cudaStream_t, LaunchCounter*);

}  // namespace sph
