// Scan / sort utilities of libsphgpu.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <utility>

namespace sph {

// Counts kernel launches issued by the library (reported by sphgpu_launch_count).
struct LaunchCounter {
  long n = 0;
  void add(long k) { n += k; }
};

size_t scanWorkspaceBytes(long n);
// out[i] = sum_{k<i} in[k] (int64); *dTotal (device) = sum of all.
template <typename Tin>
void scanExclusive(const Tin* in, long long* out, long n, void* workspace, long long* dTotal, cudaStream_t s,
                   LaunchCounter* lc);

size_t radixSortWorkspaceBytes(long n);
// Leading words of the workspace that must be zero before the sort (cleared:
// the caller has zeroed them in stream order; otherwise the sort does).
size_t radixSortClearedWords(long n, int bits);
// Stable sort of (keys, vals) by the low `bits` bits of keys (uint32_t or
// uint64_t, at most 2^30 pairs).  The pointers are ping-ponged: on return
// keys/vals point at the sorted data.  *timeout (device) is set when a bounded
// wait inside the sort ran out; the output is then not sorted.
template <typename K>
void radixSortPairs(K*& keys, int*& vals, K*& keysAlt, int*& valsAlt, long n, int bits, void* workspace, int* timeout,
                    bool cleared, cudaStream_t s, LaunchCounter* lc);

}  // namespace sph
