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
// A caller whose kernel forms the keys may count their digits there and zero the
// rest of the workspace, which saves a launch, a clear and a pass over the keys
// (radixSortPairs with counted): hist[256 d + digit] += 1 for every key and
// digit place d < digits, on a hist that is zero, and words [0, nclear) of clear
// set to zero, all in stream order before the sort.  The sort leaves hist as it
// is; whoever counts clears it for the next time.
struct SortPrep {
  unsigned* hist;
  int digits;
  unsigned* clear;
  long long nclear;
};
SortPrep radixSortPrep(void* workspace, long n, int bits);
// Stable sort of (keys, vals) by the low `bits` bits of keys (uint32_t or
// uint64_t, at most 2^30 pairs).  The pointers are ping-ponged: on return
// keys/vals point at the sorted data.  *timeout (device) is set when a bounded
// wait inside the sort ran out; the output is then not sorted.
template <typename K>
void radixSortPairs(K*& keys, int*& vals, K*& keysAlt, int*& valsAlt, long n, int bits, void* workspace, int* timeout,
                    bool counted, cudaStream_t s, LaunchCounter* lc);

}  // namespace sph
