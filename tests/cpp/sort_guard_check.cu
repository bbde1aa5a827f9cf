// What the neighbour build does after a node sort that gave up waiting: the
// keys are in no order (a cell comes up in several runs, cellEnd holds the end
// of one of them), and no item, list or entry may be formed from them.
#include "kernels.cuh"

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

using namespace sph;

#define OK(expr)                                                                    \
  do {                                                                              \
    const cudaError_t e_ = (expr);                                                  \
    if (e_ != cudaSuccess) { std::printf("%s: %s\n", #expr, cudaGetErrorString(e_)); return 2; } \
  } while (0)

template <class T>
T* device(const std::vector<T>& v) {
  T* p = nullptr;
  if (cudaMalloc(&p, v.size() * sizeof(T)) != cudaSuccess) return nullptr;
  cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
  return p;
}
template <class T>
std::vector<T> host(const T* p, size_t n) {
  std::vector<T> v(n);
  cudaMemcpy(v.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost);
  return v;
}

int main() {
  const long n = 5000;
  const int width = 32, bound = 4 * (int)n, cells = 64;
  std::mt19937 rng(7);
  for (int broken = 0; broken < 2; ++broken) {
    std::vector<uint32_t> keys(n);
    std::vector<int> end(cells, 0);
    for (auto& k : keys) k = rng() % cells;
    if (!broken) std::sort(keys.begin(), keys.end());
    for (long k = 0; k < n; ++k) end[keys[k]] = (int)k + 1;
    StepScratch s;
    std::memset(&s, 0, sizeof s);
    s.sortTimeout = broken;
    Fields32 P{};
    std::vector<float4> posh(n, make_float4(0.5f, 0.5f, 0.5f, 1.0f));
    std::vector<uint32_t> cellc(n, 0u);
    P.posh = device(posh);
    P.cell = device(cellc);
    Grid g{};
    for (int a = 0; a < 3; ++a) { g.nc[a] = 1; g.cellf[a] = 1.0f; g.cell[a] = 1.0; }
    g.ext2f = 4.0f;
    uint32_t* dKeys = device(keys);
    int* dEnd = device(end);
    int* items = device(std::vector<int>(2 * bound, -1));
    int* chunkOf = device(std::vector<int>(n, -1));
    int* counts = device(std::vector<int>(n, 7));
    float4* box = device(std::vector<float4>(3 * (size_t)bound, make_float4(0, 0, 0, 0)));
    StepScratch* sc = device(std::vector<StepScratch>(1, s));
    uint32_t* nbr = device(std::vector<uint32_t>(((n + 31) / 32) * 32 * 32, 0xffffffffu));
    LaunchCounter lc;
    launchItems(dKeys, n, 0, cells, dEnd, width, bound, g, false, P, items, chunkOf, counts, box, sc, 0, &lc);
    OK(cudaGetLastError());
    if (broken) {
      Fields F{};
      launchNeighborsWarp(F, P, n, items, bound, sc, width, g, dEnd, dEnd, counts, nbr, 32, 4.0, false, box, chunkOf, 0,
                          &lc);
      OK(cudaGetLastError());
    }
    OK(cudaDeviceSynchronize());
    const auto it = host(items, 2 * bound);
    const auto cn = host(counts, n);
    const StepScratch r = host(sc, 1)[0];
    if (broken) {
      for (const int v : it) if (v != -1) { std::printf("an item after a failed sort: %d\n", v); return 1; }
      for (const int v : cn) if (v != 0) { std::printf("a list after a failed sort: %d entries\n", v); return 1; }
      for (const uint32_t v : host(nbr, ((n + 31) / 32) * 32 * 32))
        if (v != 0xffffffffu) { std::printf("an entry after a failed sort\n"); return 1; }
      if (r.items != 0 || r.maxCount != 0) { std::printf("items %d, maxCount %d\n", r.items, r.maxCount); return 1; }
    } else {   // the sorted keys of the same cells: every node in exactly one chunk
      std::vector<int> seen(n, 0);
      for (int k = 0; k < r.items; ++k)
        for (long j = it[k]; j < n && j < it[k] + width && keys[j] == keys[it[k]]; ++j) ++seen[j];
      for (const int v : seen) if (v != 1) { std::printf("a node in %d chunks\n", v); return 1; }
    }
  }
  std::printf("ok\n");
  return 0;
}
