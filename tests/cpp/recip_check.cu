// Error of rcp64 and rsqrt64 (recip64.cuh) in units in the last place against
// quotients and roots in the host's long double, over random mantissas at every
// exponent of their ranges and the values next to powers of two.  Prints, per
// function: largest error, mean signed error, count.
#include "recip64.cuh"

#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

__global__ void evaluate(const double* x, double* r, double* q, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  r[i] = sph::dev::rcp64(x[i]);
  q[i] = sph::dev::rsqrt64(fabs(x[i]));
}

int main() {
  std::vector<double> x;
  std::mt19937_64 rng(11);
  for (int e = -1022; e <= 1020; ++e) {
    const double p = std::ldexp(1.0, e);
    x.push_back(p);
    x.push_back(std::nextafter(p, 2.0 * p));
    x.push_back(std::nextafter(2.0 * p, p));
    x.push_back(-p);
    for (int k = 0; k < 500; ++k) {
      const double m = std::ldexp(1.0 + (double)(rng() >> 12) * std::ldexp(1.0, -52), e);
      x.push_back(k & 1 ? -m : m);
    }
  }
  const int n = (int)x.size();
  double *dx, *dr, *dq;
  if (cudaMalloc(&dx, 8 * n) || cudaMalloc(&dr, 8 * n) || cudaMalloc(&dq, 8 * n)) return 2;
  cudaMemcpy(dx, x.data(), 8 * n, cudaMemcpyHostToDevice);
  evaluate<<<(n + 255) / 256, 256>>>(dx, dr, dq, n);
  std::vector<double> r(n), q(n);
  cudaMemcpy(r.data(), dr, 8 * n, cudaMemcpyDeviceToHost);
  if (cudaMemcpy(q.data(), dq, 8 * n, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  auto report = [&](const char* name, const std::vector<double>& y, auto ref) {
    long double worst = 0.0L, mean = 0.0L;
    for (int i = 0; i < n; ++i) {
      const long double want = ref((long double)x[i]);
      int e;
      std::frexp((double)fabsl(want), &e);
      const long double err = ((long double)y[i] - want) / ldexpl(1.0L, e - 53) * (want < 0 ? -1.0L : 1.0L);
      if (!(fabsl(err) <= worst)) worst = fabsl(err);
      mean += err / n;
    }
    std::printf("%s %.6f %.6f %d\n", name, (double)worst, (double)mean, n);
  };
  report("rcp", r, [](long double v) { return 1.0L / v; });
  report("rsqrt", q, [](long double v) { return 1.0L / sqrtl(fabsl(v)); });
  return 0;
}
