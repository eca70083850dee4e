// Compares root() with the rounded square root over mantissas and exponents, and
// rsqrt_approx() with 1 / sqrt. Prints the largest difference in units of the last
// place and the largest relative error of the approximation, in units of 2^-19.
#include <cstdio>

#include "root.cuh"

struct Worst {
  unsigned long long ulps;
  double at, approx, approx_at;
};

__device__ double sample(unsigned long long k) {
  // Exponents -996 .. 1023 in turn (both parities; 1e-300 is 2^-997); mantissas
  // from a hash, and every 16th close to the ends of its binade.
  unsigned long long h = k * 0x9E3779B97F4A7C15ull;
  h = (h ^ (h >> 31)) * 0xBF58476D1CE4E5B9ull;
  h ^= h >> 29;
  unsigned long long m = h >> 12;
  if (k % 16 == 0) m &= 0xff;
  if (k % 16 == 1) m |= 0xfffffffffff00ull;
  return __longlong_as_double((long long)(((k % 2020 + 27) << 52) | m));
}

__global__ void check(unsigned long long n, Worst *out) {
  Worst w{0, 0.0, 0.0, 0.0};
  const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long k = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += step) {
    const double x = sample(k), s = sqrt(x);
    const long long d = __double_as_longlong(fln::root(x)) - __double_as_longlong(s);
    const unsigned long long u = (unsigned long long)(d < 0 ? -d : d);
    if (u > w.ulps) w.ulps = u, w.at = x;
    const double e = fabs(fma(fln::rsqrt_approx(x), s, -1.0)) * 0x1p19;
    if (!(e <= w.approx)) w.approx = e, w.approx_at = x;
  }
  out[blockIdx.x * blockDim.x + threadIdx.x] = w;
}

int main() {
  constexpr int kBlocks = 592, kThreads = 256;
  Worst *w;
  if (cudaMallocManaged(&w, kBlocks * kThreads * sizeof(Worst)) != cudaSuccess) return 1;
  check<<<kBlocks, kThreads>>>(1ull << 28, w);
  if (cudaDeviceSynchronize() != cudaSuccess) return 1;
  Worst a = w[0];
  for (int k = 1; k < kBlocks * kThreads; ++k) {
    if (w[k].ulps > a.ulps) a.ulps = w[k].ulps, a.at = w[k].at;
    if (!(w[k].approx <= a.approx)) a.approx = w[k].approx, a.approx_at = w[k].approx_at;
  }
  std::printf("%llu %.17g %.6f %.17g\n", a.ulps, a.at, a.approx, a.approx_at);
  return 0;
}
