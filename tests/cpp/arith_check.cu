// arith_check.cu -- the branch-free reciprocal, square root, quotient and logarithm
// argument of ilc_device.cuh / ilc_quantity.cuh against the compiler's correctly
// rounded operations (-prec-div=true -prec-sqrt=true): prints one line per check,
// "name arguments mismatches".
#include <cstdio>
#include <cstring>

#include "ilc_device.cuh"
#include "ilc_quantity.cuh"

using namespace ilc;

__device__ bool differ(float a, float b) { return __float_as_uint(a) != __float_as_uint(b); }

// All significands at the exponents [e0, e1] (biased) within [lo, hi].
__global__ void rcp_kernel(int e0, int e1, float lo, float hi, unsigned long long* bad,
                           unsigned long long* n) {
  const unsigned long long all = (unsigned long long)(e1 - e0 + 1) << 23;
  unsigned long long b = 0, k = 0;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < all;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const float x = __uint_as_float(((unsigned)e0 << 23) + (unsigned)i);
    if (!(x >= lo && x <= hi)) continue;
    ++k;
    b += differ(rcp_normal(x), 1.0f / x);
  }
  atomicAdd(bad, b);
  atomicAdd(n, k);
}
__global__ void sqrt_kernel(int e0, int e1, float lo, float hi, unsigned long long* bad,
                            unsigned long long* n) {
  const unsigned long long all = (unsigned long long)(e1 - e0 + 1) << 23;
  unsigned long long b = 0, k = 0;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < all;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const float x = __uint_as_float(((unsigned)e0 << 23) + (unsigned)i);
    if (!(x >= lo && x <= hi)) continue;
    ++k;
    b += differ(sqrt_normal(x), sqrtf(x));
  }
  atomicAdd(bad, b);
  atomicAdd(n, k);
}
__global__ void log_ratio_kernel(unsigned first, unsigned last, unsigned long long* bad,
                                 unsigned long long* n) {
  unsigned long long b = 0, k = 0;
  for (unsigned i = first + blockIdx.x * blockDim.x + threadIdx.x; i <= last;
       i += gridDim.x * blockDim.x) {
    const float m = __uint_as_float(i);
    ++k;
    b += differ(log_ratio(m), (m - 1.0f) / (m + 1.0f));
  }
  atomicAdd(bad, b);
  atomicAdd(n, k);
}

__device__ unsigned hash(unsigned long long x) {  // splitmix64, upper half
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return (unsigned)((x ^ (x >> 31)) >> 32);
}
// A float of a seeded significand (every fourth one all ones, next to one or a power
// of two) and an exponent of [lo, hi].
__device__ float draw(unsigned long long k, int lo, int hi) {
  const unsigned r = hash(k), s = hash(k ^ 0x5555555555555555ull);
  unsigned m = r & 0x7fffffu;
  if ((s & 3u) == 0u) m = (s & 4u) ? 0x7fffffu - ((s >> 3) & 3u) : (s >> 3) & 3u;
  return __uint_as_float(((unsigned)(127 + lo + (int)((s >> 8) % (unsigned)(hi - lo + 1))) << 23) |
                         m);
}
// a / b with a in 2^[a0, a1], b in 2^[b0, b1] and the quotient in 2^[q0, q1].
__global__ void div_kernel(unsigned long long count, unsigned long long seed, int a0, int a1,
                           int b0, int b1, float qmin, float qmax, unsigned long long* bad,
                           unsigned long long* n) {
  unsigned long long w = 0, k = 0;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
       i < count; i += (unsigned long long)gridDim.x * blockDim.x) {
    const float a = draw(2 * (seed + i), a0, a1), b = draw(2 * (seed + i) + 1, b0, b1);
    const float q = a / b;
    if (!(q >= qmin && q <= qmax)) continue;
    ++k;
    w += differ(div_by(a, b, 1.0f / b), q) + differ(div_by(-a, b, 1.0f / b), -q);
  }
  atomicAdd(bad, w);
  atomicAdd(n, k);
}

static unsigned long long* counts;
static int report(const char* name) {
  unsigned long long h[2];
  if (cudaDeviceSynchronize() != cudaSuccess ||
      cudaMemcpy(h, counts, 16, cudaMemcpyDeviceToHost) != cudaSuccess) {
    std::printf("CUDA error: %s\n", cudaGetErrorString(cudaGetLastError()));
    return 1;
  }
  std::printf("%s %llu %llu\n", name, h[1], h[0]);
  return cudaMemset(counts, 0, 16) != cudaSuccess;
}

static unsigned bits(float f) {
  unsigned u;
  std::memcpy(&u, &f, 4);
  return u;
}

int main() {
  if (cudaMalloc(&counts, 16) != cudaSuccess || cudaMemset(counts, 0, 16) != cudaSuccess) return 1;
  int rc = 0;
  const int blocks = 148 * 8;
  // both exponent parities, and the ends of plain_d2's range
  struct { int e0, e1; } spans[] = {{27, 29}, {126, 129}, {225, 226}};
  for (auto s : spans) {
    rcp_kernel<<<blocks, 256>>>(s.e0, s.e1, 1e-30f, 1e30f, counts, counts + 1);
    rc |= report("rcp_normal");
    sqrt_kernel<<<blocks, 256>>>(s.e0, s.e1, 1e-30f, 1e30f, counts, counts + 1);
    rc |= report("sqrt_normal");
  }
  // mantissas as log_normal folds them: (1.41421356 / 2, 1.41421356]
  log_ratio_kernel<<<blocks, 256>>>(bits(0.70710678f), bits(1.41421356f), counts, counts + 1);
  rc |= report("log_ratio");
  // the quotients of emit(): 1e3 E / kT, log / spacing, emission / r^2, flux / E
  const unsigned long long many = 1ull << 28;
  div_kernel<<<blocks, 256>>>(many, 1ull << 40, -16, 36, -49, 49, 1e-20f, 1e26f, counts,
                              counts + 1);
  rc |= report("div_by");
  div_kernel<<<blocks, 256>>>(many, 2ull << 40, -24, 20, -20, 19, 0.0f, 3e38f, counts, counts + 1);
  rc |= report("div_by");
  div_kernel<<<blocks, 256>>>(many, 3ull << 40, -66, 93, -66, 66, 1e-26f, 1e26f, counts,
                              counts + 1);
  rc |= report("div_by");
  div_kernel<<<blocks, 256>>>(many, 4ull << 40, -86, 86, -26, 26, 1e-34f, 1e34f, counts,
                              counts + 1);
  rc |= report("div_by");
  return rc;
}
