// Test program: rc::less (csrc/rc_div.cuh) against the FP64 compare, and
// rc::twice_of against the FP64 multiply, on random bit patterns of every
// exponent, equal and neighbouring pairs among them, and on all pairs of a
// list of edge values.  Prints the counts; exits 1 on any difference.
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "rc_div.cuh"

__device__ uint64_t mix(uint64_t x) {
  x ^= x >> 33; x *= 0xff51afd7ed558ccdULL; x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ULL; x ^= x >> 33;
  return x;
}
__device__ bool same(double a, double b) {
  if (isnan(a) || isnan(b)) return isnan(a) && isnan(b);
  return __double_as_longlong(a) == __double_as_longlong(b);
}
__device__ void one(uint64_t x, uint64_t y, unsigned long long* bad) {
  const double a = __longlong_as_double((long long)x), b = __longlong_as_double((long long)y);
  if (rc::less(a, b) != (a < b) || rc::less(b, a) != (b < a) || !same(rc::twice_of(a), 2.0 * a)) atomicAdd(bad, 1ULL);
}
constexpr int NEDGE = 16;
__device__ const uint64_t edge[NEDGE] = {
    0x0000000000000000ULL, 0x8000000000000000ULL, 0x0000000000000001ULL, 0x8000000000000001ULL,
    0x000fffffffffffffULL, 0x0010000000000000ULL, 0x8010000000000000ULL, 0x3ff0000000000000ULL,
    0xbff0000000000000ULL, 0x7fefffffffffffffULL, 0xffefffffffffffffULL, 0x7fe0000000000000ULL,
    0x7ff0000000000000ULL, 0xfff0000000000000ULL, 0x7ff8000000000000ULL, 0xfff8000000000001ULL};
__global__ void check(unsigned long long n, unsigned long long* bad) {
  const unsigned long long t = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
  if (t < NEDGE * NEDGE) one(edge[t / NEDGE], edge[t % NEDGE], bad);
  for (unsigned long long i = t; i < n; i += (unsigned long long)gridDim.x * blockDim.x) {
    const uint64_t x = mix(2 * i + 1), z = mix(2 * i + 2);
    uint64_t y = z;
    if ((i & 7) == 0) y = x;
    else if ((i & 7) == 1) y = x + 1;
    else if ((i & 7) == 2) y = x ^ 0x8000000000000000ULL;
    else if ((i & 7) == 3) y = (x & 0xffffffff00000000ULL) | (z & 0xffffffffULL);
    one(x, y, bad);
  }
}
int main(int argc, char** argv) {
  const unsigned long long n = argc > 1 ? strtoull(argv[1], nullptr, 10) : 1ULL << 24;
  unsigned long long *d, bad = 0;
  if (cudaMalloc(&d, sizeof(*d)) != cudaSuccess) return 2;
  cudaMemset(d, 0, sizeof(*d));
  check<<<152 * 8, 256>>>(n, d);
  if (cudaMemcpy(&bad, d, sizeof(bad), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  printf("pairs %llu mismatches %llu\n", n, bad);
  return bad ? 1 : 0;
}
