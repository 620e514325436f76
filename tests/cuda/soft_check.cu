// Test program: the multiplication, division and square root on the integer
// pipes (csrc/rc_soft.cuh) against the hardware's, bit for bit.  Compiled by
// nvcc it runs on the GPU, compiled as C++ on the processor (where it also
// shifts the reciprocal seeds by an ulp each way).  Operands: random
// significands with runs of zeros and ones, exponents within and beyond the
// integer path's range, zeros, subnormals, infinities and NaNs; products that
// are ties and squares of short numbers with their neighbours.  Prints the
// counts; exits 1 on any difference (NaNs compare as NaN == NaN).
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "rc_soft.cuh"

#ifdef __CUDACC__
#define HD __host__ __device__
#else
#define HD
#endif

HD inline uint64_t mix(uint64_t x) {
  x ^= x >> 33; x *= 0xff51afd7ed558ccdULL; x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ULL; x ^= x >> 33;
  return x;
}
HD inline uint64_t bits(double x) { return ((uint64_t)rcs::hi32(x) << 32) | rcs::lo32(x); }
HD inline bool nan(double x) { return (bits(x) << 1) > 0xffe0000000000000ULL; }
HD inline bool same(double a, double b) { return (nan(a) && nan(b)) || bits(a) == bits(b); }
HD inline double operand(uint64_t s) {
  const uint64_t r = mix(s), k = r & 15;
  uint64_t m = mix(s + 0x9e3779b97f4a7c15ULL) & 0xfffffffffffffULL;
  if (k == 0) m = 0;
  if (k == 1) m = 0xfffffffffffffULL;
  if (k == 2) m &= ~0xffffffffULL;
  if (k == 3) m |= 0xffffffffULL;
  if (k == 4) m &= 0xff;
  if (k == 5) m = 0xfffffffffffffULL - (m & 0xff);
  if (k == 6) m = 1ULL << (m % 52);
  if (k == 7) m &= ~0x3ffffffULL;  // 26 bits: products of two are exact or ties
  uint64_t e = 1023 + (r >> 8) % 9 - 4;
  if ((r >> 40 & 3) == 0) e = 1023 + (r >> 8) % 830 - 415;
  if ((r >> 40 & 63) == 1) e = (r >> 8) & 0x7ff;
  if ((r >> 40 & 63) == 2) { e = 0; m = (r & 16) ? m : 0; }
  if ((r >> 40 & 255) == 3) e = 0x7ff;
  return rcs::make64(r >> 63 << 63 | e << 52 | m);
}
HD inline int differences(uint64_t i) {
  const double a = operand(2 * i), b = operand(2 * i + 1);
  int bad = !same(rcs::mul(a, b), a * b) + !same(rcs::div(a, b), a / b) + !same(rcs::div(a * b, b), (a * b) / b);
  double x = rcs::make64(bits(a) & 0x7fffffffffffffffULL);
  if (i % 3 == 0) { const float f = (float)b; x = (double)f * (double)f; }
  if (i % 5 == 0) x = rcs::make64(bits(x) + i % 15 / 5 - 1);
  if (i % 64 == 7) x = a;
#ifdef __CUDA_ARCH__
  bad += !same(rcs::sqrt(x), ::sqrt(x));
#else
  bad += !same(rcs::sqrt(x), std::sqrt(x));
#endif
  return bad;
}

#ifdef __CUDACC__
__global__ void check(unsigned long long n, unsigned long long* bad) {
  unsigned long long nb = 0;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x)
    nb += differences(i);
  if (nb) atomicAdd(bad, nb);
}
#endif
int main(int argc, char** argv) {
  const unsigned long long n = argc > 1 ? strtoull(argv[1], nullptr, 10) : 1ULL << 24;
  unsigned long long bad = 0;
#ifdef __CUDACC__
  unsigned long long* d;
  if (cudaMalloc(&d, sizeof(*d)) != cudaSuccess) return 2;
  cudaMemset(d, 0, sizeof(*d));
  check<<<152 * 8, 256>>>(n, d);
  if (cudaMemcpy(&bad, d, sizeof(bad), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
#else
  for (rcs::seed_ulps = -1; rcs::seed_ulps <= 1; ++rcs::seed_ulps)
    for (unsigned long long i = 0; i < n; ++i) bad += differences(i);
#endif
  printf("samples %llu mismatches %llu\n", n, bad);
  return bad ? 1 : 0;
}
