// Largest distance, in units in the last place, of rcp_fast and rsqrt_fast (rds_math.cuh) from
// the library's 1 / x and rsqrt(x) over numbers spread over the exponent range. Prints both.
#include "rds_math.cuh"

#include <cstdio>

__global__ void distance(long long *worst)
{
  const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  // exponents 2^-1000 .. 2^1000, mantissa bits from a multiplicative hash
  const unsigned long long h = (i + 1) * 0x9E3779B97F4A7C15ull;
  const double x = ldexp(1.0 + (double)(h >> 12) * 0x1p-52, (int)(i % 2001) - 1000);
  auto ulp = [](double a, double b) {
    const long long d = __double_as_longlong(a) - __double_as_longlong(b);
    return d < 0 ? -d : d;
  };
  atomicMax(worst, ulp(rds::rcp_fast(x), 1.0 / x));
  atomicMax(worst + 1, ulp(rds::rcp_fast(-x), -1.0 / x));
  atomicMax(worst + 2, ulp(rds::rsqrt_fast(x), rsqrt(x)));
}

int main()
{
  long long *d = nullptr, h[3] = {-1, -1, -1};
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess)
    return 1;
  distance<<<4096, 256>>>(d);
  if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess)
    return 1;
  std::printf("%lld %lld %lld\n", h[0], h[1], h[2]);
  return 0;
}
