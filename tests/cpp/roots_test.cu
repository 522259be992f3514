// Points evaluated, and the largest distance in units in the last place: of rcp_fast from 1 / x, of
// rsqrt_fast from rsqrt(x), of the FP32 root of sqrt_and_inverse from the correctly rounded one (the
// FP64 root rounded: exact by its 53 bits), of the FP64 root from sqrt(x), and of both inverses from
// 1 / root. Exits with a number other than 0 if anything failed to run.
#include "rds_math.cuh"

#include <cstdio>

__global__ void distances(unsigned long long *out)
{
  const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned long long h = (i + 1) * 0x9E3779B97F4A7C15ull; // mantissas: multiplicative hash
  const double m             = 1.0 + (double)(h >> 12) * 0x1p-52;
  const double x             = ldexp(m, (int)(i % 2001) - 1000);
  const float xf             = (float)ldexp(m, (int)(i % 241) - 120);
  auto ulp = [](double a, double b) {
    const long long d = __double_as_longlong(a) - __double_as_longlong(b);
    return (unsigned long long)(d < 0 ? -d : d);
  };
  atomicAdd(out, 1ull);
  atomicMax(out + 1, ulp(rds::rcp_fast(x), 1.0 / x));
  atomicMax(out + 2, ulp(rds::rsqrt_fast(x), rsqrt(x)));
  double inv      = 0.0;
  const float s   = rds::sqrt_and_inverse(xf, inv);
  const int d     = __float_as_int(s) - __float_as_int((float)sqrt((double)xf));
  atomicMax(out + 3, (unsigned long long)(d < 0 ? -d : d));
  atomicMax(out + 5, ulp(inv, 1.0 / (double)s));
  const double r = rds::sqrt_and_inverse(x, inv);
  atomicMax(out + 4, ulp(r, sqrt(x)));
  atomicMax(out + 5, ulp(inv, 1.0 / r));
}

int main()
{
  unsigned long long *d = nullptr, h[6];
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess)
    return 1;
  distances<<<4096, 256>>>(d);
  if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess)
    return 2;
  if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess)
    return 3;
  std::printf("%llu %llu %llu %llu %llu %llu\n", h[0], h[1], h[2], h[3], h[4], h[5]);
  return 0;
}
