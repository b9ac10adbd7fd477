// FP64 helpers of the FMA build at the ends of their ranges, for
// test_gpu_fp64_floors.py: prints a name and a number per group: of the values
// that differ from CUDA's own functions, or the largest relative error in 2^-53.
#include <cmath>
#include <cstdio>
#include "ek_hydro.cuh"
#include "ek_mhd.cuh"
using namespace ek_fast;

__device__ unsigned g_bad[2];
__device__ double   g_err[3];

__device__ void
same(int k, double x, double y)
{
  if (!(x == y))
    atomicAdd(&g_bad[k], 1u);
}

__global__ void
floors()
{
  const double v[] = { 0.0,   5e-324, 3e-310, 2.3e-308, 1e-300, 1e-160, 1e-30, 1e-20, 6e-11, 1e-10,
                       1e-5,  0.1,    0.4,    0.5,      0.9,    1.0,    1.1,   2.0,   3.0,   1e10,
                       1e150, 1e300,  1.7e308 };
  const int    n = sizeof v / sizeof v[0];
  for (int i = 0; i < n; ++i)
    for (int k = 0; k < n; ++k)
    {
      same(0, max_floor64(v[i], v[k]), fmax(v[i], v[k]));
      same(0, max_floor64(-v[i], v[k]), fmax(-v[i], v[k]));
      same(0, max_floor64(INFINITY, v[k]), INFINITY);
      for (int j = 0; j < n; ++j)
        if (v[k] > 0.0 && v[j] * v[k] < INFINITY) // density v[k], floor v[j]
        {
          const double f = v[k] * v[j];
          same(0, floor_ratio64(v[i], v[k], v[j]), fmax(v[i], f));
          same(0, floor_ratio64(-v[i], v[k], v[j]), fmax(-v[i], f));
          same(0, floor_ratio64(INFINITY, v[k], v[j]), INFINITY);
          // beside the floor itself
          for (double r : { 0.49, 0.999999, 1.0, 1.000001, 2.01 })
            same(0, floor_ratio64(r * f, v[k], v[j]), fmax(r * f, f));
        }
    }
}

__global__ void
nans()
{
  const double v[] = { 0.0, 5e-324, 1e-300, 1e-20, 1e-10, 0.3, 1.0, 7.0, 1e200 };
  for (double f : v)
    for (long long bits : { 0x7ff8000000000000ll, 0x7ff0000000000001ll, 0x7fffffffffffffffll })
      for (long long sign : { 0ll, (long long)0x8000000000000000ull })
      {
        const double x = __longlong_as_double(bits | sign);
        same(1, max_floor64(x, f), f);
        same(1, floor_ratio64(x, 0.3, f), 0.3 * f);
        same(1, floor_ratio64(x, 1e10, f), 1e10 * f);
        same(1, max_cand64(f, x), f);
      }
}

// SplitMix64's finaliser
__device__ unsigned long long
mix(unsigned long long z)
{
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
// a random significand with a binary exponent in [-spread, spread)
__device__ double
value(unsigned long long z, int spread)
{
  return __longlong_as_double((z & 0x000fffffffffffffull) | ((1023ull - spread + (z >> 53) % (2 * spread)) << 52));
}
__device__ void
at_most(int k, double got, double want) // relative error in 2^-53
{
  double e = fabs(got / want - 1.0) * 0x1p53;
  if (!(e < 1e30))
    e = 1e30;
  atomicMax((unsigned long long *)&g_err[k], (unsigned long long)__double_as_longlong(e));
}
__global__ void
roots()
{
  const unsigned long long t = blockIdx.x * blockDim.x + threadIdx.x;
  for (int i = 0; i < 64; ++i)
  {
    unsigned long long z = mix(t * 64 + i + 1);
    auto   next = [&](int spread) { return value(z = mix(z + 0x9E3779B97F4A7C15ull), spread); };
    const double n1 = next(1000), d1 = next(1000), n2 = next(1000), d2 = next(1000);
    auto   ok = [](double n, double d) { return n / d > 1e-300 && n / d < 1e300; };
    if (ok(n1, d1))
      at_most(0, sqrt_ratio64(n1, d1), sqrt(n1 / d1));
    if (ok(n1, d1) && ok(n2, d2))
    {
      at_most(1, sqrt_larger_ratio64(n1, d1, n2, d2), fmax(sqrt(n1 / d1), sqrt(n2 / d2)));
      at_most(1, sqrt_larger_ratio64(0.0, d1, n2, d2), sqrt(n2 / d2));
    }
    // rho c_fast^2 scales with its terms
    const double gp = next(8), b2 = next(8), bn2 = b2 * 0.7, s = scale_pos64<1>(b2 + gp);
    const double want = s + sqrt(fmax(fma(s, s, -(gp * bn2)), 0.0));
    for (int k = -1000; k <= 1000; k += 100)
    {
      const double f = ldexp(1.0, k);
      at_most(2, ldexp(fast_num64(gp * f, b2 * f, bn2 * f), -k), want);
    }
  }
  // no field and no pressure
  if (t == 0 && !(sqrt_ratio64(0.0, 1e-10) == 0.0 && sqrt_larger_ratio64(0.0, 1.0, 0.0, 2.0) == 0.0 &&
                  fast_num64(0.0, 0.0, 0.0) == 0.0 && isnan(sqrt_ratio64(NAN, 1.0))))
    at_most(0, 0.0, 1.0);
}

int
main()
{
  floors<<<1, 1>>>();
  nans<<<1, 1>>>();
  roots<<<64, 256>>>();
  unsigned h[2];
  double   e[3];
  if (cudaMemcpyFromSymbol(h, g_bad, sizeof h) != cudaSuccess || cudaMemcpyFromSymbol(e, g_err, sizeof e) != cudaSuccess)
    return 1;
  printf("floors %u\nnan %u\nratio %.9g\nlarger %.9g\nfast %.9g\n", h[0], h[1], e[0], e[1], e[2]);
  return 0;
}
