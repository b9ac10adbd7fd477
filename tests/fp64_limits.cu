// FP64 helpers of the FMA build at the ends of their ranges, for
// test_gpu_fp64_floors.py: prints a name and a number per group, of the values
// that differ from CUDA's own functions.
#include <cmath>
#include <cstdio>
#include "ek_hydro.cuh"
using namespace ek_fast;

__device__ unsigned g_bad[2];

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

int
main()
{
  floors<<<1, 1>>>();
  nans<<<1, 1>>>();
  unsigned h[2];
  if (cudaMemcpyFromSymbol(h, g_bad, sizeof h) != cudaSuccess)
    return 1;
  printf("floors %u\nnan %u\n", h[0], h[1]);
  return 0;
}
