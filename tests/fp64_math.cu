// FP64 helpers of the FMA build against CUDA's own functions, for
// test_gpu_fp64_math.py: prints the largest errors in units of 2^-53.
#include <cmath>
#include <cstdio>
#include "ek_hydro.cuh"
using namespace ek_fast;

__device__ double g_out[64];

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
at_most(int k, double e)
{
  atomicMax((unsigned long long *)&g_out[k], (unsigned long long)__double_as_longlong(e * 0x1p53));
}

__global__ void
errors(int spread)
{
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  for (int i = 0; i < 64; ++i)
  {
    const unsigned long long z = mix(t * 64ull + i + 1);
    const double x = value(z, spread), n = value(mix(z), spread / 2), d = value(mix(z + 1), spread / 2);
    // residuals by FMA: 1 - x y, (1 - x y^2) / 2, (x - s^2) / 2x
    at_most(0, fabs(fma(-x, rcp64(x), 1.0)));
    const double q = rsqrt64(x), h = q * q, l = fma(q, q, -h);
    at_most(1, 0.5 * fabs(fma(-x, l, fma(-x, h, 1.0))));
    const double s = sqrt64(x);
    at_most(2, 0.5 * fabs(fma(-s, s, x)) / x);
    at_most(3, fabs(sqrt_ratio64(n, d) / sqrt(n / d) - 1.0));
    // scaling and slopes are exact: any difference counts as 2^53
    const double a = flip64(n, z & 1), b = flip64(d, z & 2), c = flip64(value(mix(z + 2), spread / 2), z & 4);
    at_most(4, half64(a) == 0.5 * a && scale_pos64<2>(d) == 0.25 * d && abs64(a) == fabs(a) ? 0.0 : 1.0);
    for (int st = 0; st < 3; ++st)
    {
      const double dl = st * (a - b), dr = st * (c - a), dc = 0.5 * (c - b);
      const double m = dl * dr <= 0.0 ? 0.0 : fmin(fmin(fabs(dl), fabs(dr)), fabs(dc));
      at_most(5, half_slope64(a, c, b, st) == 0.5 * (dc >= 0.0 ? m : -m) ? 0.0 : 1.0);
    }
    at_most(6, max_floor64(a, d) == fmax(a, d) && min_pos64(n, d) == fmin(n, d) &&
                 floor_ratio64(a, d, x * 1e-3) == fmax(a, d * (x * 1e-3)) && max_cand64(a, d) == fmax(a, d)
                 ? 0.0 : 1.0);
  }
}
__global__ void
specials()
{
  const double inf = INFINITY;
  const bool   ok = rcp64(0.0) == inf && rcp64(-0.0) == -inf && rcp64(inf) == 0.0 && isnan(rcp64(NAN)) &&
                  rsqrt64(0.0) == inf && rsqrt64(inf) == 0.0 && isnan(rsqrt64(-1.0)) && isnan(rsqrt64(NAN)) &&
                  sqrt64(0.0) == 0.0 && sqrt64(inf) == inf && isnan(sqrt64(-1.0)) && isnan(sqrt64(NAN)) &&
                  sqrt_ratio64(0.0, 2.0) == 0.0 && isnan(sqrt_ratio64(NAN, 1.0)) && isnan(half64(NAN)) &&
                  half64(inf) == inf && half64(-0.0) == 0.0 && half64(5e-324) == 0.0 && half64(-3e-308) == -1.5e-308 &&
                  scale_pos64<2>(0.0) == 0.0 &&
                  max_cand64(1.0, NAN) == 1.0 && max_cand64(-inf, 2.0) == 2.0 && floor_ratio64(-3.0, 8.0, 1e-20) == 8e-20;
  g_out[7] = ok ? 0.0 : 1.0;
}

int
main(int, char ** argv)
{
  errors<<<64, 256>>>(atoi(argv[1]));
  specials<<<1, 1>>>();
  double h[8];
  if (cudaMemcpyFromSymbol(h, g_out, sizeof h) != cudaSuccess)
    return 1;
  for (int k = 0; k < 8; ++k)
    printf("%.17g\n", h[k]);
  return 0;
}
