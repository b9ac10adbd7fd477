// The mixed form's FP32 HLLD flux and 2D HLLD emf against the FP64 ones, over
// densities of 1e-20 to 1e15, sound speeds of 1e-3 to 1e3 and fields down to
// 1e-32, for test_gpu_mhd_weak_field.py: prints the largest errors (relative to
// the states' own scales; a NaN or an infinity counts as 1e30) and the number
// of faces solved.
#include <cmath>
#include <cstdio>
#include "ek_mhd.cuh"
using namespace ek_fast;

__device__ unsigned g_out[2];
__device__ unsigned long long g_faces;

// SplitMix64's finaliser
__device__ unsigned long long
mix(unsigned long long z)
{
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
struct Rng
{
  unsigned long long s;
  __device__ double
  operator()(double lo, double hi) // uniform
  {
    s += 0x9E3779B97F4A7C15ull;
    return lo + (hi - lo) * ((mix(s) >> 11) * 0x1p-53);
  }
};
__device__ void
at_most(int k, double e)
{
  const float f = e < 1e30 ? (float)e : 1e30f; // NaN too
  atomicMax(&g_out[k], __float_as_uint(f));
}

__global__ void
errors()
{
  Rng          g{ mix(blockIdx.x * blockDim.x + threadIdx.x + 1) };
  const double gamma = 5.0 / 3.0, entho = 1.0 / (gamma - 1.0), smallc = 1e-10;
  for (int it = 0; it < 64; ++it)
  {
    const double c = exp10(g(-3.0, 3.0)), rho = exp10(g(-20.0, 15.0)), p = rho * c * c / gamma;
    // from a field as strong as the pressure down to the weakest whose products with rho c^2, rho^(1/2) and c^3 (the
    // star states, the mean of two stars, the emf's wave speeds) are numbers of FP32, or none
    const double bmax = 0.5 * sqrt(p), bmin = fmax(fmax(1e-32 / (rho * c * c), 1e-32 / sqrt(rho)), 1e-26 / (c * c * c));
    const double b = bmin > bmax || g(0.0, 1.0) < 0.1 ? 0.0 : bmax * pow(bmin / bmax, g(0.0, 1.0));
    auto         one = [&](double x) { return (double)(float)(x * g(0.7, 1.3)); };
    auto         vel = [&]() { return (double)(float)(c * g(-0.4, 0.4)); };
    auto         sgn = [&](double x) { return (double)(float)(x * g(-1.0, 1.0)); };
    // corner: a along a row, b along a column
    const double a0 = sgn(b), a1 = sgn(b), b0 = sgn(b), b1 = sgn(b);
    EdgeQ<double> d[4];
    EdgeQ<float>  f[4];
    const double  da[4] = { a0, a0, a1, a1 }, db[4] = { b0, b1, b0, b1 }; // LL, RL, LR, RR
    for (int q = 0; q < 4; ++q)
    {
      d[q].r = one(rho), d[q].p = one(p), d[q].u = vel(), d[q].v = vel(), d[q].c = sgn(b);
      d[q].a = da[q], d[q].b = db[q];
      f[q].r = d[q].r, f[q].p = d[q].p, f[q].u = d[q].u, f[q].v = d[q].v, f[q].a = d[q].a, f[q].b = d[q].b, f[q].c = d[q].c;
    }
    const double E = mag_riemann2d_hlld64(d[0], d[1], d[2], d[3], gamma, smallc);
    const float  e = mag_riemann2d_hlld_f32(f[0], f[1], f[2], f[3], (float)gamma, (float)smallc);
    if (b > 0.0)
      at_most(0, fabs((double)e - E) / (2.0 * c * b));
    else
      at_most(0, e == 0.f ? 0.0 : INFINITY);
    // face
    double ql[8], qr[8], F[6];
    float  sl[8], sr[8], h[6];
    for (int v = 0; v < 8; ++v)
    {
      ql[v] = v == ID ? one(rho) : v == IP ? one(p) : v < IA ? vel() : sgn(b);
      qr[v] = v == ID ? one(rho) : v == IP ? one(p) : v < IA ? vel() : sgn(b);
    }
    qr[IA] = ql[IA];
    for (int v = 0; v < 8; ++v)
      sl[v] = ql[v], sr[v] = qr[v];
    mhd_hlld64<6>(ql, qr, F, gamma, entho);
    if (!mhd_hlld_f32<6>(sl, sr, h, (float)gamma, (float)entho))
      continue;
    atomicAdd(&g_faces, 1ull);
    for (int v = 0; v < 6; ++v)
    {
      // (the field between the two Alfven waves is up to rho^(1/2) times the jump of w, however weak b is)
      const double scale = v == ID ? rho * c : v == IP ? rho * c * c * c : v < IA ? rho * c * c : c * (b + sqrt(rho) * c);
      at_most(1, fabs((double)h[v] - F[v]) / (2.0 * scale));
    }
  }
}

int
main()
{
  errors<<<64, 256>>>();
  unsigned           o[2];
  unsigned long long n = 0;
  if (cudaMemcpyFromSymbol(o, g_out, sizeof o) != cudaSuccess || cudaMemcpyFromSymbol(&n, g_faces, sizeof n) != cudaSuccess)
    return 1;
  for (unsigned x : o)
  {
    float f;
    memcpy(&f, &x, sizeof f);
    printf("%.9g\n", f);
  }
  printf("%llu\n", n);
  return 0;
}
