// Check program built and run by tests/test_gpu_root_edges.py: grhd::root_safe_newton (FP32
// screen) against grhd::root_reference (every residual in FP64), both of physics.cuh, bit for
// bit, on operands at the limits of the screen.  Prints, per family, samples and differing roots
// or flags.
#include <cstdio>

#include <math_constants.h>

#include "common.cuh"

using namespace grhd;

__device__ unsigned long long g_tests, g_bad;

__device__ __forceinline__ unsigned long long mix(unsigned long long h) {
  h ^= h >> 30; h *= 0xbf58476d1ce4e5b9ULL;
  h ^= h >> 27; h *= 0x94d049bb133111ebULL;
  return h ^ (h >> 31);
}

// kind 0: NaN of either sign among D, tau and Q2; 1: Q2 up to 1e10 E^2; 2: D / E around the
// limits +-1.25, where V^2 is largest; 3: nearly at rest, W - 1 from 1e-12 to 1e-1
__global__ void check(long long n, unsigned long long seed, int kind) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= n) return;
  unsigned long long h = mix((unsigned long long)t + seed);
  auto u = [&]() { h = mix(h); return (double)(h >> 11) * 0x1p-53; };
  const double adbs[4] = {4.0 / 3.0, 5.0 / 3.0, 2.0, 3.0};
  const double adb = adbs[h & 3];
  double g1 = adb / (adb - 1.0);
  const double E = exp2(80.0 * (u() - 0.5)), sgn = u() < 0.3 ? -1.0 : 1.0;
  double D = E * u(), tau = E - D, Q2 = E * E * u();
  if (kind == 0) {
    const double nan = u() < 0.5 ? CUDART_NAN : -CUDART_NAN;
    const int m = 1 + (int)(u() * 7.0);
    if (m & 1) D = nan;
    if (m & 2) tau = nan;
    if (m & 4) Q2 = nan;
  }
  if (kind == 1) Q2 = E * E * exp2(34.0 * u() - 1.0);
  if (kind == 2) {
    if (u() < 0.3) g1 = 1.9 + 1e-3 * (u() - 0.5);
    D = sgn * E * 1.25 * (1.0 + 1e-6 * (u() - 0.5)) * (u() < 0.5 ? 1.0 : -1.0);
    tau = sgn * E - D;
    Q2 = E * E * u() * 2.5;
  }
  if (kind == 3) {
    const double y = exp2(-40.0 + 37.0 * u()), W = 1.0 + y, V = (g1 * W * W * E - D * W) / (g1 * W * W - 1.0);
    Q2 = V * V * (y * (2.0 + y) / (W * W));
  }
  unsigned fa = 0, fb = 0;
  const double a = root_safe_newton(g1, 1.0e-10, D, tau, Q2, fa), b = root_reference(g1, 1.0e-10, D, tau, Q2, fb);
  atomicAdd(&g_tests, 1ull);
  const bool same = __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b);
  if (!same || fa != fb) atomicAdd(&g_bad, 1ull);
}

int main() {
  const long long n = 1LL << 22;
  for (int kind = 0; kind < 4; ++kind) {
    unsigned long long c[2], z = 0;
    cudaMemcpyToSymbol(g_tests, &z, 8);
    cudaMemcpyToSymbol(g_bad, &z, 8);
    check<<<(unsigned)(n / 256), 256>>>(n, 0x9e3779b9ULL * (kind + 1), kind);
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) { printf("error %s\n", cudaGetErrorString(e)); return 1; }
    cudaMemcpyFromSymbol(&c[0], g_tests, 8);
    cudaMemcpyFromSymbol(&c[1], g_bad, 8);
    printf("kind %d samples %llu bad %llu\n", kind, c[0], c[1]);
  }
  return 0;
}
