// Check program for grhd::root_safe_newton (physics.cuh), built and run by
// tests/test_gpu_root.py: the screened root finder against the plain iteration of
// equations.f90:249-340 (restated here with every residual in FP64), bit for bit, on seeded
// conserved states.  Prints, per family of states, the samples, the differing roots and
// flags, and the FP64 residuals per root of the plain iteration.
#include <cstdio>

#include <math_constants.h>

#include "common.cuh"

using namespace grhd;

__device__ unsigned long long g_tests, g_bad, g_evals;

__device__ double plain(double g1, double rho_floor, double D, double tau, double Q2, unsigned &flags, int &n) {
  double f_low, f_high, df, f, xl, xh;
  residual(g1, 1.0, D, tau, Q2, f_low, df);
  const double x2 = rmax(1.0e3, (sqrt(Q2) + D) / rmax(D, rho_floor) * 2.0);
  residual(g1, x2, D, tau, Q2, f_high, df);
  n = 2;
  if (fabs(f_low) < 1.0e-14) return 1.0;
  if (fabs(f_high) < 1.0e-14) return x2;
  if (sgn1(f_low) * sgn1(f_high) > 0.0) return -1.0;
  if (f_low < 0.0) { xl = 1.0; xh = x2; } else { xh = 1.0; xl = x2; }
  double root = 0.5 * (1.0 + x2), dxo = fabs(x2 - 1.0), dx = dxo;
  residual(g1, root, D, tau, Q2, f, df);
  ++n;
  for (int it = 0; it < 100; ++it) {
    if (((root - xh) * df - f) * ((root - xl) * df - f) > 0.0 || fabs(2.0 * f) > fabs(dxo * df)) {
      dxo = dx;
      dx = 0.5 * (xh - xl);
      root = xl + dx;
      if (fabs(xl - root) < 1.0e-14) return root;
    } else {
      dxo = dx;
      dx = f / df;
      const double t = root;
      root = root - dx;
      if (fabs(t - root) < 1.0e-14) return root;
    }
    if (fabs(dx) < 1.0e-10) return root;
    residual(g1, root, D, tau, Q2, f, df);
    ++n;
    if (f < 0.0) xl = root; else xh = root;
  }
  flags |= C2P_BRENT;
  return root_brent(g1, rho_floor, D, tau, Q2);
}

__device__ __forceinline__ unsigned long long mix(unsigned long long h) {
  h ^= h >> 30; h *= 0xbf58476d1ce4e5b9ULL;
  h ^= h >> 27; h *= 0x94d049bb133111ebULL;
  return h ^ (h >> 31);
}

// kind 0: states of rho, p, v (densities over 40 binades, v up to 1 - 1e-5); 1: the same with
// every conserved value off by up to 3 (no physical state behind it); 2: near the tests'
// edges (Q2 ~ 1e-14, E ~ 1e-12 and 1e12, D ~ 1.25 E); 3: zeros, negative and infinite values; 4: E < 0
__global__ void check(long long n, unsigned long long seed, int kind) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= n) return;
  unsigned long long h = mix((unsigned long long)t + seed);
  auto u = [&]() { h = mix(h); return (double)(h >> 11) * 0x1p-53; };
  const double adbs[4] = {4.0 / 3.0, 5.0 / 3.0, 2.0, 3.0};
  const double adb = adbs[h & 3], g1 = adb / (adb - 1.0);
  const double rho = exp2(-34.0 + 40.0 * u()), p = rho * exp2(-30.0 + 40.0 * u());
  const double v = u() < 0.5 ? u() : 1.0 - exp2(-17.0 * u()), s2 = fmin(v * v, 1.0 - 1e-5), W = 1.0 / sqrt(1.0 - s2);
  const double rhW2 = (rho + g1 * p) * W * W, sq = exp2(12.0 * u() - 2.0);
  double D = rho * W * sq, tau = (rhW2 - p) * sq - D, Q2 = rhW2 * rhW2 * s2 * sq * sq;
  if (kind == 1) { D *= 1.0 + 2.0 * u(); tau *= 1.0 + 2.0 * (u() - 0.5); Q2 *= 1.0 + 2.0 * (u() - 0.5); }
  if (kind == 2) {
    const double e = u() < 0.5 ? 1e-12 : 1e12, x = exp2(0.01 * (u() - 0.5));
    if (u() < 0.3) Q2 = 1e-14 * x;
    if (u() < 0.3) { const double k = e * x / (D + tau); D *= k; tau *= k; Q2 *= k * k; }
    if (u() < 0.3) tau = -0.2 * D * x;
    if (u() < 0.3) Q2 = (tau + D) * (tau + D) * (1.0 + exp2(-20.0 * u()) * (u() - 0.5));
  }
  if (kind == 3) {
    const double odd[8] = {0.0, -1.0, 1e-300, 1e300, CUDART_INF, -CUDART_INF, 1e-14, -1e-20};
    if (u() < 0.5) D = odd[mix(h) & 7];
    if (u() < 0.5) tau = odd[(mix(h) >> 8) & 7];
    if (u() < 0.5) Q2 = odd[(mix(h) >> 16) & 7];
  }
  if (kind == 4) {  // E = tau + D < 0
    tau = -D * (1.0 + (u() < 0.5 ? 4.0 * u() : exp2(-20.0 * u())));
    Q2 = fmax(0.0, (tau + D) * (tau + D) - (u() < 0.5 ? D * D : 0.0)) * u();
  }
  unsigned fa = 0, fb = 0;
  int ne = 0;
  const double a = root_safe_newton(g1, 1.0e-10, D, tau, Q2, fa), b = plain(g1, 1.0e-10, D, tau, Q2, fb, ne);
  atomicAdd(&g_tests, 1ull);
  atomicAdd(&g_evals, (unsigned long long)ne);
  const bool same = __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b);
  if (!same || fa != fb) atomicAdd(&g_bad, 1ull);
}

int main() {
  const long long n = 1LL << 23;
  for (int kind = 0; kind < 5; ++kind) {
    unsigned long long c[3], z = 0;
    cudaMemcpyToSymbol(g_tests, &z, 8);
    cudaMemcpyToSymbol(g_bad, &z, 8);
    cudaMemcpyToSymbol(g_evals, &z, 8);
    check<<<(unsigned)(n / 256), 256>>>(n, 0x2545f491ULL * (kind + 1), kind);
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) { printf("error %s\n", cudaGetErrorString(e)); return 1; }
    cudaMemcpyFromSymbol(&c[0], g_tests, 8);
    cudaMemcpyFromSymbol(&c[1], g_bad, 8);
    cudaMemcpyFromSymbol(&c[2], g_evals, 8);
    printf("kind %d samples %llu bad %llu plain residuals per root %.2f\n", kind, c[0], c[1], (double)c[2] / (double)c[0]);
  }
  return 0;
}
