// The branch-free operations of the flux functions (Fast64) and what is built on them, on arrays: as a
// kernel (nvcc, the seeds of the GPU) or on the host (g++, seeds of 20 leading bits from a table of
// roundings).  Each item gives the branch-free value, the plain operators' and the bad() flag.
#include <math.h>
#include <stdint.h>
#include <string.h>
#ifdef __CUDACC__
#include <cuda_runtime.h>
#define RUN __device__
#else
#include <algorithm>
#define RUN static
static inline int64_t __double_as_longlong(double x) { int64_t i; memcpy(&i, &x, 8); return i; }
static inline double __longlong_as_double(int64_t i) { double x; memcpy(&x, &i, 8); return x; }
static inline int __double2hiint(double x) { return (int)(__double_as_longlong(x) >> 32); }
static inline int __double2loint(double x) { return (int)__double_as_longlong(x); }
static inline double __hiloint2double(int h, int l) {
  return __longlong_as_double((int64_t)(((uint64_t)(uint32_t)h << 32) | (uint32_t)l));
}
static inline unsigned min(unsigned a, unsigned b) { return std::min(a, b); }
static inline unsigned max(unsigned a, unsigned b) { return std::max(a, b); }
// Seeds: the operand's 20 leading mantissa bits, the result rounded to 20 bits (0 nearest, 1 down, 2 up).
static int g_round = 0;
static double seed_round(double x) {
  int e;
  const double m = ldexp(frexp(x, &e), 21);
  return ldexp(g_round == 1 ? floor(m) : g_round == 2 ? ceil(m) : nearbyint(m), e - 21);
}
static double lead(double x) { return __longlong_as_double(__double_as_longlong(x) & ~0xffffffffll); }
static double fast64_rcp_seed(double b) { return seed_round(1.0 / lead(b)); }
static double fast64_rsqrt_seed(double a) { return seed_round(1.0 / sqrt(lead(a))); }
#endif
#include "physics.cuh"

using namespace cfdb;

template <typename O>
RUN double op(O &o, int k, double a, double b) {
  switch (k) {
    case 0: return o.div(a, b);
    case 1: return o.div_signed(a, b);
    case 2: return o.inv(b);
    case 3: return o.root(b);
    case 4: return o.div_gm1(a);
    case 5: return O::fast ? Fast64::rcp_seed(b) : 1.0 / b;
    case 6: return O::fast ? Fast64::rsqrt_seed(b) : 1.0 / sqrt(b);
    default: return 0.0;
  }
}
RUN double slope(Fast64 &o, int kind, double a, double b) {
  if (kind == LIM_VANLEER) return muscl_half_slope<LIM_VANLEER>(o, a, b);
  if (kind == LIM_VANALBADA) return muscl_half_slope<LIM_VANALBADA>(o, a, b);
  return muscl_half_slope<LIM_MINMOD>(o, a, b);
}
// k 0 - 4: operations; 10 + limiter: half the limited slope of the gradient-MUSCL form.
RUN void item(int k, double a, double b, double *fast, double *plain, int *bad) {
  Fast64 f;
  Ieee<double> p;
  if (k >= 10) {
    *fast = slope(f, k - 10, a, b);
    *plain = 0.5 * muscl_slope<double>(k - 10, a, b);
  } else {
    *fast = op(f, k, a, b);
    *plain = op(p, k, a, b);
  }
  *bad = f.bad() ? 1 : 0;
}
// HLLC flux of primitive states q [8]: (rho, u, v, p) of both sides, normal and length n [3].
RUN void hllc(const double *q, const double *n, double *fast, double *plain, int *bad) {
  double qq[2][5], U[2][4];
  for (int s = 0; s < 2; s++) {
    const double r = q[4 * s], u = q[4 * s + 1], v = q[4 * s + 2], p = q[4 * s + 3];
    const double x[5] = {r, u, v, p, sqrt(kGamma * p / r)};
    const double c[4] = {r, r * u, r * v, p / kGM1 + 0.5 * r * (u * u + v * v)};
    for (int k = 0; k < 5; k++) qq[s][k] = x[k];
    for (int k = 0; k < 4; k++) U[s][k] = c[k];
  }
  Fast64 f;
  Ieee<double> p;
  hllc_face<double>(f, qq[0], U[0], qq[1], U[1], n[0], n[1], n[2], fast);
  hllc_face<double>(p, qq[0], U[0], qq[1], U[1], n[0], n[1], n[2], plain);
  *bad = f.bad() ? 1 : 0;
}

#ifdef __CUDACC__
__global__ void k_items(int k, int n, const double *a, const double *b, double *fast, double *plain, int *bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) item(k, a[i], b[i], fast + i, plain + i, bad + i);
}
extern "C" int ops_items(int k, int n, const double *a, const double *b, double *fast, double *plain, int *bad) {
  double *d = nullptr;
  int *db = nullptr;
  if (cudaMalloc(&d, 4 * sizeof(double) * n) != cudaSuccess || cudaMalloc(&db, sizeof(int) * n) != cudaSuccess) return 1;
  cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
  k_items<<<(n + 255) / 256, 256>>>(k, n, d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n, db);
  cudaMemcpy(fast, d + 2 * (size_t)n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(plain, d + 3 * (size_t)n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  const cudaError_t e = cudaMemcpy(bad, db, sizeof(int) * n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(db);
  return e == cudaSuccess ? 0 : 1;
}
#else
extern "C" void ops_seed_rounding(int r) { g_round = r; }
extern "C" int ops_items(int k, int n, const double *a, const double *b, double *fast, double *plain, int *bad) {
  for (int i = 0; i < n; i++) item(k, a[i], b[i], fast + i, plain + i, bad + i);
  return 0;
}
extern "C" int ops_hllc(int n, const double *q, const double *nrm, double *fast, double *plain, int *bad) {
  for (int i = 0; i < n; i++) hllc(q + 8 * i, nrm + 3 * i, fast + 4 * i, plain + 4 * i, bad + i);
  return 0;
}
#endif
