// Device functions of the radius solve behind plain C entry points, for the unit tests.
#include <cuda_runtime.h>

#include "crp_device.cuh"
#include "radius.cuh"

namespace {

using namespace crp;

// n bubbles of rest radius 3 um from rest with liquid pressure and wall velocity pl[i]
// and v[i] added, over ten sub-steps: out[2 i] whether the solve failed, then its sub-steps.
template <bool TIGHT, typename T, int FORM>
__global__ void solve(const BubbleParams bp, int n, const double* pl, const double* v, int* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  RpState<T, FORM> s;
  const double R0 = 3e-6;
  radius_const(bp, R0, s);
  s.Rt = s.Rp = s.Rn = R0;
  s.d1Rp = v[i];
  s.PGp = bp.PL0 + 2.0 * bp.sig / R0;
  s.dtL = bp.dt0;
  s.re_n = 0.0;
  s.remain = 10.0 * bp.dt0;
  s.time = 0.0;
  s.PC0 = bp.PL0 + pl[i];
  s.PC1 = s.PC2 = s.heat = s.vis = 0.0;
  s.count = 0;
  while (rp_more(bp, s)) rp_substep_full<TIGHT>(bp, s);
  out[2 * i] = rp_failed(s) ? 1 : 0;
  out[2 * i + 1] = s.count;
}

// recip(b), quotient(a, b), rsqrt_pos(b), sqrt_pos(b), rroot4_pos(b), then the operators'
// 1 / b, a / b, sqrt(b): rows of n values each.
__global__ void helpers(int n, const double* a, const double* b, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = b[i];
  const double v[8] = {recip(x),      quotient(a[i], x), rsqrt_pos(x), sqrt_pos(x),
                       rroot4_pos(x), 1.0 / x,           a[i] / x,     sqrt(x)};
  for (int q = 0; q < 8; q++) out[(size_t)q * n + i] = v[q];
}

}  // namespace

extern "C" int units_helpers(int n, const double* a, const double* b, double* out) {
  double* d = nullptr;
  cudaError_t e = cudaMalloc(&d, 10 * sizeof(double) * n);
  if (e == cudaSuccess) e = cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    helpers<<<(n + 255) / 256, 256>>>(n, d, d + n, d + 2 * (size_t)n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * (size_t)n, 8 * sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}

// form: 0 quiet lean, 1 lean for stiff launches, 2 lean of the mixed path, 3 with heat.
extern "C" int units_solve(int form, int cap, int n, const double* pl, const double* v, int* out) {
  BubbleParams bp{};
  bp.PL0 = 101325.0, bp.T0 = 293.15, bp.gam = 1.4, bp.sig = 0.0725, bp.mu = 1e-3, bp.rho = 998.0, bp.K0 = 26.2e-3;
  bp.dt0 = 1e-9, bp.pi = 3.14159265358979323846, bp.step_cap = cap;
  derive_bubble_constants(bp);
  double* d = nullptr;
  int* o = nullptr;
  cudaError_t e = cudaMalloc(&d, 2 * sizeof(double) * n);
  if (e == cudaSuccess) e = cudaMalloc(&o, 2 * sizeof(int) * n);
  if (e == cudaSuccess) e = cudaMemcpy(d, pl, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, v, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    const int blocks = (n + 63) / 64;
    if (form == 0) solve<false, double, kLean><<<blocks, 64>>>(bp, n, d, d + n, o);
    if (form == 1) solve<true, double, kLean><<<blocks, 64>>>(bp, n, d, d + n, o);
    if (form == 2) solve<false, float, kLean><<<blocks, 64>>>(bp, n, d, d + n, o);
    if (form == 3) solve<false, double, kHeat><<<blocks, 64>>>(bp, n, d, d + n, o);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, o, 2 * sizeof(int) * n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(o);
  return (int)e;
}
