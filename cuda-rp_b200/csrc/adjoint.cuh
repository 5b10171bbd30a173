// Discrete adjoint of the FDTD/PML step without bubbles (crp_adjoint).
//
// Without bubbles the step is linear in the fields (f_g = 0, rho_m = rho_inf):
//   faces       v'(f) = (v(f) A(f) - q (p0(f+1) - p0(f)) rdx) B(f)     (zeroed walls excepted)
//   components  px'(c) = px(c) a(c) - s3p b(c) (k_e(c) vx'(c) - k_w(c) vx'(c-1)),  py' likewise
//   p0          p0 = px + py inside, 0 on PML ghost cells, the source value on
//               the source row, the mirror of row 1 on the y0 ghost row
// with the factors of velocity_face_q / pressure_component (A, a = 1 - s;
// B, b = 1 / (1 + s); q = dt / rho_inf).  One reverse step applies the
// transposes in the opposite order: the pressure update's transpose takes the
// face adjoints L to Lt, then the velocity update's and p0's transposes take
// Lt and the component adjoints M one step back, and the source's share of the
// p0 adjoint times the source's derivatives with respect to the element
// amplitudes and phases goes into per-column gradient sums.  The objective
// sum_n dt sum_focal w p0^2 adds 2 dt w p0^n to both component adjoints at
// every step, from the focal pressures the forward recorded (adj_record).
//
// adj_march does all of one reverse step in one pass, organised as fdtd_march: a
// warp covers 64 columns, two per lane, and marches up a few rows.  A lane forms the
// Lt of the three x faces and the north faces of its columns from the previous step's
// L and M (the faces shared with other lanes twice, by the same expression; the south
// faces are the north faces of the row below) and writes the next step's L and M into
// the other of two frame sets.  The column coefficients stay in registers over the
// chunk's rows, and the source's derivatives come from a table (source_derivative_rows),
// so the pass carries no transcendental code.  Per cell and step it reads 4 doubles
// (L_x, L_y, M_x, M_y; the neighbours' values come through L1/L2) and writes 4: 64 bytes.
// Bound by the latency of the loads at 16 warps per SM: 600 x 701 takes 11.6 us cold
// (27 MB: 2.3 TB/s).  A call of 300 steps there took 8.2 ms with one cell per
// thread, each reading the coefficients of its row and column again and evaluating
// the source's derivatives where the source row lies, 7.5 with this pass, 6.4 since the
// FDTD pass records the focal pressures, and 5.2 with 3 rows per chunk instead of 2.
#pragma once
#include "crp_device.cuh"

namespace crp {

// One set of adjoint fields (two alternate over the reverse sweep).
struct AdjFrames {
  double* LX;  // adjoint of the x faces
  double* LY;  // adjoint of the y faces
  double* MX;  // adjoint of px
  double* MY;  // adjoint of py
};
// Per column: d J / d (its element's amplitude factor), d J / d (its phase offset).
struct AdjGrad {
  double* gA;
  double* gP;
};

// Faces the forward updates (the others are set to zero): the x0 axis and the
// x1 and y1 walls without a PML.  The y0 face without a PML keeps its update
// when the source is a pressure source, the only kind supported here.
__device__ __forceinline__ bool adj_xface_on(const GridParams& g, int f) {
  return !((f == 0 && !g.pml_x0) || (f == g.f.X && !g.pml_x1));
}
__device__ __forceinline__ bool adj_yface_on(const GridParams& g, int f) { return !(f == g.f.Y && !g.pml_y1); }
// d v'(f) / d p0(f) of a face (-d v'(f) / d p0(f+1)), and d v'(f) / d v(f).
__device__ __forceinline__ double adj_cx(const GridParams& g, int f) { return g.dt_rho * g.rdx * g.vbx[f + 1]; }
__device__ __forceinline__ double adj_cy(const GridParams& g, int f) { return g.dt_rho * g.rdx * g.vby[f + 1]; }
__device__ __forceinline__ double adj_ax(const GridParams& g, int f) { return g.vax[f + 1] * g.vbx[f + 1]; }
__device__ __forceinline__ double adj_ay(const GridParams& g, int f) { return g.vay[f + 1] * g.vby[f + 1]; }
// Weights of the east and west faces in the x divergence of cell c.
__device__ __forceinline__ double adj_kx_east(const GridParams& g, int c) {
  return g.cyl ? g.xu[c + 1] * g.rdx * g.rxp[c] : g.rdx;
}
__device__ __forceinline__ double adj_kx_west(const GridParams& g, int c) {
  return g.cyl ? g.xu[c] * g.rdx * g.rxp[c] : g.rdx;
}

// Focal box: cells [bi0, bi0 + bw) x [bj0, bj0 + bh), weights w (0 outside
// the focal disk and on the source row).
struct FocalBox {
  int bi0, bj0, bw, bh;
  const double* w;
};

// Derivatives of the source's row (source_derivatives) at the times of up to
// kDerivBatch reverse steps: rows of X + 2 values, d / d amplitude then d / d phase of
// each step.
constexpr int kDerivBatch = 32;
struct DerivTimes {
  double t[kDerivBatch];
};
__global__ void __launch_bounds__(64) source_derivative_rows(const __grid_constant__ GridParams g,
                                                             const __grid_constant__ DerivTimes d, double* out) {
  const int i = blockIdx.x * 64 + threadIdx.x, w = g.f.X + 2;
  if (i < 1 || i > g.f.X) return;
  double dA, dP;
  source_derivatives(g, ((double)i - 0.5) * g.dx, ((double)g.source_row - 0.5) * g.dy, d.t[blockIdx.y], dA, dP);
  out[(2 * (size_t)blockIdx.y) * w + i] = dA;
  out[(2 * (size_t)blockIdx.y + 1) * w + i] = dP;
}

constexpr int kAdjWarps = 4, kAdjMinBlocks = 4;

// One reverse step: the transposes of the pressure update, the velocity update
// and p0, from `in` into `out`; dA, dP: the source derivatives of the values that the
// step read (null without elements).  p0 (the focal pressures of the step before, or
// null for the first step) adds that step's objective term.
__global__ void __launch_bounds__(32 * kAdjWarps, kAdjMinBlocks) adj_march(const __grid_constant__ GridParams g,
                                                               const AdjFrames in, const AdjFrames out, const AdjGrad gr,
                                                               const double* __restrict__ dA,
                                                               const double* __restrict__ dP, const FocalBox b,
                                                               const double* __restrict__ p0, int rows, int strips) {
  const Frame& f = g.f;
  const int X = f.X, Y = f.Y;
  const int i = 1 + (blockIdx.x % strips) * 64 + 2 * (threadIdx.x & 31);
  const int j0 = 1 + ((blockIdx.x / strips) * kAdjWarps + (threadIdx.x >> 5)) * rows, j1 = min(Y, j0 + rows - 1);
  if (i > X || j0 > Y) return;
  const bool two = i + 1 <= X;
  const unsigned pitch = (unsigned)f.pitch;
  auto get2 = [](const double* p, unsigned k) { return *reinterpret_cast<const double2*>(p + k); };
  // Column coefficients of the faces i - 1, i, i + 1: the pressure update's weights of
  // the cells west (cw) and east (ce) of the face, d v' / d p0, and d v' / d v.
  double cw[3], ce[3], cx[3], ax[3];
  bool on[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const int q = min(i - 1 + c, X);
    on[c] = adj_xface_on(g, q);
    cw[c] = q >= 1 ? g.s3p * g.pbx[q] * adj_kx_east(g, q) : 0.0;
    ce[c] = q + 1 <= X ? g.s3p * g.pbx[q + 1] * adj_kx_west(g, q + 1) : 0.0;
    cx[c] = adj_cx(g, q);
    ax[c] = adj_ax(g, q);
  }
  const double pax[2] = {g.pax[i], g.pax[min(i + 1, X)]};
  unsigned k = (unsigned)(j0 + 1) * pitch + (unsigned)(i + 1);
  // Lt of the south faces (adj_lyt of row j0 - 1).
  double ys[2];
  double2 my = get2(in.MY, k);
  {
    const double2 l = get2(in.LY, k - pitch), m = get2(in.MY, k - pitch);
    const double lv[2] = {l.x, l.y}, mb[2] = {m.x, m.y}, mc[2] = {my.x, my.y};
    const double wb = j0 >= 2 ? g.s3p * g.pby[j0 - 1] * g.rdy : 0.0, wt = g.s3p * g.pby[j0] * g.rdy;
#pragma unroll
    for (int c = 0; c < 2; c++) {
      ys[c] = lv[c];
      if (j0 >= 2) ys[c] = fma(-wb, mb[c], ys[c]);
      ys[c] = fma(wt, mc[c], ys[c]);
    }
  }
  for (int j = j0; j <= j1; j++, k += pitch) {
    const double2 lx = get2(in.LX, k), ly = get2(in.LY, k), mx = get2(in.MX, k), mn = get2(in.MY, k + pitch);
    const double lw = in.LX[k - 1], mw = in.MX[k - 1], me = in.MX[k + 2];
    const double m4[4] = {mw, mx.x, mx.y, me}, l3[3] = {lw, lx.x, lx.y};
    double xt[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      double v = l3[c];
      if (i - 1 + c >= 1) v = fma(-cw[c], m4[c], v);
      if (i + c <= X) v = fma(ce[c], m4[c + 1], v);
      xt[c] = v;
    }
    const double wb = g.s3p * g.pby[j] * g.rdy, wt = j + 1 <= Y ? g.s3p * g.pby[j + 1] * g.rdy : 0.0;
    const double cyn = adj_cy(g, j), cys = adj_cy(g, j - 1), ayn = adj_ay(g, j), pay = g.pay[j];
    const bool on_n = adj_yface_on(g, j), on_s = adj_yface_on(g, j - 1);
    const double lyv[2] = {ly.x, ly.y}, myv[2] = {my.x, my.y}, mnv[2] = {mn.x, mn.y};
    double yn[2], nmx[2], nmy[2];
#pragma unroll
    for (int c = 0; c < 2; c++) {
      yn[c] = fma(-wb, myv[c], lyv[c]);
      if (j + 1 <= Y) yn[c] = fma(wt, mnv[c], yn[c]);
      // Adjoint of p0(i + c, j): the faces that read it.
      double L0 = 0.0;
      if (on[c + 1]) L0 = fma(cx[c + 1], xt[c + 1], L0);
      if (on[c]) L0 = fma(-cx[c], xt[c], L0);
      if (on_n) L0 = fma(cyn, yn[c], L0);
      if (on_s) L0 = fma(-cys, ys[c], L0);
      if (c == 1 && !two) break;
      const int col = i + c;
      if (j == 1 && !g.pml_y0) {
        // The y0 face also reads the ghost value p0(i, 0): the source on the ghost
        // row (source_row 0), else the mirror of p0(i, 1).
        const double m = __dmul_rn(adj_cy(g, 0), ys[c]);
        if (g.source_row == 0) {
          if (dA) {
            gr.gA[col] += m * dA[col];
            gr.gP[col] += m * dP[col];
          }
        } else {
          L0 += m;
        }
      }
      double ux = m4[c + 1], uy = myv[c];
      if (g.source_row > 0 && j == g.source_row) {
        if (dA) {
          gr.gA[col] += L0 * dA[col];
          gr.gP[col] += L0 * dP[col];
        }
      } else {
        ux = fma(pax[c], ux, L0);
        uy = fma(pay, uy, L0);
      }
      if (p0) {  // d J / d p0 of the step before: M += 2 dt w p0 on the focal box
        const int bi = col - b.bi0, bj = j - b.bj0;
        if (bi >= 0 && bi < b.bw && bj >= 0 && bj < b.bh) {
          const int q = bj * b.bw + bi;
          const double v = __dmul_rn(2.0 * g.dt * b.w[q], p0[q]);
          ux += v;
          uy += v;
        }
      }
      nmx[c] = ux;
      nmy[c] = uy;
    }
    // Face adjoints one step back (each cell takes its east and north faces; the
    // first column and row also the x0 and y0 faces).
    const double fx[2] = {on[1] ? ax[1] * xt[1] : 0.0, on[2] ? ax[2] * xt[2] : 0.0};
    const double fy[2] = {on_n ? ayn * yn[0] : 0.0, on_n ? ayn * yn[1] : 0.0};
    auto put = [&](double* q, double v, double w) {
      if (two)
        *reinterpret_cast<double2*>(q + k) = make_double2(v, w);
      else
        q[k] = v;
    };
    put(out.MX, nmx[0], nmx[1]);
    put(out.MY, nmy[0], nmy[1]);
    put(out.LX, fx[0], fx[1]);
    put(out.LY, fy[0], fy[1]);
    if (i == 1) out.LX[k - 1] = on[0] ? ax[0] * xt[0] : 0.0;
    if (j == 1) {
      out.LY[k - pitch] = adj_ay(g, 0) * ys[0];
      if (two) out.LY[k - pitch + 1] = adj_ay(g, 0) * ys[1];
    }
    ys[0] = yn[0];
    ys[1] = yn[1];
    my = mn;
  }
}

// p0 of the focal box after a forward step (interior cells: px + py).
template <typename S>
__global__ void adj_record(const __grid_constant__ GridParams g, const S px, const S py, const FocalBox b,
                           double* __restrict__ out) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= b.bw * b.bh) return;
  const long k = g.f.idx(b.bi0 + q % b.bw, b.bj0 + q / b.bw);
  out[q] = px.get(k) + py.get(k);
}

// d J / d p0 of the last step: MX, MY += 2 dt w p0 (the earlier steps' terms
// are added by adj_march).
__global__ void adj_force(const __grid_constant__ GridParams g, const AdjFrames a, const FocalBox b,
                          const double* __restrict__ p0) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= b.bw * b.bh) return;
  const long k = g.f.idx(b.bi0 + q % b.bw, b.bj0 + q / b.bw);
  const double v = 2.0 * g.dt * b.w[q] * p0[q];
  a.MX[k] += v;
  a.MY[k] += v;
}

// sum_focal w p0^2 of every recorded step (one block per step, fixed order).
constexpr int kAdjSumThreads = 256;
__global__ void __launch_bounds__(kAdjSumThreads) adj_objective(const FocalBox b, const double* __restrict__ hist,
                                                                double* __restrict__ Jn) {
  __shared__ double sh[kAdjSumThreads];
  const int cells = b.bw * b.bh;
  const double* p = hist + (long)blockIdx.x * cells;
  double s = 0.0;
  for (int q = threadIdx.x; q < cells; q += kAdjSumThreads) s += b.w[q] * p[q] * p[q];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = kAdjSumThreads / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) Jn[blockIdx.x] = sh[0];
}

}  // namespace crp
