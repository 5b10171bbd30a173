// The 3-D Cartesian simulation (ext.grid_z > 0): the same bubbly-mixture
// model as the 2-D path on a staggered grid of X x Y x Z cells, with a PML on
// all six faces and a hemispherical phased array as its source.  The
// reference is 2-D only; each of its formulas gains its third component:
// VelocityKernel and MixturePressureKernel (inc/bubble_CUDA_kernel.cuh:635-677,
// 816-867) for vz and pz, init_sigma's profiles per axis, the smooth delta
// (:214-222) and the bubble stencils (:361-448, :576-619) over 2 x 2 x 2
// cells.  oracle/oracle3d.inc restates every step on the host.
//
// Kernels of one mixture step:
//   fdtd3        fused velocity update (three faces per cell), void-fraction
//                prediction, split-pressure update, source forcing and
//                residual; warps of 64 columns march along z, the face below
//                in registers: one pass over the state
//   move3        bubble state rotation, velocity gather over the staggered
//                2 x 2 x 2 stencils, motion, cell indices, bounding box
//   bin3_*       counting sort of bubbles by cell (when a bubble changed cell)
//   rp3 / rk3    pressure gather + radius solve (reference scheme or rk45) +
//                the eight void-fraction contributions of each bubble,
//                persistent with a work queue
//   couple3      per-cell gather of the void fraction from its eight bins,
//                pressure re-evaluation, source forcing, residual, over the
//                box where the void fraction can be nonzero
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "crp.h"
#include "crp_device.cuh"
#include "radius.cuh"
#include "rk45.cuh"
#include "lpt.cuh"
#include "launch_shapes.h"
#include "sim3d.h"

namespace crp {

void philox_block(uint64_t seed, uint64_t counter, uint32_t stream, uint32_t out[4]);

namespace d3 {

struct Frame3 {
  int X, Y, Z, pitch;
  __host__ __device__ __forceinline__ long idx(int i, int j, int k) const {
    return ((long)(k + 1) * (Y + 4) + (j + 1)) * pitch + (i + 1);
  }
};

// Grid, PML and source parameters of the kernels.
struct Grid3 {
  Frame3 f;
  double dx, dy, dz, rdx, rdy, rdz, dt;
  double rho_inf, c_inf, P_inf;
  double dt_rho, s3p;  // dt / rho_inf, dt rho_inf c_inf^2
  int px0, px1;        // cells i <= px0 and i >= px1 lie in the x PML
  // PML factors 1 - s and 1 / (1 + s): faces va?/vb?[n + 1], n in [-1, N+1];
  // cells pa?/pb?[n], n in [0, N+1].
  const double *vax, *vbx, *vay, *vby, *vaz, *vbz, *pax, *pbx, *pay, *pby, *paz, *pbz;
  const short* src;  // element + 1 of every frame cell, 0 = not a source cell
  const double* elem_amp;
  const double* elem_phase;
  double pamp, omega, period, on_time, ramp_time;
};

__device__ __forceinline__ double burst_env(const Grid3& g, double tau) {
  if (!(g.ramp_time > 0.0)) return 1.0;
  const double pi = 3.14159265358979323846;
  double w = 1.0;
  if (tau < g.ramp_time) w = fmin(w, 0.5 * (1.0 - cos(pi * tau / g.ramp_time)));
  const double rest = g.on_time - tau;
  if (rest < g.ramp_time) w = fmin(w, rest > 0.0 ? 0.5 * (1.0 - cos(pi * rest / g.ramp_time)) : 0.0);
  return w;
}

// Pressure of element e at time t (0 at t = 0 and outside the burst).
__device__ __noinline__ double element_pressure(const Grid3& g, int e, double t) {
  if (!(t > 0.0)) return 0.0;
  const double tau = fmod(t, g.period);
  if (!(tau <= g.on_time)) return 0.0;
  return g.pamp * g.elem_amp[e] * burst_env(g, tau) * sin(g.omega * t + g.elem_phase[e]);
}

__device__ __forceinline__ double void_half3(const Grid3& g, double fg, double fgn) {
  if (fg == 0.0 && fgn == 0.0) return 0.0;
  return 0.5 * (-(fg - fgn) / g.dt / (1.0 - 0.5 * (fg + fgn)));
}

// Tiles of 32 x 8 x 8 cells (ghost cells included) and the last coupling in which
// bubbles touched each (mark_tiles).  Couplings are counted by the steps whose Picard
// loop ran.  A step's void fraction is nonzero at most where bubbles touched it in that
// coupling, or, without one, where it was in the three steps before.  Steps without a
// coupling can so hand an old coupling's void fraction on for as long as one of them
// falls into every three steps; the host keeps the oldest coupling that each of the last
// three steps reaches back to, and a tile not touched since the oldest of them holds
// zeros only.
constexpr int kTile3X = 32, kTile3Y = 8, kTile3Z = 8;
struct Tiles3 {
  int nx, ny, nz;
  int* last;  // coupling index of the last touch (very negative: never)
  int* list;  // active tiles of the step
  __host__ __device__ __forceinline__ int at(int x, int y, int z) const { return (z * ny + y) * nx + x; }
};

template <typename P>
struct Fdtd3Args {
  typename P::V vx_old, vy_old, vz_old, vx_new, vy_new, vz_new;
  typename P::S pnx, pny, pnz, px, py, pz;
  typename P::G fgA, fgB, fgC;  // f_g, f_gn, f_gm of the previous step; fgC receives the prediction
  int rho_const;
  // Where the void fraction can be nonzero: whether there are bubbles, and the
  // support boxes {i0, j0, k0, i1, j1, k1} of the last three steps.
  int bubbles;
  int supp[3][6];
  Tiles3 tiles;
  int oldest;            // coupling that the void fraction reaches back to
  const double* elem_p;  // pressure of every source element at the end of the step
  unsigned long long* residual;
};

// The fused pass over the grid.  A warp covers 64 columns of one row, two adjacent
// ones per lane (16-byte accesses), and marches up a chunk of planes; a block's warps
// take consecutive rows.  The plane below stays in registers and the next one is
// loaded ahead; the neighbours across rows and columns are read again (the block's
// other warps have just loaded them) and the west and south faces formed twice, so
// that no thread waits for another: no shared memory, no barriers.
//
// As in the 2-D pass the void fraction takes part only where the supports of the last
// three steps say that it can be nonzero: 96 bytes per cell elsewhere instead of
// 128, and no divisions.
//
// Bound by the latency of its loads at 16 warps per SM (128 registers); DRAM traffic is
// 1.14 times the 96 bytes per cell.  256^3 with a small cloud 366 us (4.4 TB/s of the 96
// bytes; 718 before, with each thread's inputs staged through shared memory and two
// barriers per plane), 141 x 125 x 133 without bubbles 61 us (155).
constexpr int kRows3 = 8;   // warps per block
constexpr int kCols3 = 64;  // columns per warp
constexpr double kCloudShare3 = 0.25;

enum March3Form { kPlain3 = 0, kEdges3 = 1, kVoid3 = 2 };  // inside; with x PML; with void fraction as well

struct Three {
  double2 x, y, z;
  __device__ __forceinline__ double2 sum() const { return make_double2(x.x + y.x + z.x, x.y + y.y + z.y); }
};

// The predictions of the ghost cells beside a boundary cell (every combination of
// the faces it touches).
template <typename P>
__device__ __noinline__ void predict_ghosts3(const Grid3& g, const Fdtd3Args<P>& a, int i, int j, int k) {
  using G = typename P::G;
  const Frame3& f = g.f;
  const int gi = i == 1 ? 0 : (i == f.X ? f.X + 1 : -2);
  const int gj = j == 1 ? 0 : (j == f.Y ? f.Y + 1 : -2);
  const int gk = k == 1 ? 0 : (k == f.Z ? f.Z + 1 : -2);
  for (int ci = 0; ci < 2; ci++)
    for (int cj = 0; cj < 2; cj++)
      for (int ck = 0; ck < 2; ck++) {
        if (!(ci || cj || ck)) continue;
        if ((ci && gi == -2) || (cj && gj == -2) || (ck && gk == -2)) continue;
        const long q = f.idx(ci ? gi : i, cj ? gj : j, ck ? gk : k);
        a.fgC.put(q, G::stored(3.0 * a.fgA.get(q) - 3.0 * a.fgB.get(q) + a.fgC.get(q)));
      }
}

// Columns i and i + 1 (i odd, i <= X) of row j, planes k0..k1.
template <typename P, int FORM>
__device__ __forceinline__ unsigned long long march3_chunk(const Grid3& g, const Fdtd3Args<P>& a, int i, int j,
                                                           int k0, int k1) {
  using G = typename P::G;
  using S = typename P::S;
  constexpr bool EDGE = FORM >= kEdges3, VOID = FORM == kVoid3;
  const Frame3& f = g.f;
  const bool two = i + 1 <= f.X;
  const unsigned pitch = (unsigned)f.pitch, plane = (unsigned)(f.Y + 4) * pitch;
  auto own = [&](unsigned q) -> Three { return {a.pnx.get2(q), a.pny.get2(q), a.pnz.get2(q)}; };
  auto one = [&](unsigned q) -> double { return a.pnx.get(q) + a.pny.get(q) + a.pnz.get(q); };
  auto rho_of = [&](double fa) -> double { return a.rho_const ? g.rho_inf : (1.0 - fa) * g.rho_inf; };
  // face3 with the roundings of v_old fa - q s2: the product q s2 rounded first.
  auto face = [&](double v, double p0a, double p0b, double q, double rh, double fa, double fb) -> double {
    return fma(v, fa, -__dmul_rn(q, (-p0a + p0b) * rh)) * fb;
  };
  // dt / mean(rho) of a face, the same for every cell that forms it: dt_rho, the plain
  // forms' value, where the mean is rho_inf (the quotient's last bit can differ from it).
  auto slow = [&](double ra, double rb) -> double {
    if (!VOID) return g.dt_rho;
    const double m = (ra + rb) * 0.5, q = quotient(g.dt, m);
    return m == g.rho_inf ? g.dt_rho : q;
  };
  unsigned q = ((unsigned)k0 * (unsigned)(f.Y + 4) + (unsigned)(j + 1)) * pitch + (unsigned)(i + 1);  // plane k0 - 1
  const double vayn = g.vay[j + 1], vbyn = g.vby[j + 1], vays = g.vay[j], vbys = g.vby[j];
  const double pay = g.pay[j], pby = g.pby[j];
  Three cur = own(q + plane);
  double2 pc = cur.sum();
  double2 fc = make_double2(0.0, 0.0);  // f_g of this plane
  double zb[2];                         // the faces below
  {
    const double2 pb = own(q).sum(), vb = a.vz_old.get2(q);
    double rb[2] = {0.0, 0.0}, rc[2] = {0.0, 0.0};
    if (VOID) {
      const double2 fb = a.fgA.get2(q);
      fc = a.fgA.get2(q + plane);
      rb[0] = rho_of(fb.x), rb[1] = rho_of(fb.y);
      rc[0] = rho_of(fc.x), rc[1] = rho_of(fc.y);
    }
    zb[0] = face(vb.x, pb.x, pc.x, slow(rb[0], rc[0]), g.rdz, g.vaz[k0], g.vbz[k0]);
    zb[1] = face(vb.y, pb.y, pc.y, slow(rb[1], rc[1]), g.rdz, g.vaz[k0], g.vbz[k0]);
    if (k0 == 1) {
      a.vz_new.put(q, zb[0]);
      if (two) a.vz_new.put(q + 1, zb[1]);
    }
  }
  q += plane;  // plane k0
  Three nxt = own(q + plane);
  double2 vx2 = a.vx_old.get2(q), vy2 = a.vy_old.get2(q), vs2 = a.vy_old.get2(q - pitch), vz2 = a.vz_old.get2(q);
  double vxl = a.vx_old.get(q - 1);
  unsigned long long res = 0ull;
#pragma unroll 1
  for (int k = k0; k <= k1; k++, q += plane) {
    const double2 vxo = vx2, vyo = vy2, vso = vs2, vzo = vz2;
    const double vxw = vxl;
    const Three up = nxt;
    const double2 pu = up.sum();
    // The neighbours of this plane, then what the next one needs.
    const double pl = one(q - 1), pr = one(q + 2);
    const double2 ps = own(q - pitch).sum(), pn = own(q + pitch).sum();
    const short2 e = *reinterpret_cast<const short2*>(g.src + q);
    if (k < k1) {
      nxt = own(q + 2 * plane);
      vx2 = a.vx_old.get2(q + plane);
      vy2 = a.vy_old.get2(q + plane);
      vs2 = a.vy_old.get2(q + plane - pitch);
      vz2 = a.vz_old.get2(q + plane);
      vxl = a.vx_old.get(q + plane - 1);
    }
    double qx[3] = {g.dt_rho, g.dt_rho, g.dt_rho}, qn[2] = {g.dt_rho, g.dt_rho}, qs[2] = {g.dt_rho, g.dt_rho},
           qz[2] = {g.dt_rho, g.dt_rho}, h[2] = {0.0, 0.0};
    double2 fu = fc;
    if (VOID) {
      fu = a.fgA.get2(q + plane);
      const double2 fs = a.fgA.get2(q - pitch), fn = a.fgA.get2(q + pitch), fB = a.fgB.get2(q), fC = a.fgC.get2(q);
      const double fl = a.fgA.get(q - 1), fr = a.fgA.get(q + 2);
      const double fg[2] = {G::stored(3.0 * fc.x - 3.0 * fB.x + fC.x), G::stored(3.0 * fc.y - 3.0 * fB.y + fC.y)};
      // Nothing to divide where all of the warp's void fraction is zero, nor to store
      // where the prediction is the stored zero.
      const bool some = fc.x != 0.0 || fc.y != 0.0 || fu.x != 0.0 || fu.y != 0.0 || fs.x != 0.0 || fs.y != 0.0 ||
                        fn.x != 0.0 || fn.y != 0.0 || fl != 0.0 || fr != 0.0 || fg[0] != 0.0 || fg[1] != 0.0;
      if (some || fC.x != 0.0 || fC.y != 0.0) {
        if (two)
          a.fgC.put2(q, fg[0], fg[1]);
        else
          a.fgC.put(q, fg[0]);
      }
      if (i == 1 || i + 1 >= f.X || j == 1 || j == f.Y || k == 1 || k == f.Z) {
        predict_ghosts3<P>(g, a, i, j, k);
        if (two) predict_ghosts3<P>(g, a, i + 1, j, k);
      }
      if (some) {
        const double r0 = rho_of(fc.x), r1 = rho_of(fc.y);
        qx[0] = slow(rho_of(fl), r0);
        qx[1] = slow(r0, r1);
        qx[2] = slow(r1, rho_of(fr));
        qs[0] = slow(rho_of(fs.x), r0);
        qs[1] = slow(rho_of(fs.y), r1);
        qn[0] = slow(r0, rho_of(fn.x));
        qn[1] = slow(r1, rho_of(fn.y));
        qz[0] = slow(r0, rho_of(fu.x));
        qz[1] = slow(r1, rho_of(fu.y));
        const double fo[2] = {fc.x, fc.y};
#pragma unroll
        for (int c = 0; c < 2; c++)
          h[c] = 0.5 * quotient(quotient(-(fg[c] - fo[c]), g.dt), 1.0 - 0.5 * (fg[c] + fo[c]));
      }
    }
    const double p4[4] = {pl, pc.x, pc.y, pr}, vo[3] = {vxw, vxo.x, vxo.y};
    double fx[3];
#pragma unroll
    for (int c = 0; c < 3; c++)
      fx[c] = face(vo[c], p4[c], p4[c + 1], qx[c], g.rdx, EDGE ? g.vax[i + c] : 1.0, EDGE ? g.vbx[i + c] : 1.0);
    const double vaz = g.vaz[k + 1], vbz = g.vbz[k + 1], paz = g.paz[k], pbz = g.pbz[k];
    const double yn[2] = {face(vyo.x, pc.x, pn.x, qn[0], g.rdy, vayn, vbyn),
                          face(vyo.y, pc.y, pn.y, qn[1], g.rdy, vayn, vbyn)};
    const double ys[2] = {face(vso.x, ps.x, pc.x, qs[0], g.rdy, vays, vbys),
                          face(vso.y, ps.y, pc.y, qs[1], g.rdy, vays, vbys)};
    const double zt[2] = {face(vzo.x, pc.x, pu.x, qz[0], g.rdz, vaz, vbz),
                          face(vzo.y, pc.y, pu.y, qz[1], g.rdz, vaz, vbz)};
    double nx[2], ny[2], nz[2];
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const double px = c ? cur.x.y : cur.x.x, py = c ? cur.y.y : cur.y.x, pz = c ? cur.z.y : cur.z.x;
      // pn pa - s3p (divergence + h) pb, the last product rounded first.
      nx[c] = fma(px, EDGE ? g.pax[i + c] : 1.0,
                  -__dmul_rn(__dmul_rn(g.s3p, fma(-fx[c] + fx[c + 1], g.rdx, h[c])), EDGE ? g.pbx[i + c] : 1.0));
      ny[c] = fma(py, pay, -__dmul_rn(__dmul_rn(g.s3p, fma(-ys[c] + yn[c], g.rdy, h[c])), pby));
      nz[c] = fma(pz, paz, -__dmul_rn(__dmul_rn(g.s3p, fma(-zb[c] + zt[c], g.rdz, h[c])), pbz));
      double p0new = nx[c] + ny[c] + nz[c];
      const int el = c ? e.y : e.x;
      if (el > 0) {
        p0new = a.elem_p[el - 1];
        nx[c] = p0new;
        ny[c] = nz[c] = 0.0;
      }
      if (c == 0 || two) res = max(res, (unsigned long long)__double_as_longlong(fabs((c ? pc.y : pc.x) - p0new)));
    }
    if (two) {
      a.vx_new.put2(q, fx[1], fx[2]);
      a.vy_new.put2(q, yn[0], yn[1]);
      a.vz_new.put2(q, zt[0], zt[1]);
      a.px.put2(q, nx[0], nx[1]);
      a.py.put2(q, ny[0], ny[1]);
      a.pz.put2(q, nz[0], nz[1]);
    } else {
      a.vx_new.put(q, fx[1]);
      a.vy_new.put(q, yn[0]);
      a.vz_new.put(q, zt[0]);
      a.px.put(q, nx[0]);
      a.py.put(q, ny[0]);
      a.pz.put(q, nz[0]);
    }
    if (i == 1) a.vx_new.put(q - 1, fx[0]);  // the x0 and y0 faces of the domain
    if (j == 1) {
      a.vy_new.put(q - pitch, ys[0]);
      if (two) a.vy_new.put(q - pitch + 1, ys[1]);
    }
    zb[0] = zt[0];
    zb[1] = zt[1];
    cur = up;
    pc = pu;
    fc = fu;
  }
  return res;
}

template <typename P>
__device__ __noinline__ unsigned long long march3_void(const Grid3& g, const Fdtd3Args<P>& a, int i, int j, int k0,
                                                       int k1) {
  return march3_chunk<P, kVoid3>(g, a, i, j, k0, k1);
}

// CLOUD: the supports cover much of the grid (kCloudShare3).  The void-fraction form
// then stands in line; elsewhere it is called, so that its registers are not spilled
// in the other forms' loops (256^3 with a small cloud 398 us in line, 366 called;
// 384^3 with a cloud over half of the grid 1675 and 1975).
template <typename P, bool CLOUD>
__global__ void __launch_bounds__(32 * kRows3, 2) fdtd3(const __grid_constant__ Grid3 g,
                                                        const __grid_constant__ Fdtd3Args<P> a, int planes) {
  const Frame3& f = g.f;
  const int lane = threadIdx.x, i0 = 1 + blockIdx.x * kCols3, i = i0 + 2 * lane;
  const int j = 1 + blockIdx.y * kRows3 + threadIdx.y;
  const int k0 = 1 + blockIdx.z * planes, k1 = min(f.Z, k0 + planes - 1);
  if (j > f.Y) return;
  const int i1 = min(f.X, i0 + kCols3 - 1);
  bool fg = false;
  if (a.bubbles) {
#pragma unroll
    for (int s = 0; s < 3; s++) {
      const int* b = a.supp[s];
      fg = fg || (b[0] <= b[3] && b[1] <= b[4] && b[2] <= b[5] && b[0] <= i1 + 1 && b[3] >= i0 - 1 &&
                  b[1] <= j + 1 && b[4] >= j - 1 && b[2] <= k1 + 1 && b[5] >= k0 - 1);
    }
    if (fg) {  // the supports' boxes meet the chunk: so does an active tile?
      const int x0 = (i0 - 1) / kTile3X, y0 = (j - 1) / kTile3Y, z0 = (k0 - 1) / kTile3Z;
      const int nx = (i1 + 1) / kTile3X - x0 + 1, ny = (j + 1) / kTile3Y - y0 + 1, nz = (k1 + 1) / kTile3Z - z0 + 1;
      bool live = false;
      for (int t = lane; t < nx * ny * nz; t += 32) {
        const int last = a.tiles.last[a.tiles.at(x0 + t % nx, y0 + t / nx % ny, z0 + t / (nx * ny))];
        live = live || last >= a.oldest;
      }
      fg = __any_sync(0xffffffffu, live);
    }
  }
  unsigned long long res = 0ull;
  if (i <= f.X) {
    if (fg)
      res = CLOUD ? march3_chunk<P, kVoid3>(g, a, i, j, k0, k1) : march3_void<P>(g, a, i, j, k0, k1);
    else if (i0 <= g.px0 || i1 >= g.px1)
      res = march3_chunk<P, kEdges3>(g, a, i, j, k0, k1);
    else
      res = march3_chunk<P, kPlain3>(g, a, i, j, k0, k1);
  }
  for (int o = 16; o > 0; o >>= 1) res = max(res, __shfl_xor_sync(0xffffffffu, res, o));
  if (lane == 0 && res) atomicMax(a.residual, res);
}

// ---------------------------------------------------------------------------
// Bubbles.

struct Bub3 {
  int n;
  double *x, *y, *z, *R0, *n_B, *R_t, *R_p, *R_pn, *R_n, *R_nn, *d1_R_p, *d1_R_n, *PG_p, *PG_n, *PL_p, *PL_n,
      *PL_m, *Q_B, *dt, *dt_n, *re, *re_n, *vbx, *vby, *vbz, *contrib;
  int *ibmx, *ibmy, *ibmz, *ibnx, *ibny, *ibnz, *bin, *nsub, *pos;
};

struct Scalars3 {
  unsigned long long residual;
  long long substep_max;
  int err;
  int next;
  int moved;
  int box[6];  // bubbles' ibn box: min x, y, z, max x, y, z
  int tiles;   // active tiles of this step (mark_tiles)
  double t[2];
  unsigned long long reused;  // radius solves kept (ext.rp_reuse), summed over the handle's life
};

// Start of a step: its times, the accumulators cleared, and the pressure of every
// source element at its end.
constexpr int kBeginThreads3 = 64;
__global__ void __launch_bounds__(kBeginThreads3) step_begin3(const __grid_constant__ Grid3 g, Scalars3* s,
                                                              double t_prev, double t, int elems, double* elem_p) {
  const int e = blockIdx.x * kBeginThreads3 + threadIdx.x;
  if (e < elems) elem_p[e] = element_pressure(g, e, t);
  if (e != 0) return;
  s->t[0] = t_prev;
  s->t[1] = t;
  s->residual = 0ull;
  s->moved = 0;
  s->box[0] = s->box[1] = s->box[2] = INT_MAX;
  s->box[3] = s->box[4] = s->box[5] = INT_MIN;
}

// Element pressures at the ends of up to kElemBatch steps (step blockIdx.y at t[q]).
constexpr int kElemBatch = 32;
struct ElemTimes {
  double t[kElemBatch];
};
__global__ void __launch_bounds__(kBeginThreads3) elem_batch(const __grid_constant__ Grid3 g,
                                                             const __grid_constant__ ElemTimes s, int elems,
                                                             double* elem_p) {
  const int e = blockIdx.x * kBeginThreads3 + threadIdx.x;
  if (e < elems) elem_p[(size_t)blockIdx.y * elems + e] = element_pressure(g, e, s.t[blockIdx.y]);
}

__device__ __forceinline__ int bin3_of(const Frame3& f, int ix, int iy, int iz) {
  if (ix < -1 || ix > f.X + 1 || iy < -1 || iy > f.Y + 1 || iz < -1 || iz > f.Z + 1) return -1;
  return ((iz + 1) * (f.Y + 3) + (iy + 1)) * (f.X + 3) + (ix + 1);
}

__device__ __forceinline__ double dcos(const BubbleParams& bp, double c, int pos, double h, double b) {
  return cos(c * (((double)pos - 0.5) * h - b));
}

__device__ __forceinline__ void index3(const Grid3& g, Bub3& b, int n) {
  const double x = b.x[n], y = b.y[n], z = b.z[n];
  b.ibmx[n] = (int)floor(x * g.rdx + 1.0);
  b.ibmy[n] = (int)floor(y * g.rdy + 1.0);
  b.ibmz[n] = (int)floor(z * g.rdz + 1.0);
  b.ibnx[n] = (int)floor(x * g.rdx + 0.5);
  b.ibny[n] = (int)floor(y * g.rdy + 0.5);
  b.ibnz[n] = (int)floor(z * g.rdz + 0.5);
}

__global__ void index3_kernel(const __grid_constant__ Grid3 g, Bub3 b, Scalars3* s) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= b.n) return;
  index3(g, b, n);
  b.bin[n] = bin3_of(g.f, b.ibnx[n], b.ibny[n], b.ibnz[n]);
  atomicMin(&s->box[0], b.ibnx[n]);
  atomicMin(&s->box[1], b.ibny[n]);
  atomicMin(&s->box[2], b.ibnz[n]);
  atomicMax(&s->box[3], b.ibnx[n]);
  atomicMax(&s->box[4], b.ibny[n]);
  atomicMax(&s->box[5], b.ibnz[n]);
}

// Velocity of a staggered component at the bubble: points i in ia + {0, 1},
// j in ja + {0, 1}, k in ka + {0, 1} of the array V whose logical window is
// [ilo, ihi] x [jlo, jhi] x [klo, khi].
template <typename V>
__device__ __forceinline__ double gather_v(const Grid3& g, const BubbleParams& bp, const V& v, int ia, int ja, int ka,
                                           double x, double y, double z, int ilo, int ihi, int jlo, int jhi, int klo,
                                           int khi) {
  const double cx = dcos(bp, bp.dcy, ia, g.dx, x), cy = dcos(bp, bp.dcz, ja, g.dy, y);
  const double cz = cos(2.0 * bp.pi / 2.0 * g.rdz * (((double)ka - 0.5) * g.dz - z));
  double s = 0.0;
  for (int ci = 0; ci < 2; ci++) {
    const int i = ia + ci;
    const double wx = delta_w(bp, cx, ci);
    for (int cj = 0; cj < 2; cj++) {
      const int j = ja + cj;
      const double wy = delta_w(bp, cy, cj);
      for (int ck = 0; ck < 2; ck++) {
        const int k = ka + ck;
        if (i >= ilo && i <= ihi && j >= jlo && j <= jhi && k >= klo && k <= khi)
          s += v.get(g.f.idx(i, j, k)) * wx * wy * delta_w(bp, cz, ck);
      }
    }
  }
  return s;
}

// store_variables' rotation of the bubble state, the velocity gather
// (BubbleInterpolationVelocityKernel, :398-448, with its z component), the
// motion (BubbleMotionKernel, :451-468) and the new cell indices.
template <typename V>
__device__ __forceinline__ void move3_one(const Grid3& g, const BubbleParams& bp, Bub3& b, const V& vx, const V& vy,
                                          const V& vz, Scalars3* s, int n, int* s_box) {
  b.R_pn[n] = b.R_p[n];
  b.R_nn[n] = b.R_n[n];
  b.d1_R_n[n] = b.d1_R_p[n];
  b.PG_n[n] = b.PG_p[n];
  b.PL_m[n] = b.PL_n[n];
  b.PL_n[n] = b.PL_p[n];
  b.dt_n[n] = b.dt[n];
  b.re_n[n] = b.re[n];
  const Frame3& f = g.f;
  const double x = b.x[n], y = b.y[n], z = b.z[n];
  const int mx = b.ibmx[n], my = b.ibmy[n], mz = b.ibmz[n], nx = b.ibnx[n], ny = b.ibny[n], nz = b.ibnz[n];
  const double ux = gather_v(g, bp, vx, mx - 1, ny, nz, x, y, z, -1, f.X + 1, 0, f.Y + 1, 0, f.Z + 1);
  const double uy = gather_v(g, bp, vy, nx, my - 1, nz, x, y, z, 0, f.X + 1, -1, f.Y + 1, 0, f.Z + 1);
  const double uz = gather_v(g, bp, vz, nx, ny, mz - 1, x, y, z, 0, f.X + 1, 0, f.Y + 1, -1, f.Z + 1);
  b.vbx[n] = ux;
  b.vby[n] = uy;
  b.vbz[n] = uz;
  b.x[n] = x + ux * g.dt;
  b.y[n] = y + uy * g.dt;
  b.z[n] = z + uz * g.dt;
  index3(g, b, n);
  const int ix = b.ibnx[n], iy = b.ibny[n], iz = b.ibnz[n];
  const int bin = bin3_of(f, ix, iy, iz);
  if (bin != b.bin[n]) {
    atomicOr(&s->moved, 1);
    b.bin[n] = bin;
  }
  // The bubbles' box: over the warp, then the block, then one atomic each per block
  // (six per bubble on the same words took most of the launch: 2 M bubbles 477 us).
  const unsigned m = __activemask();
  const int r[6] = {__reduce_min_sync(m, ix), __reduce_min_sync(m, iy), __reduce_min_sync(m, iz),
                    __reduce_max_sync(m, ix), __reduce_max_sync(m, iy), __reduce_max_sync(m, iz)};
  if ((threadIdx.x & 31) == __ffs(m) - 1) {
    for (int q = 0; q < 3; q++) {
      atomicMin(&s_box[q], r[q]);
      atomicMax(&s_box[q + 3], r[q + 3]);
    }
  }
}
template <typename V>
__global__ void __launch_bounds__(256) move3(const __grid_constant__ Grid3 g, const __grid_constant__ BubbleParams bp,
                                             Bub3 b, const V vx, const V vy, const V vz, Scalars3* s) {
  __shared__ int s_box[6];
  if (threadIdx.x < 6) s_box[threadIdx.x] = threadIdx.x < 3 ? INT_MAX : INT_MIN;
  __syncthreads();
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n < b.n) move3_one(g, bp, b, vx, vy, vz, s, n, s_box);
  __syncthreads();
  if (threadIdx.x < 3)
    atomicMin(&s->box[threadIdx.x], s_box[threadIdx.x]);
  else if (threadIdx.x < 6)
    atomicMax(&s->box[threadIdx.x], s_box[threadIdx.x]);
}

// Counting sort of bubbles by bin (ascending bubble index within a bin).
constexpr int kScan = 1024;

__device__ __forceinline__ int block_scan(int v, int* total) {
  __shared__ int s_w[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_w[w] = x;
  __syncthreads();
  if (w == 0) {
    int t = s_w[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    s_w[lane] = t;
  }
  __syncthreads();
  const int before = (w > 0 ? s_w[w - 1] : 0) + x - v;
  if (total) *total = s_w[31];
  return before;
}

__global__ void bin3_count(const int* __restrict__ bin, int n, int* __restrict__ count) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n && bin[k] >= 0) atomicAdd(&count[bin[k]], 1);
}
__global__ void __launch_bounds__(kScan) bin3_scan(const int* __restrict__ count, int* __restrict__ start,
                                                  int* __restrict__ partial, int nbins) {
  const int k = blockIdx.x * kScan + threadIdx.x;
  int total;
  const int e = block_scan(k < nbins ? count[k] : 0, &total);
  if (k < nbins) start[k] = e;
  if (threadIdx.x == 0) partial[blockIdx.x] = total;
}
__global__ void __launch_bounds__(kScan) bin3_partials(int* __restrict__ partial, int nparts) {
  int carry = 0;
  for (int base = 0; base < nparts; base += kScan) {
    const int k = base + threadIdx.x;
    int total;
    const int e = block_scan(k < nparts ? partial[k] : 0, &total);
    __syncthreads();
    if (k < nparts) partial[k] = e + carry;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[nparts] = carry;
}
__global__ void bin3_add(int* __restrict__ start, const int* __restrict__ partial, int nbins, int nparts) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < nbins) start[k] += partial[k / kScan];
  if (k == nbins) start[nbins] = partial[nparts];
}
__global__ void bin3_fill(const int* __restrict__ bin, int n, const int* __restrict__ start, int* __restrict__ count,
                          int* __restrict__ idx) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n || bin[b] < 0) return;
  idx[start[bin[b]] + atomicSub(&count[bin[b]], 1) - 1] = b;
}
// One thread per bin: its bubbles in ascending index order.
__global__ void bin3_sort(const int* __restrict__ start, int* __restrict__ idx, int nbins) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nbins) return;
  const int a = start[c], e = start[c + 1];
  for (int q = a + 1; q < e; q++) {
    const int v = idx[q];
    int m = q - 1;
    while (m >= a && idx[m] > v) {
      idx[m + 1] = idx[m];
      m--;
    }
    idx[m + 1] = v;
  }
}
__global__ void bin3_pos(const int* __restrict__ idx, int total, int* __restrict__ pos) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < total) pos[idx[k]] = k;
}

// Pressure gather at the bubble (BubbleInterpolationScalarKernel, :361-395,
// over 2 x 2 x 2 cells) and its eight void-fraction contributions
// (VoidFractionReverseLookupKernel, :576-619, with the z factor), stored at
// 8 pos so that each cell reads contiguous runs.
template <typename S>
__device__ __forceinline__ double gather_pl3(const Grid3& g, const BubbleParams& bp, const Bub3& b, const S& px,
                                             const S& py, const S& pz, int n) {
  const Frame3& f = g.f;
  const double x = b.x[n], y = b.y[n], z = b.z[n];
  const int ix = b.ibnx[n], iy = b.ibny[n], iz = b.ibnz[n];
  const double cx = dcos(bp, bp.dcy, ix, g.dx, x), cy = dcos(bp, bp.dcz, iy, g.dy, y);
  const double cz = cos(2.0 * bp.pi / 2.0 * g.rdz * (((double)iz - 0.5) * g.dz - z));
  double s = 0.0;
  for (int ci = 0; ci < 2; ci++)
    for (int cj = 0; cj < 2; cj++)
      for (int ck = 0; ck < 2; ck++) {
        const int i = ix + ci, j = iy + cj, k = iz + ck;
        if (i >= 0 && i <= f.X + 1 && j >= 0 && j <= f.Y + 1 && k >= 0 && k <= f.Z + 1) {
          const long q = f.idx(i, j, k);
          s += (px.get(q) + py.get(q) + pz.get(q)) * delta_w(bp, cx, ci) * delta_w(bp, cy, cj) * delta_w(bp, cz, ck);
        }
      }
  return s;
}

__device__ __forceinline__ void contrib3(const Grid3& g, const BubbleParams& bp, const Bub3& b, int n, double Rt) {
  const int p = b.pos[n];
  if (p < 0) return;
  const double x = b.x[n], y = b.y[n], z = b.z[n];
  const int ix = b.ibnx[n], iy = b.ibny[n], iz = b.ibnz[n];
  const double cx = dcos(bp, bp.dcy, ix, g.dx, x), cy = dcos(bp, bp.dcz, iy, g.dy, y);
  const double cz = cos(2.0 * bp.pi / 2.0 * g.rdz * (((double)iz - 0.5) * g.dz - z));
  const double vol = bp.pi4r3 * b.n_B[n] * (Rt * Rt * Rt) * g.rdx * g.rdy * g.rdz;
  double* c = b.contrib + 8 * (long)p;
  for (int ci = 0; ci < 2; ci++)
    for (int cj = 0; cj < 2; cj++)
      for (int ck = 0; ck < 2; ck++)
        c[ci * 4 + cj * 2 + ck] = vol * delta_w(bp, cx, ci) * delta_w(bp, cy, cj) * delta_w(bp, cz, ck);
}

constexpr int kRpThreads3 = 128;
// Resident blocks per SM the register budget is set for, and the sub-step count from
// which a launch waits for its stiffest bubble (TIGHT): as the 2-D radius kernel's.
template <typename P, bool TIGHT>
constexpr int radius3_min_blocks() {
  return TIGHT ? 3 : sizeof(typename P::T) == sizeof(double) ? 7 : 5;
}
constexpr long long kTightSubsteps3 = 150;

// The radius solves: the reference scheme's sub-steps (rp_substep_full) or
// the rk45 scheme (rk_attempt), from the state stored at the step's start,
// persistent lanes claiming bubbles from a queue.  With `reuse` (a solve of
// this step has completed), a bubble whose gathered pressure has the bit
// pattern of the last solve's keeps that solve's results: every input of its
// solve is unchanged.
template <typename P, bool RK, bool TIGHT>
__global__ void __launch_bounds__(kRpThreads3, RK ? 1 : radius3_min_blocks<P, TIGHT>()) radius3(const __grid_constant__ Grid3 g,
                                                       const __grid_constant__ BubbleParams bp, Bub3 b,
                                                       const typename P::S px, const typename P::S py,
                                                       const typename P::S pz, Scalars3* sc, int reuse,
                                                       const int* __restrict__ order) {
  const double dt = g.dt;
  RpState<typename P::T, kLean> s;
  RkState r;
  int n = -1;
  bool drained = false;
  long long worst = 0;
  unsigned long long kept = 0;
  const int lane = threadIdx.x & 31;
  for (;;) {
    const unsigned need = __ballot_sync(0xffffffffu, n < 0 && !drained);
    if (need) {
      const int leader = __ffs(need) - 1;
      int base = 0;
      if (lane == leader) base = atomicAdd(&sc->next, __popc(need));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (need & (1u << lane)) {
        const int q = base + __popc(need & ((1u << lane) - 1u));
        const int bn = q < b.n ? (order ? order[q] : q) : -1;  // heaviest first once an order is built
        const double PLp = bn >= 0 ? gather_pl3(g, bp, b, px, py, pz, bn) : 0.0;
        if (bn < 0) {
          drained = true;
        } else if (reuse && __double_as_longlong(PLp) == __double_as_longlong(b.PL_p[bn])) {
          kept++;
        } else {
          n = bn;
          b.PL_p[n] = PLp;
          const double PLn = b.PL_n[n], PLm = b.PL_m[n];
          const double PC0 = PLn + bp.PL0, PC1 = 0.5 * (PLp - PLm) / dt,
                       PC2 = 0.5 * (PLp + PLm - 2.0 * PLn) / (dt * dt);
          if (RK) {
            r.r = bubble_r0(bp, b.R0[n]);
            r.R = b.R_pn[n];
            r.V = b.d1_R_n[n];
            r.PG = b.PG_n[n];
            r.h = b.dt_n[n];
            r.t = 0.0;
            r.tend = dt;
            r.Q = 0.0;
            r.count = 0;
            r.fresh = true;
            r.PC0 = PC0;
            r.PC1 = PC1;
            r.PC2 = PC2;
            r.K = 3.0 * (bp.gam - 1.0) * bp.K0 * bp.T0 * r.r.inv_PG0;
          } else {
            radius_const(bp, b.R0[n], s);
            s.Rt = b.R_t[n];
            s.Rp = b.R_pn[n];
            s.Rn = b.R_nn[n];
            s.d1Rp = b.d1_R_n[n];
            s.PGp = b.PG_n[n];
            s.dtL = b.dt_n[n];
            s.re_n = b.re_n[n];
            s.remain = s.re_n + dt;
            s.time = -s.re_n;
            s.PC0 = PC0;
            s.PC1 = PC1;
            s.PC2 = PC2;
            s.heat = 0.0;
            s.vis = 0.0;
            s.count = 0;
          }
        }
      }
    }
    if (!__any_sync(0xffffffffu, n >= 0 || !drained)) break;
    if (n < 0) continue;
    if (RK) {
      if (r.t < r.tend && r.count < bp.step_cap) {
        if (!rk_attempt<typename P::T>(bp, r, bp.rk_rtol, g.c_inf)) r.count = bp.step_cap;
        continue;
      }
      if (r.t < r.tend) atomicOr(&sc->err, 1);
      b.R_t[n] = b.R_p[n] = b.R_n[n] = r.R;
      b.d1_R_p[n] = r.V;
      b.PG_p[n] = r.PG;
      b.dt[n] = fmin(r.h, dt);
      b.re[n] = 0.0;
      b.Q_B[n] = r.Q / dt;
      b.nsub[n] = (int)min(r.count, (long long)INT32_MAX);
      contrib3(g, bp, b, n, r.R);
      worst = max(worst, r.count);
    } else {
      if (rp_more(bp, s)) {
        rp_substep_full<TIGHT>(bp, s);
        continue;
      }
      if (rp_failed(s)) atomicOr(&sc->err, 1);
      b.R_t[n] = s.Rt;
      b.R_p[n] = s.Rp;
      b.R_n[n] = s.Rn;
      b.d1_R_p[n] = s.d1Rp;
      b.PG_p[n] = s.PGp;
      b.dt[n] = s.dtL;
      b.re[n] = s.remain;
      b.Q_B[n] = (s.heat + s.vis) / (dt - s.remain + s.re_n);
      b.nsub[n] = s.count;
      contrib3(g, bp, b, n, s.Rt);
      worst = max(worst, (long long)s.count);
    }
    n = -1;
  }
  for (int o = 16; o > 0; o >>= 1) worst = max(worst, __shfl_xor_sync(0xffffffffu, worst, o));
  if (lane == 0 && worst > 0) atomicMax(&sc->substep_max, worst);
  for (int o = 16; o > 0; o >>= 1) kept += __shfl_xor_sync(0xffffffffu, kept, o);
  if (lane == 0 && kept) atomicAdd(&sc->reused, kept);
}

template <typename P>
struct Couple3Args {
  typename P::V vx, vy, vz;
  typename P::S pnx, pny, pnz, px, py, pz;
  typename P::G fg, fgn;
  const int* start;
  const double* contrib;
  Tiles3 tiles;
  const int* n_tiles;
  int pressure;
  const double* elem_p;
  unsigned long long* residual;
};

// One warp per tile: whether a bin that touches its cells holds bubbles (the bins
// of a row of cells are contiguous runs of the bin starts), and the list of the tiles
// that may hold void fraction.  Only the tiles [lo, lo + n) that the bubbles' and the
// supports' boxes meet.
struct TileRange {
  int lo[3], n[3];
};
__global__ void __launch_bounds__(256) mark_tiles(const Frame3 f, const int* __restrict__ start, Tiles3 t,
                                                  TileRange r, int coupling, int oldest, int* __restrict__ n_tiles) {
  const int q = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (q >= r.n[0] * r.n[1] * r.n[2]) return;
  const int tile = t.at(r.lo[0] + q % r.n[0], r.lo[1] + q / r.n[0] % r.n[1], r.lo[2] + q / (r.n[0] * r.n[1]));
  const int i0 = tile % t.nx * kTile3X, j0 = tile / t.nx % t.ny * kTile3Y, k0 = tile / (t.nx * t.ny) * kTile3Z;
  const int bx0 = i0 - 1, bx1 = min(i0 + kTile3X - 1, f.X + 1);
  bool some = false;
  for (int c = lane; c < (kTile3Y + 1) * (kTile3Z + 1); c += 32) {
    const int by = j0 - 1 + c % (kTile3Y + 1), bz = k0 - 1 + c / (kTile3Y + 1);
    if (by > f.Y + 1 || bz > f.Z + 1) continue;
    const int row = ((bz + 1) * (f.Y + 3) + (by + 1)) * (f.X + 3);
    some = some || start[row + bx0 + 1] != start[row + bx1 + 2];
  }
  some = __any_sync(0xffffffffu, some);
  if (lane != 0) return;
  int last = t.last[tile];
  if (some) t.last[tile] = last = coupling;
  if (last >= oldest) t.list[atomicAdd(n_tiles, 1)] = tile;
}

// Per cell of the active tiles: the void fraction from the eight bins whose bubbles
// touch it (their runs in order, bins in a fixed order), then the pressure
// re-evaluation with it, the source forcing and the residual.
//
// A block takes a plane of a tile, a warp 32 cells of a row.  The bins that touch them are four
// contiguous runs of the bin starts, so two starts per run tell the warp which of the
// runs hold bubbles at all.  (One thread per cell of the supports' box, each with its
// 16 bin starts, took 868 us on 384^3 with a Gaussian cloud, most of it in cells without
// void fraction.)
template <typename P>
__global__ void __launch_bounds__(256, 4) couple3(const __grid_constant__ Grid3 g, const Couple3Args<P> a) {
  using G = typename P::G;
  const Frame3& f = g.f;
  unsigned long long res = 0ull;
  const int n = *a.n_tiles * kTile3Z;
  for (int t = blockIdx.x; t < n; t += gridDim.x) {
    const int tile = a.tiles.list[t / kTile3Z];
    const int i0 = tile % a.tiles.nx * kTile3X, i = i0 + threadIdx.x;
    const int j = tile / a.tiles.nx % a.tiles.ny * kTile3Y + threadIdx.y;
    const int k = tile / (a.tiles.nx * a.tiles.ny) * kTile3Z + t % kTile3Z;
    if (k <= f.Z + 1) {
      bool some = false;
      if (threadIdx.x < 4 && j <= f.Y + 1) {
        const int by = j - (int)(threadIdx.x >> 1), bz = k - (int)(threadIdx.x & 1);
        const int row = ((bz + 1) * (f.Y + 3) + (by + 1)) * (f.X + 3);
        some = a.start[row + i0] != a.start[row + min(i0 + kTile3X - 1, f.X + 1) + 2];
      }
      // Bit cj * 2 + ck: the run of bins (.., j - cj, k - ck) holds bubbles.
      const unsigned runs = __ballot_sync(0xffffffffu, some);
      if (i > f.X + 1 || j > f.Y + 1) continue;
      const long o = f.idx(i, j, k);
      double fgv = 0.0;
      if (runs) {
        // The starts of bins i - 1, i, i + 1 of the four runs, all at once; then each
        // bin's values four at a time, added in order (absent ones as zeros).
        int st[4][3];
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const int row = ((k - (r & 1) + 1) * (f.Y + 3) + (j - (r >> 1) + 1)) * (f.X + 3) + i;
#pragma unroll
          for (int c = 0; c < 3; c++) st[r][c] = runs >> r & 1u ? a.start[row + c] : 0;
        }
#pragma unroll
        for (int ci = 0; ci < 2; ci++)
#pragma unroll
          for (int r = 0; r < 4; r++) {
            const double* __restrict__ v = a.contrib + ci * 4 + r;
            double run = 0.0;
            for (int q = st[r][1 - ci]; q < st[r][2 - ci]; q += 4) {
              double w[4];
#pragma unroll
              for (int d = 0; d < 4; d++) w[d] = q + d < st[r][2 - ci] ? v[8 * (long)(q + d)] : 0.0;
#pragma unroll
              for (int d = 0; d < 4; d++) run += w[d];
            }
            fgv += run;
          }
      }
      fgv = G::stored(fgv);
      // No bubble touches the cell and its void fraction was zero in the
      // prediction and the step before: the gathered value is the stored 0
      // and the pressure evaluation would repeat the FDTD pass's (no
      // void-fraction rate), so the cell is left as it is.
      if (fgv == 0.0 && a.fg.get(o) == 0.0 && a.fgn.get(o) == 0.0) continue;
      a.fg.put(o, fgv);
      if (!(a.pressure && i >= 1 && i <= f.X && j >= 1 && j <= f.Y && k >= 1 && k <= f.Z)) continue;
      const double h = void_half3(g, fgv, a.fgn.get(o));
      const long ox = o - 1, oy = o - f.pitch, oz = o - (long)(f.Y + 4) * f.pitch;
      const double s1x = (-a.vx.get(ox) + a.vx.get(o)) * g.rdx;
      const double s1y = (-a.vy.get(oy) + a.vy.get(o)) * g.rdy;
      const double s1z = (-a.vz.get(oz) + a.vz.get(o)) * g.rdz;
      const double qx = a.pnx.get(o) * g.pax[i] - g.s3p * (s1x + h) * g.pbx[i];
      const double qy = a.pny.get(o) * g.pay[j] - g.s3p * (s1y + h) * g.pby[j];
      const double qz = a.pnz.get(o) * g.paz[k] - g.s3p * (s1z + h) * g.pbz[k];
      const double old = a.px.get(o) + a.py.get(o) + a.pz.get(o);
      double p0new = qx + qy + qz;
      const int e = g.src[o];
      if (e > 0) {
        p0new = a.elem_p[e - 1];
        a.px.put(o, p0new);
        a.py.put(o, 0.0);
        a.pz.put(o, 0.0);
      } else {
        a.px.put(o, qx);
        a.py.put(o, qy);
        a.pz.put(o, qz);
      }
      res = max(res, (unsigned long long)__double_as_longlong(fabs(old - p0new)));
    }
  }
  for (int off = 16; off > 0; off >>= 1) res = max(res, __shfl_xor_sync(0xffffffffu, res, off));
  if (threadIdx.x == 0 && res) atomicMax(a.residual, res);
}

// Contributions of every bubble at its current radius (set-up).
__global__ void contrib_init3(const __grid_constant__ Grid3 g, const __grid_constant__ BubbleParams bp, Bub3 b) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n < b.n) contrib3(g, bp, b, n, b.R_t[n]);
}

// Dense read-back of a window of the frame (x fastest).  kind 0: velocity or
// split-pressure storage; 1: void-fraction storage; 2: p0 = px + py + pz;
// 3: the mixture density (1 - f_g) rho_inf the next velocity update uses.
__global__ void read3(Frame3 f, int kind, int mixed, const void* buf, const void* px, const void* py, const void* pz,
                      int ilo, int jlo, int klo, int nx, int ny, int nz, double rho_inf, int rho_const,
                      double* __restrict__ out) {
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long)nx * ny * nz) return;
  const int i = ilo + (int)(e % nx), j = jlo + (int)((e / nx) % ny), k = klo + (int)(e / ((long)nx * ny));
  const long q = f.idx(i, j, k);
  auto sv = [&](const void* p) -> double {
    return mixed ? F32c{(float2*)p}.get(q) : F64{(double*)p}.get(q);
  };
  auto gv = [&](const void* p) -> double { return mixed ? F32{(float*)p}.get(q) : F64{(double*)p}.get(q); };
  double v;
  switch (kind) {
    case 0: v = sv(buf); break;
    case 1: v = gv(buf); break;
    case 2: v = sv(px) + sv(py) + sv(pz); break;
    default: v = rho_const ? rho_inf : (1.0 - gv(buf)) * rho_inf; break;
  }
  out[e] = v;
}

// Plain FP64 / mixed storage of the fields, as the 2-D path.
struct P64 {
  using V = F64;
  using S = F64;
  using G = F64;
  using T = double;
  static constexpr int kIndex = 0;
};
struct PMix {
  using V = F32c;
  using S = F32c;
  using G = F32;
  using T = float;
  static constexpr int kIndex = 1;
};

// ---------------------------------------------------------------------------
// Discrete adjoint of the bubble-free 3-D step (crp_adjoint).  Without bubbles
// the step is linear in the state:
//   v'_f  = (v_f va - dt_rho rd (p0_b - p0_a)) vb           every computed face f
//                                                            between cells a and b,
//   p'_c  = p_c pa_c - s3p pb_c (v'_east - v'_west) rd_c     interior cells, c = x, y, z,
//   p'_x  = s_e(t), p'_y = p'_z = 0                         source cells,
// with p0 = px + py + pz (0 in the ghost cells, which are never written).  The
// reverse of one step, given the adjoint of the state after it:
//   1. adj3_source: the source cells' share of the gradient, their adjoint zeroed;
//   2. adj3_march, one pass from one set of adjoint frames into the other:
//      the face adjoints take the pressure update's transpose; the component
//      adjoints become pa_c M_c plus the velocity update's transpose into p0
//      (the same for all three components); the face adjoints are multiplied
//      by va vb; and 2 dt w p0 of the step before is added for the focal cells
//      (adj3_force adds the last step's before the sweep).
// Each cell forms the transposed values of its faces (its west and south faces by the
// same expression as the neighbour that owns them), so a step reads 6 doubles per
// cell (L and M; neighbours through L1/L2) and writes 6: 96 bytes.
struct Adj3 {
  double *LX, *LY, *LZ;  // adjoints of vx, vy, vz (frame layout)
  double *MX, *MY, *MZ;  // adjoints of px, py, pz
};
struct Box3 {
  int i0, j0, k0, nx, ny, nz;
  const double* w;  // weight of each box cell (0 outside the focal sphere)
};

template <typename S>
__global__ void adj3_record(const Frame3 f, const S px, const S py, const S pz, const Box3 b, double* out) {
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= (long)b.nx * b.ny * b.nz) return;
  const int i = b.i0 + (int)(t % b.nx), j = b.j0 + (int)((t / b.nx) % b.ny), k = b.k0 + (int)(t / ((long)b.nx * b.ny));
  const long q = f.idx(i, j, k);
  out[t] = px.get(q) + py.get(q) + pz.get(q);
}

__global__ void adj3_objective(const Box3 b, const double* p0, double* Jn) {
  // One block per recorded step: sum of w p0^2 in a fixed order.
  __shared__ double part[256];
  const long n = (long)b.nx * b.ny * b.nz;
  const double* p = p0 + blockIdx.x * n;
  double s = 0.0;
  for (long t = threadIdx.x; t < n; t += blockDim.x) s += b.w[t] * p[t] * p[t];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) Jn[blockIdx.x] = part[0];
}

__global__ void adj3_force(const Frame3 f, const Adj3 a, const Box3 b, const double* p0, double two_dt) {
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= (long)b.nx * b.ny * b.nz) return;
  const double w = b.w[t];
  if (w == 0.0) return;
  const int i = b.i0 + (int)(t % b.nx), j = b.j0 + (int)((t / b.nx) % b.ny), k = b.k0 + (int)(t / ((long)b.nx * b.ny));
  const long q = f.idx(i, j, k);
  const double d = two_dt * w * p0[t];
  a.MX[q] += d;
  a.MY[q] += d;
  a.MZ[q] += d;
}

// The source's factors at the times of up to kElemBatch reverse steps: whether the
// burst is on, the envelope, every element's sine and cosine.
struct SourceFactors {
  double* env;  // [step][on, envelope]
  double* sn;   // [step][element]
  double* cs;
};
__global__ void __launch_bounds__(kBeginThreads3) adj3_factors(const __grid_constant__ Grid3 g,
                                                               const __grid_constant__ ElemTimes s, int elems,
                                                               const SourceFactors o) {
  const int e = blockIdx.x * kBeginThreads3 + threadIdx.x;
  const double t = s.t[blockIdx.y], tau = fmod(t, g.period);
  if (e == 0) {
    const bool on = t > 0.0 && tau <= g.on_time;
    o.env[2 * blockIdx.y] = on ? 1.0 : 0.0;
    o.env[2 * blockIdx.y + 1] = on ? g.pamp * burst_env(g, tau) : 0.0;
  }
  if (e >= elems) return;
  double sn, cs;
  sincos(g.omega * t + g.elem_phase[e], &sn, &cs);
  o.sn[(size_t)blockIdx.y * elems + e] = sn;
  o.cs[(size_t)blockIdx.y * elems + e] = cs;
}

// Source cell c (frame index cells[c], element elem[c]) at the step whose factors
// these are: d p'_x / d amp_e and d p'_x / d phase_e times the adjoint of p'_x, summed
// over the steps per cell; the cell's adjoints then end (the forced values do
// not depend on the state).  Three dependent loads long: 6.7 us for the bowl of
// 141 x 125 x 133, 9.6 with the loads after the stores.
__global__ void adj3_source(const __grid_constant__ Grid3 g, const Adj3 a, const long* cells, const int* elem, int n,
                            const SourceFactors t, double* gA, double* gP) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  // All loads before the first store, which they would otherwise have to wait for.
  const long q = cells[c];
  const int e = elem[c];
  const double on = t.env[0], env = t.env[1], ga = gA[c], gp = gP[c], amp = g.elem_amp[e], sn = t.sn[e], cs = t.cs[e];
  const double m = a.MX[q];
  a.MX[q] = 0.0;
  a.MY[q] = 0.0;
  a.MZ[q] = 0.0;
  if (on == 0.0) return;
  gA[c] = fma(m * env, sn, ga);
  gP[c] = fma(__dmul_rn(m * env, amp), cs, gp);
}

// One reverse step after adj3_source, from `in` into `out`; p0 (the focal
// pressures of the step before, or null) adds that step's objective term.  Warps of 64
// columns, two per lane, march along z as in fdtd3; the value of the face below is that
// of the top face one plane down.  Every lane forms the transposed values
// L + s3p rd (pb_b M_b - pb_a M_a) of its faces (computed faces: vx for i in [0, X] with j,
// k interior; vy for j in [0, Y]; vz for k in [0, Z]); the first column, row and plane also
// write the 0 faces.  Bound by the latency of the loads at 16 warps per SM: 141 x 125 x 133
// takes 45.9 us (96 bytes per cell: 4.9 TB/s), 56 with one cell per thread.
__global__ void __launch_bounds__(32 * kRows3, 2) adj3_march(const __grid_constant__ Grid3 g, const Adj3 in,
                                                             const Adj3 out, const Box3 b,
                                                             const double* __restrict__ p0, double two_dt, int planes) {
  const Frame3& f = g.f;
  const int i = 1 + blockIdx.x * kCols3 + 2 * threadIdx.x, j = 1 + blockIdx.y * kRows3 + threadIdx.y;
  const int k0 = 1 + blockIdx.z * planes, k1 = min(f.Z, k0 + planes - 1);
  if (i > f.X || j > f.Y) return;
  const bool two = i + 1 <= f.X;
  const unsigned pitch = (unsigned)f.pitch, plane = (unsigned)(f.Y + 4) * pitch;
  auto get2 = [](const double* p, unsigned q) { return *reinterpret_cast<const double2*>(p + q); };
  const double sx = -g.s3p * g.rdx, sy = -g.s3p * g.rdy, sz = -g.s3p * g.rdz;
  // Lt of the face between cells a and b.
  auto lt = [](double L, double s, double pa, double ma, double pb, double mb) -> double {
    return fma(s, fma(pa, ma, -__dmul_rn(pb, mb)), L);
  };
  double pbx[4], vbx[3], ax[3], pax[2];
#pragma unroll
  for (int c = 0; c < 4; c++) pbx[c] = g.pbx[min(i - 1 + c, f.X + 1)];
#pragma unroll
  for (int c = 0; c < 3; c++) vbx[c] = g.vbx[i + c], ax[c] = g.vax[i + c] * vbx[c];
  pax[0] = g.pax[i], pax[1] = g.pax[i + 1];
  const double pbs = g.pby[j - 1], pbj = g.pby[j], pbn = g.pby[j + 1], pay = g.pay[j];
  const double vbs = g.vby[j], vbn = g.vby[j + 1], ayn = g.vay[j + 1] * vbn, ays = g.vay[j] * vbs;
  unsigned q = ((unsigned)(k0 + 1) * (unsigned)(f.Y + 4) + (unsigned)(j + 1)) * pitch + (unsigned)(i + 1);
  double2 mz = get2(in.MZ, q);
  double zb[2];
  {
    const double2 l = get2(in.LZ, q - plane), m = get2(in.MZ, q - plane);
    const double pa = g.pbz[k0 - 1], pb = g.pbz[k0];
    zb[0] = lt(l.x, sz, pa, m.x, pb, mz.x);
    zb[1] = lt(l.y, sz, pa, m.y, pb, mz.y);
  }
#pragma unroll 1
  for (int k = k0; k <= k1; k++, q += plane) {
    const double2 lx = get2(in.LX, q), ly = get2(in.LY, q), ls = get2(in.LY, q - pitch), lz = get2(in.LZ, q);
    const double2 mx = get2(in.MX, q), my = get2(in.MY, q), ms = get2(in.MY, q - pitch), mn = get2(in.MY, q + pitch);
    const double2 mu = get2(in.MZ, q + plane);
    const double lw = in.LX[q - 1], mw = in.MX[q - 1], me = in.MX[q + 2];
    const double m4[4] = {mw, mx.x, mx.y, me}, l3[3] = {lw, lx.x, lx.y};
    double xt[3];
#pragma unroll
    for (int c = 0; c < 3; c++) xt[c] = lt(l3[c], sx, pbx[c], m4[c], pbx[c + 1], m4[c + 1]);
    const double yn[2] = {lt(ly.x, sy, pbj, my.x, pbn, mn.x), lt(ly.y, sy, pbj, my.y, pbn, mn.y)};
    const double ys[2] = {lt(ls.x, sy, pbs, ms.x, pbj, my.x), lt(ls.y, sy, pbs, ms.y, pbj, my.y)};
    const double pbk = g.pbz[k], pbu = g.pbz[k + 1], vbt = g.vbz[k + 1], vbb = g.vbz[k];
    const double zt[2] = {lt(lz.x, sz, pbk, mz.x, pbu, mu.x), lt(lz.y, sz, pbk, mz.y, pbu, mu.y)};
    const double azt = g.vaz[k + 1] * vbt, paz = g.paz[k];
    const double m3[2][3] = {{mx.x, my.x, mz.x}, {mx.y, my.y, mz.y}};
    double nm[3][2];
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const double dx = fma(vbx[c + 1], xt[c + 1], -__dmul_rn(vbx[c], xt[c]));
      const double dy = fma(vbn, yn[c], -__dmul_rn(vbs, ys[c]));
      const double dz = fma(vbt, zt[c], -__dmul_rn(vbb, zb[c]));
      const double lp0 = __dmul_rn(g.dt_rho, fma(g.rdz, dz, fma(g.rdx, dx, __dmul_rn(g.rdy, dy))));
      nm[0][c] = fma(pax[c], m3[c][0], lp0);
      nm[1][c] = fma(pay, m3[c][1], lp0);
      nm[2][c] = fma(paz, m3[c][2], lp0);
      if (p0) {
        const int bi = i + c - b.i0, bj = j - b.j0, bk = k - b.k0;
        if (bi >= 0 && bi < b.nx && bj >= 0 && bj < b.ny && bk >= 0 && bk < b.nz) {
          const long t = bi + (long)b.nx * (bj + (long)b.ny * bk);
          const double w = b.w[t];
          if (w != 0.0) {
            const double d = __dmul_rn(two_dt * w, p0[t]);
            nm[0][c] += d;
            nm[1][c] += d;
            nm[2][c] += d;
          }
        }
      }
    }
    auto put = [&](double* p, unsigned r, double v, double w) {
      if (two)
        *reinterpret_cast<double2*>(p + r) = make_double2(v, w);
      else
        p[r] = v;
    };
    put(out.MX, q, nm[0][0], nm[0][1]);
    put(out.MY, q, nm[1][0], nm[1][1]);
    put(out.MZ, q, nm[2][0], nm[2][1]);
    put(out.LX, q, xt[1] * ax[1], xt[2] * ax[2]);
    put(out.LY, q, yn[0] * ayn, yn[1] * ayn);
    put(out.LZ, q, zt[0] * azt, zt[1] * azt);
    if (i == 1) out.LX[q - 1] = xt[0] * ax[0];
    if (j == 1) put(out.LY, q - pitch, ys[0] * ays, ys[1] * ays);
    if (k == 1) {
      const double az0 = g.vaz[1] * g.vbz[1];
      put(out.LZ, q - plane, zb[0] * az0, zb[1] * az0);
    }
    zb[0] = zt[0];
    zb[1] = zt[1];
    mz = mu;
  }
}

}  // namespace d3

// ---------------------------------------------------------------------------
// Host side.

struct Sim3Impl {
  crp_config cfg{};
  d3::Grid3 g{};
  BubbleParams bp{};
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  int device = 0, sms = 1;
  bool mixed = false;
  std::string err;
  char* pool = nullptr;
  size_t pool_bytes = 0;
  size_t cells = 0;
  void *vx[2]{}, *vy[2]{}, *vz[2]{}, *px[2]{}, *py[2]{}, *pz[2]{}, *fg[3]{};
  double* d_fac = nullptr;  // PML factors
  short* d_src = nullptr;
  double* d_elem = nullptr;
  double* elem_p = nullptr;  // pressure of every element at the end of the step
  double* scratch = nullptr;  // dense read-back
  d3::Bub3 bub{};
  int* bin_count = nullptr;
  int* bin_start = nullptr;
  int* bin_idx = nullptr;
  int* bin_partial = nullptr;
  int nbins = 0;
  d3::Scalars3* d_sc = nullptr;
  d3::Scalars3* h_sc = nullptr;
  int elem_n = 0;
  int src_cells = 0;
  int cur_v = 0, cur_p = 0, fg_a = 0, fg_b = 1, fg_c = 2;
  double tstep = 0.0, tstepx = 0.0, t_prev = 0.0;
  double picard_tol = 1.0e-7f;
  bool bins_stale = true;
  int* lpt_hist = nullptr;    // solve order (lpt.cuh): bucket counts, cursors, order
  int* lpt_cursor = nullptr;
  int* lpt_order = nullptr;
  bool use_order = false;     // the order was built for this step's radius solves
  int rp_grid = 1;
  int rp_grid_tight = 1;  // the same of the kernel for launches with stiff bubbles
  int rp_grid_full = 1;  // one lane per bubble, up to the occupancy limit
  int rp_blocks_req = 0;  // crp_set_tuning (0: rp_grid_full)
  int supp[3][6];
  crp_stats stats{};
  int64_t launches = 0;
  // Profiling (crp_set_profiling): events around the FDTD launch of a step.
  bool prof_on = false, prof_pending = false;
  cudaEvent_t ev_f0 = nullptr, ev_f1 = nullptr;
  crp_status set_profiling(bool on) {
    if (on && !ev_f0) {
      if (cudaEventCreate(&ev_f0) != cudaSuccess || cudaEventCreate(&ev_f1) != cudaSuccess)
        return CRP_ERR_CUDA;
    }
    prof_on = on;
    return CRP_OK;
  }

  crp_status fail(crp_status s, const char* what, cudaError_t e = cudaSuccess) {
    err = what;
    if (e != cudaSuccess) err += std::string(": ") + cudaGetErrorString(e);
    return s;
  }
#define C3(call)                                                   \
  do {                                                             \
    cudaError_t e_ = (call);                                       \
    if (e_ != cudaSuccess) return fail(CRP_ERR_CUDA, #call, e_);   \
  } while (0)

  template <typename T>
  T* carve(size_t count, size_t& off, bool dry) {
    const size_t bytes = (count * sizeof(T) + 255) & ~size_t(255);
    T* p = dry ? nullptr : reinterpret_cast<T*>(pool + off);
    off += bytes;
    return p;
  }

  size_t layout(bool dry, int n) {
    size_t off = 0;
    for (int q = 0; q < 2; q++) {
      vx[q] = carve<double>(cells, off, dry);
      vy[q] = carve<double>(cells, off, dry);
      vz[q] = carve<double>(cells, off, dry);
      px[q] = carve<double>(cells, off, dry);
      py[q] = carve<double>(cells, off, dry);
      pz[q] = carve<double>(cells, off, dry);
    }
    for (int q = 0; q < 3; q++) fg[q] = carve<double>(cells, off, dry);
    d_src = carve<short>(cells, off, dry);
    const int FX = g.f.X, FY = g.f.Y, FZ = g.f.Z;
    d_fac = carve<double>(4 * (size_t)(FX + 3 + FY + 3 + FZ + 3), off, dry);
    d_elem = carve<double>(2 * (size_t)std::max(elem_n, 1), off, dry);
    elem_p = carve<double>((size_t)std::max(elem_n, 1) * (n > 0 ? 1 : d3::kElemBatch), off, dry);
    scratch = carve<double>((size_t)(FX + 3) * (FY + 3) * (FZ + 3), off, dry);
    d_sc = carve<d3::Scalars3>(1, off, dry);
    bub.n = n;
    double** dp[] = {&bub.x, &bub.y, &bub.z, &bub.R0, &bub.n_B, &bub.R_t, &bub.R_p, &bub.R_pn, &bub.R_n, &bub.R_nn,
                     &bub.d1_R_p, &bub.d1_R_n, &bub.PG_p, &bub.PG_n, &bub.PL_p, &bub.PL_n, &bub.PL_m, &bub.Q_B,
                     &bub.dt, &bub.dt_n, &bub.re, &bub.re_n, &bub.vbx, &bub.vby, &bub.vbz};
    for (double** p : dp) *p = carve<double>(std::max(n, 1), off, dry);
    bub.contrib = carve<double>(8 * (size_t)std::max(n, 1), off, dry);
    int** ip[] = {&bub.ibmx, &bub.ibmy, &bub.ibmz, &bub.ibnx, &bub.ibny, &bub.ibnz, &bub.bin, &bub.nsub, &bub.pos};
    for (int** p : ip) *p = carve<int>(std::max(n, 1), off, dry);
    if (n > 0) {
      nbins = (FX + 3) * (FY + 3) * (FZ + 3);
      bin_count = carve<int>(nbins, off, dry);
      bin_start = carve<int>(nbins + 1, off, dry);
      bin_idx = carve<int>(std::max(n, 1), off, dry);
      bin_partial = carve<int>((nbins + d3::kScan - 1) / d3::kScan + 1, off, dry);
      tiles.nx = (FX + 2 + d3::kTile3X - 1) / d3::kTile3X;
      tiles.ny = (FY + 2 + d3::kTile3Y - 1) / d3::kTile3Y;
      tiles.nz = (FZ + 2 + d3::kTile3Z - 1) / d3::kTile3Z;
      tiles.last = carve<int>((size_t)tiles.nx * tiles.ny * tiles.nz, off, dry);
      tiles.list = carve<int>((size_t)tiles.nx * tiles.ny * tiles.nz, off, dry);
      lpt_hist = carve<int>(kLptBuckets, off, dry);
      lpt_cursor = carve<int>(kLptBuckets, off, dry);
      lpt_order = carve<int>(n, off, dry);
    }
    return off;
  }

  template <typename P>
  typename P::V vview(void* p) const;
  template <typename A>
  A view(void* p) const;

  crp_status create(const crp_config& c, const crp_bubbles_in* bin, void* user_stream);
  crp_status step_once();
  // Steps without bubbles, queued back to back: `left` more follow in this call.
  // Nothing the host decides depends on their scalars; finish_plain reads those of the
  // last step (a non-finite pressure stays non-finite in the linear step).
  bool plain_ok() const { return bub.n == 0 && !prof_on && stats.steps > 0; }
  int elem_next = 0, elem_made = 0;  // steps of the current batch of element pressures used and evaluated
  crp_status queue_plain(int left);
  crp_status finish_plain();
  void rotate() {
    cur_v ^= 1;
    cur_p ^= 1;
    const int a = fg_a, b = fg_b, c = fg_c;
    fg_a = c;  // predicted f_g
    fg_b = a;
    fg_c = b;
  }
  template <typename P>
  crp_status launch_fdtd(const double* elem);
  template <typename P>
  crp_status launch_move();
  template <typename P>
  auto radius_kernel(bool tight) const {
    return cfg.ext_rp_scheme == CRP_RP_RK45 ? d3::radius3<P, true, false>
           : tight                          ? d3::radius3<P, false, true>
                                            : d3::radius3<P, false, false>;
  }
  template <typename P>
  crp_status launch_radius(int done);
  template <typename P>
  crp_status launch_couple(bool pressure);
  d3::Tiles3 tiles{};
  int64_t coupling = 0;  // couplings so far: steps whose Picard loop ran
  int64_t reach[3]{};    // oldest coupling in the void fraction of the last three steps (Tiles3)
  int64_t oldest() const { return std::min(reach[0], std::min(reach[1], reach[2])); }
  // The active tiles of the next couplings of this step, from the current bins;
  // now: the bubbles' box.
  crp_status mark_tiles(const int now[6]);
  crp_status build_bins();
  crp_status build_order();
  cudaError_t begin_step(double t0, double t1) {
    d3::step_begin3<<<std::max(1, (elem_n + d3::kBeginThreads3 - 1) / d3::kBeginThreads3), d3::kBeginThreads3, 0,
                      stream>>>(g, d_sc, t0, t1, elem_n, elem_p);
    return cudaGetLastError();
  }
  void bubble_box(int box[6]) const;
  static double as_double(unsigned long long b) {
    double d;
    std::memcpy(&d, &b, sizeof(d));
    return d;
  }
  crp_status read_field(crp_field w, double* host);
  crp_status read_bubbles(crp_bubble_field w, double* host);
  crp_status adjoint(const crp_objective* obj, double* J, double* grad_amp, double* grad_phase);
  void* adj_ws = nullptr;  // crp_adjoint's device workspace, kept between calls
  size_t adj_ws_bytes = 0;
  // Source cells (frame index, element) in frame order, and the focus the bowl's phases aim at.
  std::vector<long> src_list;
  std::vector<int> src_elem;
  double focus[3] = {0.0, 0.0, 0.0};
  crp_status set_elements(int n, const double* amp, const double* phase);
  ~Sim3Impl();
};

template <>
F64 Sim3Impl::view<F64>(void* p) const {
  return F64{(double*)p};
}
template <>
F32c Sim3Impl::view<F32c>(void* p) const {
  return F32c{(float2*)p};
}
template <>
F32 Sim3Impl::view<F32>(void* p) const {
  return F32{(float*)p};
}

Sim3Impl::~Sim3Impl() {
  if (adj_ws) cudaFree(adj_ws);
  if (ev_f0) cudaEventDestroy(ev_f0);
  if (ev_f1) cudaEventDestroy(ev_f1);
  if (pool) cudaFree(pool);
  if (h_sc) cudaFreeHost(h_sc);
  if (own_stream && stream) cudaStreamDestroy(stream);
}

// PML profile of one axis (init_sigma's closed forms, src/bubble_CUDA.cu:946-1205,
// with a PML at both ends): factors 1 - s and 1 / (1 + s) of the faces
// (index n + 1, n in [-1, N+1]) and cells (index n, n in [0, N+1]).
static void axis_factors(int N, int npml, double h, double sig, int order, double s4, std::vector<double>& va,
                         std::vector<double>& vb, std::vector<double>& pa, std::vector<double>& pb) {
  std::vector<double> m(N + 2, 0.0), fc(N + 3, 0.0);
  const double smax = -std::log(sig) * 0.5 * ((double)order + 1.0) / (h * (double)npml);
  for (int n = 1; n <= std::min(N, npml); n++)
    m[n] = smax * std::pow(((double)(npml - n + 1) - 0.5) / ((double)npml), (double)order);
  for (int n = std::max(1, N - npml + 1); n <= N; n++)
    m[n] = smax * std::pow(((double)(n - N + npml) - 0.5) / ((double)npml), (double)order);
  for (int n = 0; n <= std::min(N, npml - 1); n++)
    fc[n + 1] = smax * std::pow(((double)(npml - n)) / ((double)npml), (double)order);
  for (int n = std::max(0, N - npml + 1); n <= N; n++)
    fc[n + 1] = smax * std::pow(((double)(n - N + npml)) / ((double)npml), (double)order);
  va.resize(N + 3);
  vb.resize(N + 3);
  pa.resize(N + 3, 1.0);
  pb.resize(N + 3, 1.0);
  for (int q = 0; q < N + 3; q++) {
    const double s = s4 * fc[q];  // (c + c) / 2 * dt / 2 * sigma_n
    va[q] = 1.0 - s;
    vb[q] = 1.0 / (1.0 + s);
  }
  for (int q = 0; q < N + 2; q++) {
    const double s = s4 * m[q];
    pa[q] = 1.0 - s;
    pb[q] = 1.0 / (1.0 + s);
  }
}

crp_status Sim3Impl::create(const crp_config& c, const crp_bubbles_in* bin, void* user_stream) {
  cfg = c;
  const int X = c.grid_x, Y = c.grid_y, Z = c.ext_grid_z;
  if (X < 4 || Y < 4 || Z < 4 || !(c.grid_lx > 0) || !(c.grid_ly > 0) || !(c.ext_grid_lz > 0))
    return fail(CRP_ERR_INVALID, "3-D grid needs at least 4 cells and a positive length per axis");
  if (!(c.pml_x0 && c.pml_x1 && c.pml_y0 && c.pml_y1 && c.ext_pml_z0 && c.ext_pml_z1))
    return fail(CRP_ERR_UNSUPPORTED, "the 3-D path implements a PML on all six faces");
  if (c.tr_cylindrical) return fail(CRP_ERR_UNSUPPORTED, "3-D grids are Cartesian (transducer.cylindrical = 0)");
  if (c.sim_order != 2 || c.sim_smooth_delta_band != 2)
    return fail(CRP_ERR_UNSUPPORTED, "simulation.order = 2 and smooth_delta_band = 2 only");
  if (c.ext_precision != CRP_PREC_FP64 && c.ext_precision != CRP_PREC_MIXED)
    return fail(CRP_ERR_INVALID, "ext.precision must be fp64 or mixed");
  if (c.ext_rp_scheme != CRP_RP_REF && c.ext_rp_scheme != CRP_RP_RK45)
    return fail(CRP_ERR_INVALID, "ext.rp_scheme must be ref or rk45");
  if ((long long)(X + 4) * (Y + 4) * (Z + 4) >= (1ll << 31))
    return fail(CRP_ERR_UNSUPPORTED, "3-D frame of 2^31 cells or more");
  mixed = c.ext_precision == CRP_PREC_MIXED;
  picard_tol = c.ext_picard_tol > 0.0 ? c.ext_picard_tol : (mixed ? 1.0e-5 : (double)1.0e-7f);
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(CRP_ERR_NO_DEVICE, "no CUDA device");
  C3(cudaGetDevice(&device));
  C3(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  if (user_stream) {
    stream = (cudaStream_t)user_stream;
  } else {
    C3(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    own_stream = true;
  }
  const double pi = std::acos(-1.0);
  d3::Frame3 f{X, Y, Z, ((X + 4) + 31) / 32 * 32};
  g.f = f;
  g.dx = (double)c.grid_lx / (double)X;
  g.dy = (double)c.grid_ly / (double)Y;
  g.dz = (double)c.ext_grid_lz / (double)Z;
  g.rdx = 1.0 / g.dx;
  g.rdy = 1.0 / g.dy;
  g.rdz = 1.0 / g.dz;
  g.rho_inf = c.ext_rho_inf;
  g.c_inf = c.ext_c_inf;
  g.P_inf = c.ext_p_inf;
  g.dt = c.sim_cfl * std::min(g.dx, std::min(g.dy, g.dz)) / g.c_inf;
  g.dt_rho = g.dt / g.rho_inf;
  g.s3p = g.dt * g.rho_inf * g.c_inf * g.c_inf;
  g.px0 = c.pml_grid_number;
  g.px1 = X - c.pml_grid_number + 1;
  g.omega = 2.0 * pi * c.tr_freq;
  g.pamp = g.rho_inf * g.c_inf * c.tr_amp;
  g.period = (double)(c.tr_on_wave + c.tr_off_wave) / c.tr_freq;
  g.on_time = (double)c.tr_on_wave / c.tr_freq;
  g.ramp_time = c.ext_ramp_cycles / c.tr_freq;
  cells = (size_t)f.pitch * (Y + 4) * (Z + 4);

  // Source: the bowl's elements (Fibonacci points on the lower hemisphere) and
  // the shell cells, each with its nearest element.
  elem_n = std::max(0, c.ext_array_elements);
  std::vector<double> ex(elem_n), ey(elem_n), ez(elem_n), eamp(elem_n, 1.0), eph(elem_n, 0.0);
  std::vector<short> src(cells, 0);
  {
    const double Ra = c.ext_array_radius;
    const double cx = 0.5 * X * g.dx, cy = 0.5 * Y * g.dy, cz = 0.5 * Z * g.dz;
    const double golden = pi * (3.0 - std::sqrt(5.0));
    const double fx = cx + c.ext_array_focus_dx;
    focus[0] = fx;
    focus[1] = cy;
    focus[2] = cz;
    if (elem_n > 32767) return fail(CRP_ERR_UNSUPPORTED, "more than 32767 array elements");
    for (int e = 0; e < elem_n; e++) {
      const double ct = -((double)e + 0.5) / (double)elem_n;
      const double st = std::sqrt(std::max(0.0, 1.0 - ct * ct));
      const double fph = golden * (double)e;
      ex[e] = cx + Ra * st * std::cos(fph);
      ey[e] = cy + Ra * st * std::sin(fph);
      ez[e] = cz + Ra * ct;
      const double d = std::sqrt((ex[e] - fx) * (ex[e] - fx) + (ey[e] - cy) * (ey[e] - cy) + (ez[e] - cz) * (ez[e] - cz));
      eph[e] = std::fmod(g.omega * d / g.c_inf, 2.0 * pi);
      if (c.ext_array_phases == 1) {
        uint32_t w[4];
        philox_block(c.ext_array_seed, (uint64_t)e, 2u, w);
        eph[e] = 2.0 * pi * (((double)w[0] + 0.5) / 4294967296.0);
      }
    }
    if (elem_n > 0) {
      const double half = 0.5 * g.dx;
      for (int k = 1; k <= Z; k++)
        for (int j = 1; j <= Y; j++)
          for (int i = 1; i <= X; i++) {
            const double xc = ((double)i - 0.5) * g.dx - cx, yc = ((double)j - 0.5) * g.dy - cy,
                         zc = ((double)k - 0.5) * g.dz - cz;
            const double r = std::sqrt(xc * xc + yc * yc + zc * zc);
            if (!(zc < 0.0) || !(std::fabs(r - Ra) <= half)) continue;
            int best = 0;
            double bd = 1e300;
            for (int e = 0; e < elem_n; e++) {
              const double dxe = ex[e] - cx - xc, dye = ey[e] - cy - yc, dze = ez[e] - cz - zc;
              const double dd = dxe * dxe + dye * dye + dze * dze;
              if (dd < bd) bd = dd, best = e;
            }
            src[f.idx(i, j, k)] = (short)(best + 1);
            src_list.push_back(f.idx(i, j, k));
            src_elem.push_back(best);
            src_cells++;
          }
    }
  }
  // Bubbles: explicit (with z), or seeded from the [ext] keys.
  std::vector<double> bx, by, bz, br0, bnb;
  if (c.bub_enable) {
    if (bin && bin->n > 0) {
      if (!bin->z) return fail(CRP_ERR_INVALID, "3-D bubbles need z coordinates");
      bx.assign(bin->x, bin->x + bin->n);
      by.assign(bin->y, bin->y + bin->n);
      bz.assign(bin->z, bin->z + bin->n);
      br0.assign(bin->r0, bin->r0 + bin->n);
      bnb.assign(bin->n_b, bin->n_b + bin->n);
    } else if (c.ext_bubble_count > 0) {
      const int n = c.ext_bubble_count;
      bx.resize(n);
      by.resize(n);
      bz.resize(n);
      br0.resize(n);
      bnb.resize(n);
      const crp_status st = crp_seed_bubbles3(&c, bx.data(), by.data(), bz.data(), br0.data(), bnb.data());
      if (st != CRP_OK) return fail(st, "bubble seeding failed");
    }
  }
  const int nb = (int)bx.size();
  pool_bytes = layout(true, nb);
  C3(cudaMalloc(&pool, pool_bytes));
  layout(false, nb);
  C3(cudaMemsetAsync(pool, 0, pool_bytes, stream));
  C3(cudaMallocHost(&h_sc, sizeof(d3::Scalars3)));
  std::memset(h_sc, 0, sizeof(d3::Scalars3));
  // PML factors: x faces, y faces, z faces (N+3 each), then x, y, z cells.
  {
    std::vector<double> va[3], vb[3], pa[3], pb[3];
    const double s4 = (g.c_inf + g.c_inf) * 0.5 * 0.5 * g.dt;
    axis_factors(X, c.pml_grid_number, g.dx, c.pml_sigma, c.pml_order, s4, va[0], vb[0], pa[0], pb[0]);
    axis_factors(Y, c.pml_grid_number, g.dy, c.pml_sigma, c.pml_order, s4, va[1], vb[1], pa[1], pb[1]);
    axis_factors(Z, c.pml_grid_number, g.dz, c.pml_sigma, c.pml_order, s4, va[2], vb[2], pa[2], pb[2]);
    std::vector<double> blk;
    size_t off[12];
    int q = 0;
    for (auto* v : {&va[0], &vb[0], &va[1], &vb[1], &va[2], &vb[2], &pa[0], &pb[0], &pa[1], &pb[1], &pa[2], &pb[2]}) {
      off[q++] = blk.size();
      blk.insert(blk.end(), v->begin(), v->end());
    }
    if (blk.size() > 4 * (size_t)(X + 3 + Y + 3 + Z + 3)) return fail(CRP_ERR_INVALID, "PML factor block");
    C3(cudaMemcpyAsync(d_fac, blk.data(), sizeof(double) * blk.size(), cudaMemcpyHostToDevice, stream));
    const double** dst[12] = {&g.vax, &g.vbx, &g.vay, &g.vby, &g.vaz, &g.vbz,
                              &g.pax, &g.pbx, &g.pay, &g.pby, &g.paz, &g.pbz};
    for (int r = 0; r < 12; r++) *dst[r] = d_fac + off[r];
    C3(cudaStreamSynchronize(stream));
  }
  C3(cudaMemcpyAsync(d_src, src.data(), sizeof(short) * cells, cudaMemcpyHostToDevice, stream));
  g.src = d_src;
  if (elem_n > 0) {
    std::vector<double> ev(eamp);
    ev.insert(ev.end(), eph.begin(), eph.end());
    C3(cudaMemcpyAsync(d_elem, ev.data(), sizeof(double) * ev.size(), cudaMemcpyHostToDevice, stream));
    C3(cudaStreamSynchronize(stream));
  }
  g.elem_amp = d_elem;
  g.elem_phase = d_elem + std::max(elem_n, 1);
  // Bubble parameters shared with the 2-D path.
  bp.PL0 = c.bub_P0;
  bp.T0 = c.bub_T0;
  bp.gam = c.bub_gamma;
  bp.sig = c.bub_sigma;
  bp.mu = c.bub_mu;
  bp.rho = c.bub_rho;
  bp.K0 = c.bub_K0;
  derive_bubble_constants(bp);
  bp.dt0 = 0.1 * g.dt;
  bp.pi = pi;
  bp.pi4r3 = pi * 4.0 / 3.0;
  bp.dcx = 1.0 / 2.0;
  bp.dcy = 2.0 * pi / 2.0 * g.rdx;
  bp.dcz = 2.0 * pi / 2.0 * g.rdy;
  bp.step_cap = c.ext_rp_step_cap;
  bp.rk_rtol = c.ext_rp_tol > 0.0 ? c.ext_rp_tol : kRk45DefaultTol;
  bp.reuse = c.ext_rp_reuse ? 1 : 0;
  for (int q = 0; q < 3; q++) supp[q][0] = supp[q][1] = supp[q][2] = 1, supp[q][3] = supp[q][4] = supp[q][5] = 0;
  if (nb > 0) {
    std::vector<double> zeros(nb, 0.0), dt0(nb, bp.dt0), pg0(nb);
    for (int k = 0; k < nb; k++) pg0[k] = c.bub_P0 + 2.0 * c.bub_sigma / br0[k];
    auto up = [&](double* d, const std::vector<double>& h) {
      return cudaMemcpyAsync(d, h.data(), sizeof(double) * nb, cudaMemcpyHostToDevice, stream);
    };
    C3(up(bub.x, bx));
    C3(up(bub.y, by));
    C3(up(bub.z, bz));
    C3(up(bub.R0, br0));
    C3(up(bub.n_B, bnb));
    for (double* d : {bub.R_t, bub.R_p, bub.R_pn, bub.R_n, bub.R_nn}) C3(up(d, br0));
    for (double* d : {bub.PG_p, bub.PG_n}) C3(up(d, pg0));
    for (double* d : {bub.dt, bub.dt_n}) C3(up(d, dt0));
    C3(cudaStreamSynchronize(stream));
    C3(begin_step(0.0, 0.0));
    d3::index3_kernel<<<(nb + 255) / 256, 256, 0, stream>>>(g, bub, d_sc);
    C3(cudaGetLastError());
    {
      const crp_status bs = build_bins();
      if (bs != CRP_OK) return bs;
    }
    // Initial void fraction (calculate_void_fraction at set-up, src/bubble_CUDA.cu:180-187):
    // every bubble's contributions at R0, gathered per cell; the history
    // buffers start equal to it.
    d3::contrib_init3<<<(nb + 255) / 256, 256, 0, stream>>>(g, bp, bub);
    C3(cudaGetLastError());
    C3(cudaMemsetAsync(tiles.last, 0xc0, sizeof(int) * tiles.nx * tiles.ny * tiles.nz, stream));  // never touched
    C3(cudaMemcpyAsync(h_sc, d_sc, sizeof(d3::Scalars3), cudaMemcpyDeviceToHost, stream));
    C3(cudaStreamSynchronize(stream));
    int box[6];
    bubble_box(box);
    {
      const crp_status ts = mark_tiles(box);
      if (ts != CRP_OK) return ts;
    }
    const crp_status st = mixed ? launch_couple<d3::PMix>(false) : launch_couple<d3::P64>(false);
    if (st != CRP_OK) return st;
    const size_t bytes = sizeof(double) * cells;
    C3(cudaMemcpyAsync(fg[fg_b], fg[fg_a], bytes, cudaMemcpyDeviceToDevice, stream));
    C3(cudaMemcpyAsync(fg[fg_c], fg[fg_a], bytes, cudaMemcpyDeviceToDevice, stream));
    for (int q = 0; q < 3; q++) std::memcpy(supp[q], box, sizeof(box));
  }
  for (int tight = 0; tight < 2; tight++) {
    int per_sm = 0;
    if (mixed)
      C3(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, radius_kernel<d3::PMix>(tight), d3::kRpThreads3, 0));
    else
      C3(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, radius_kernel<d3::P64>(tight), d3::kRpThreads3, 0));
    (tight ? rp_grid_tight : rp_grid_full) =
        std::max(1, std::min(sms * std::max(per_sm, 1), (nb + d3::kRpThreads3 - 1) / d3::kRpThreads3));
  }
  rp_grid = rp_grid_full;
  C3(cudaStreamSynchronize(stream));
  return CRP_OK;
}

// Cells whose void fraction the bubbles' stencils reach: their ibn box
// widened by one (the stencil's second point) and clipped to the frame's
// cells [0, N+1].
void Sim3Impl::bubble_box(int box[6]) const {
  const d3::Scalars3& s = *h_sc;
  const int N[3] = {g.f.X, g.f.Y, g.f.Z};
  for (int a = 0; a < 3; a++) {
    box[a] = std::max(0, s.box[a]);
    box[a + 3] = std::min(N[a] + 1, s.box[a + 3] + 1);
  }
}

static void box_union(int out[6], const int a[6], const int b[6]) {
  const bool ea = a[0] > a[3] || a[1] > a[4] || a[2] > a[5];
  const bool eb = b[0] > b[3] || b[1] > b[4] || b[2] > b[5];
  if (ea) {
    std::memcpy(out, b, 6 * sizeof(int));
    return;
  }
  if (eb) {
    std::memcpy(out, a, 6 * sizeof(int));
    return;
  }
  for (int q = 0; q < 3; q++) {
    out[q] = std::min(a[q], b[q]);
    out[q + 3] = std::max(a[q + 3], b[q + 3]);
  }
}

crp_status Sim3Impl::build_bins() {
  const int n = bub.n;
  C3(cudaMemsetAsync(bin_count, 0, sizeof(int) * nbins, stream));
  d3::bin3_count<<<(n + 255) / 256, 256, 0, stream>>>(bub.bin, n, bin_count);
  const int nparts = (nbins + d3::kScan - 1) / d3::kScan;
  d3::bin3_scan<<<nparts, d3::kScan, 0, stream>>>(bin_count, bin_start, bin_partial, nbins);
  d3::bin3_partials<<<1, d3::kScan, 0, stream>>>(bin_partial, nparts);
  d3::bin3_add<<<(nbins + 1 + 255) / 256, 256, 0, stream>>>(bin_start, bin_partial, nbins, nparts);
  d3::bin3_fill<<<(n + 255) / 256, 256, 0, stream>>>(bub.bin, n, bin_start, bin_count, bin_idx);
  d3::bin3_sort<<<(nbins + 255) / 256, 256, 0, stream>>>(bin_start, bin_idx, nbins);
  C3(cudaMemsetAsync(bub.pos, 0xff, sizeof(int) * n, stream));
  // Every bubble lies in some bin (the frame holds every cell index a bubble
  // inside the grid can have); those outside give -1 and no contributions.
  C3(cudaMemcpyAsync(&h_sc->next, bin_partial + nparts, sizeof(int), cudaMemcpyDeviceToHost, stream));
  C3(cudaStreamSynchronize(stream));
  const int total = h_sc->next;
  if (total > 0) d3::bin3_pos<<<(total + 255) / 256, 256, 0, stream>>>(bin_idx, total, bub.pos);
  C3(cudaGetLastError());
  launches += 7;
  bins_stale = false;
  return CRP_OK;
}

template <typename P>
crp_status Sim3Impl::launch_fdtd(const double* elem) {
  using V = typename P::V;
  using S = typename P::S;
  using G = typename P::G;
  const int nv = cur_v ^ 1, np = cur_p ^ 1;
  d3::Fdtd3Args<P> a;
  a.vx_old = view<V>(vx[cur_v]);
  a.vy_old = view<V>(vy[cur_v]);
  a.vz_old = view<V>(vz[cur_v]);
  a.vx_new = view<V>(vx[nv]);
  a.vy_new = view<V>(vy[nv]);
  a.vz_new = view<V>(vz[nv]);
  a.pnx = view<S>(px[cur_p]);
  a.pny = view<S>(py[cur_p]);
  a.pnz = view<S>(pz[cur_p]);
  a.px = view<S>(px[np]);
  a.py = view<S>(py[np]);
  a.pz = view<S>(pz[np]);
  a.fgA = view<G>(fg[fg_a]);
  a.fgB = view<G>(fg[fg_b]);
  a.fgC = view<G>(fg[fg_c]);
  a.rho_const = stats.steps == 0 ? 1 : 0;
  a.residual = &d_sc->residual;
  a.bubbles = bub.n > 0 ? 1 : 0;
  std::memcpy(a.supp, supp, sizeof(a.supp));
  a.tiles = tiles;
  a.oldest = (int)oldest();
  a.elem_p = elem;
  const int sx = (g.f.X + d3::kCols3 - 1) / d3::kCols3, sy = (g.f.Y + d3::kRows3 - 1) / d3::kRows3;
  const int planes = march3_planes(g.f.Z, (long)sx * sy, sms);
  const dim3 block(32, d3::kRows3), grid(sx, sy, (g.f.Z + planes - 1) / planes);
  int u[6], w[6];
  box_union(w, supp[0], supp[1]);
  box_union(u, w, supp[2]);
  const bool cloud = u[0] <= u[3] && (double)(u[3] - u[0] + 1) * (u[4] - u[1] + 1) * (u[5] - u[2] + 1) >
                                         d3::kCloudShare3 * g.f.X * g.f.Y * g.f.Z;
  if (prof_on) C3(cudaEventRecord(ev_f0, stream));
  if (cloud)
    d3::fdtd3<P, true><<<grid, block, 0, stream>>>(g, a, planes);
  else
    d3::fdtd3<P, false><<<grid, block, 0, stream>>>(g, a, planes);
  C3(cudaGetLastError());
  if (prof_on) {
    C3(cudaEventRecord(ev_f1, stream));
    prof_pending = true;
  }
  launches++;
  stats.fdtd_launches++;
  return CRP_OK;
}

template <typename P>
crp_status Sim3Impl::launch_move() {
  using V = typename P::V;
  d3::move3<V><<<(bub.n + 255) / 256, 256, 0, stream>>>(g, bp, bub, view<V>(vx[cur_v]), view<V>(vy[cur_v]),
                                                         view<V>(vz[cur_v]), d_sc);
  C3(cudaGetLastError());
  launches++;
  return CRP_OK;
}

crp_status Sim3Impl::build_order() {
  const int n = bub.n;
  lpt_count<<<(n + 255) / 256, 256, 0, stream>>>(bub.nsub, n, lpt_hist);
  lpt_scan<<<1, 32, 0, stream>>>(lpt_hist, lpt_cursor);
  lpt_scatter<<<(n + kLptScatterThreads - 1) / kLptScatterThreads, kLptScatterThreads, 0, stream>>>(
      bub.nsub, n, lpt_cursor, lpt_order);
  C3(cudaGetLastError());
  launches += 3;
  return CRP_OK;
}

template <typename P>
crp_status Sim3Impl::launch_radius(int done) {
  using S = typename P::S;
  const int reuse = bp.reuse && done > 0 ? 1 : 0;
  const int* order = use_order ? lpt_order : nullptr;
  C3(cudaMemsetAsync(&d_sc->next, 0, sizeof(int), stream));
  const bool tight = h_sc->substep_max >= d3::kTightSubsteps3;
  const auto kernel = radius_kernel<P>(tight);
  const int grid = tight && cfg.ext_rp_scheme != CRP_RP_RK45 ? std::min(rp_grid, rp_grid_tight) : rp_grid;
  kernel<<<grid, d3::kRpThreads3, 0, stream>>>(g, bp, bub, view<S>(px[cur_p]), view<S>(py[cur_p]), view<S>(pz[cur_p]),
                                               d_sc, reuse, order);
  C3(cudaGetLastError());
  launches++;
  return CRP_OK;
}

crp_status Sim3Impl::mark_tiles(const int now[6]) {
  int u[6], w[6], box[6];
  box_union(u, now, supp[0]);
  box_union(w, supp[1], supp[2]);
  box_union(box, u, w);
  C3(cudaMemsetAsync(&d_sc->tiles, 0, sizeof(int), stream));
  if (box[0] > box[3] || box[1] > box[4] || box[2] > box[5]) return CRP_OK;
  const int size[3] = {d3::kTile3X, d3::kTile3Y, d3::kTile3Z};
  d3::TileRange r;
  for (int q = 0; q < 3; q++) {
    r.lo[q] = box[q] / size[q];
    r.n[q] = box[q + 3] / size[q] - r.lo[q] + 1;
  }
  d3::mark_tiles<<<(r.n[0] * r.n[1] * r.n[2] + 7) / 8, 256, 0, stream>>>(g.f, bin_start, tiles, r, (int)coupling,
                                                                          (int)oldest(), &d_sc->tiles);
  C3(cudaGetLastError());
  launches++;
  return CRP_OK;
}

template <typename P>
crp_status Sim3Impl::launch_couple(bool pressure) {
  using V = typename P::V;
  using S = typename P::S;
  using G = typename P::G;
  d3::Couple3Args<P> a;
  a.vx = view<V>(vx[cur_v]);
  a.vy = view<V>(vy[cur_v]);
  a.vz = view<V>(vz[cur_v]);
  a.pnx = view<S>(px[cur_p ^ 1]);
  a.pny = view<S>(py[cur_p ^ 1]);
  a.pnz = view<S>(pz[cur_p ^ 1]);
  a.px = view<S>(px[cur_p]);
  a.py = view<S>(py[cur_p]);
  a.pz = view<S>(pz[cur_p]);
  a.fg = view<G>(fg[fg_a]);
  a.fgn = view<G>(fg[fg_b]);
  a.start = bin_start;
  a.contrib = bub.contrib;
  a.tiles = tiles;
  a.n_tiles = &d_sc->tiles;
  a.pressure = pressure ? 1 : 0;
  a.elem_p = elem_p;
  a.residual = &d_sc->residual;
  // The list's length is on the device: the blocks that the GPU holds stride over it.
  const int grid = std::min(tiles.nx * tiles.ny * tiles.nz, sms * 4);
  d3::couple3<P><<<grid, dim3(32, 8), 0, stream>>>(g, a);
  C3(cudaGetLastError());
  launches++;
  return CRP_OK;
}

crp_status Sim3Impl::queue_plain(int left) {
  auto advance = [&](double& t, double& carry) {
    const double s1 = t;
    t = t + g.dt + carry;
    const double s2 = t - s1;
    carry = g.dt + carry - s2;
  };
  if (elem_next == elem_made) {
    d3::ElemTimes et;
    elem_made = std::min(left + 1, d3::kElemBatch);
    elem_next = 0;
    double t = tstep, carry = tstepx;
    for (int q = 0; q < elem_made; q++) {
      advance(t, carry);
      et.t[q] = t;
    }
    if (elem_n > 0) {
      const dim3 grid((elem_n + d3::kBeginThreads3 - 1) / d3::kBeginThreads3, elem_made);
      d3::elem_batch<<<grid, d3::kBeginThreads3, 0, stream>>>(g, et, elem_n, elem_p);
      C3(cudaGetLastError());
      launches++;
    }
  }
  t_prev = tstep;
  advance(tstep, tstepx);
  if (left == 0) C3(cudaMemsetAsync(&d_sc->residual, 0, sizeof(unsigned long long), stream));
  const double* ep = elem_p + (size_t)elem_n * elem_next++;
  const crp_status st = mixed ? launch_fdtd<d3::PMix>(ep) : launch_fdtd<d3::P64>(ep);
  if (st != CRP_OK) return st;
  rotate();
  stats.steps++;
  stats.time = tstep;
  stats.picard_last = 0;
  return CRP_OK;
}

crp_status Sim3Impl::finish_plain() {
  C3(cudaMemcpyAsync(h_sc, d_sc, sizeof(d3::Scalars3), cudaMemcpyDeviceToHost, stream));
  C3(cudaStreamSynchronize(stream));
  const double res = as_double(h_sc->residual) / g.P_inf;
  if (std::isnan(res)) return fail(CRP_ERR_NONFINITE, "non-finite pressure");
  stats.residual_last = res;
  stats.rp_substeps_max = h_sc->substep_max;
  stats.rp_reused = (int64_t)h_sc->reused;
  stats.kernel_launches = launches;
  return CRP_OK;
}

crp_status Sim3Impl::step_once() {
  t_prev = tstep;
  const double s1 = tstep;
  tstep = tstep + g.dt + tstepx;
  const double s2 = tstep - s1;
  tstepx = g.dt + tstepx - s2;
  C3(begin_step(t_prev, tstep));
  launches++;
  crp_status st = mixed ? launch_fdtd<d3::PMix>(elem_p) : launch_fdtd<d3::P64>(elem_p);
  if (st != CRP_OK) return st;
  rotate();
  if (bub.n > 0) {
    st = mixed ? launch_move<d3::PMix>() : launch_move<d3::P64>();
    if (st != CRP_OK) return st;
  }
  C3(cudaMemcpyAsync(h_sc, d_sc, sizeof(d3::Scalars3), cudaMemcpyDeviceToHost, stream));
  C3(cudaStreamSynchronize(stream));
  if (prof_pending) {
    float ms = 0.0f;
    C3(cudaEventElapsedTime(&ms, ev_f0, ev_f1));
    stats.ms_fdtd += ms;
    prof_pending = false;
  }
  double res = as_double(h_sc->residual) / g.P_inf;
  int loop = 0;
  int bnow[6] = {1, 1, 1, 0, 0, 0};
  if (bub.n > 0) {
    bubble_box(bnow);
    if (h_sc->moved) bins_stale = true;
  }
  if (bub.n > 0 && res > picard_tol) {
    if (bins_stale) {
      st = build_bins();
      if (st != CRP_OK) return st;
    }
    coupling++;
    st = mark_tiles(bnow);
    if (st != CRP_OK) return st;
  }
  // Heaviest-first solve order from the last solves' sub-step counts, once
  // some bubble has needed more than the quiet phase's.
  use_order = bub.n > 0 && res > picard_tol && h_sc->substep_max > kLptMinSubsteps;
  if (use_order) {
    st = build_order();
    if (st != CRP_OK) return st;
  }
  if (bub.n > 0) {
    while (res > picard_tol) {
      if (loop >= cfg.ext_picard_cap) return fail(CRP_ERR_PICARD, "Picard iteration cap reached");
      loop++;
      C3(cudaMemsetAsync(&d_sc->residual, 0, sizeof(unsigned long long), stream));
      st = mixed ? launch_radius<d3::PMix>(loop - 1) : launch_radius<d3::P64>(loop - 1);
      if (st != CRP_OK) return st;
      st = mixed ? launch_couple<d3::PMix>(true) : launch_couple<d3::P64>(true);
      if (st != CRP_OK) return st;
      C3(cudaMemcpyAsync(h_sc, d_sc, sizeof(d3::Scalars3), cudaMemcpyDeviceToHost, stream));
      C3(cudaStreamSynchronize(stream));
      if (h_sc->err) return fail(CRP_ERR_RP_STEPS, "Rayleigh-Plesset sub-step cap reached");
      res = as_double(h_sc->residual) / g.P_inf;
      if (mixed && loop >= 3 && res > picard_tol && res < CRP_MIXED_STALL_RESIDUAL) {
        stats.picard_stalls++;
        break;
      }
    }
  }
  if (std::isnan(res)) return fail(CRP_ERR_NONFINITE, "non-finite pressure");
  int snow[6];
  if (loop > 0) {
    std::memcpy(snow, bnow, sizeof(snow));
  } else {
    int v1[6];
    box_union(v1, supp[0], supp[1]);
    box_union(snow, v1, supp[2]);
  }
  std::memcpy(supp[2], supp[1], sizeof(snow));
  std::memcpy(supp[1], supp[0], sizeof(snow));
  std::memcpy(supp[0], snow, sizeof(snow));
  const int64_t back = loop > 0 ? coupling : oldest();
  reach[2] = reach[1];
  reach[1] = reach[0];
  reach[0] = back;
  stats.steps++;
  stats.time = tstep;
  stats.picard_last = loop;
  stats.picard_total += loop;
  stats.picard_max = std::max(stats.picard_max, loop);
  stats.residual_last = res;
  stats.rp_substeps_max = h_sc->substep_max;
  stats.rp_reused = (int64_t)h_sc->reused;
  stats.kernel_launches = launches;
  return CRP_OK;
}

// Dense copies (x fastest) of a field's logical window: cells [0, N+1] per
// axis, staggered components one more along their axis from -1.
// crp_adjoint on the 3-D grid: the forward steps with the focal p0 recorded
// after each, the objective, then the reverse sweep of the kernels above.
crp_status Sim3Impl::adjoint(const crp_objective* obj, double* J, double* grad_amp, double* grad_phase) {
  if (!obj || obj->steps <= 0 || !(obj->focal_radius > 0.0))
    return fail(CRP_ERR_INVALID, "adjoint: steps > 0 and focal_radius > 0 are required");
  if ((grad_amp || grad_phase) && elem_n == 0)
    return fail(CRP_ERR_INVALID, "adjoint: gradients need ext.array_elements > 0");
  if (bub.n > 0) return fail(CRP_ERR_UNSUPPORTED, "adjoint: bubbles off only");
  const d3::Frame3& f = g.f;
  const int N = obj->steps;
  const double r = obj->focal_radius;
  // Focal box: cell centres within r of the focus along each axis.
  const int n3[3] = {f.X, f.Y, f.Z};
  const double h3[3] = {g.dx, g.dy, g.dz};
  int lo[3], hi[3];
  bool empty = false;
  for (int ax = 0; ax < 3; ax++) {
    lo[ax] = n3[ax] + 1;
    hi[ax] = 0;
    for (int m = 1; m <= n3[ax]; m++)
      if (std::fabs(((double)m - 0.5) * h3[ax] - focus[ax]) <= r) lo[ax] = std::min(lo[ax], m), hi[ax] = std::max(hi[ax], m);
    if (hi[ax] < lo[ax]) empty = true;
  }
  if (empty)
    for (int ax = 0; ax < 3; ax++) lo[ax] = hi[ax] = 1;  // one cell of weight 0
  const int bx = hi[0] - lo[0] + 1, by = hi[1] - lo[1] + 1, bz = hi[2] - lo[2] + 1;
  const size_t box_n = (size_t)bx * by * bz;
  std::vector<double> w(box_n, 0.0);
  if (!empty)
    for (int kk = 0; kk < bz; kk++)
      for (int jj = 0; jj < by; jj++)
        for (int ii = 0; ii < bx; ii++) {
          const int i = lo[0] + ii, j = lo[1] + jj, k = lo[2] + kk;
          const double x = ((double)i - 0.5) * g.dx - focus[0], y = ((double)j - 0.5) * g.dy - focus[1],
                       z = ((double)k - 0.5) * g.dz - focus[2];
          if (x * x + y * y + z * z > r * r) continue;
          if (std::binary_search(src_list.begin(), src_list.end(), f.idx(i, j, k))) continue;  // forced cells
          w[((size_t)kk * by + jj) * bx + ii] = g.dx * g.dy * g.dz;
        }
  const size_t hist_n = (size_t)N * box_n;
  if (hist_n * sizeof(double) > ((size_t)32 << 30))
    return fail(CRP_ERR_TOO_LARGE, "adjoint: focal history above 32 GiB (steps x focal cells)");
  const int ns = (int)src_list.size(), ns1 = std::max(ns, 1);
  // Two sets of six adjoint frames, per-source-cell gradients, weights,
  // history, objective per step; then the source cells' frame indices and
  // elements.
  const size_t n_fac = d3::kElemBatch * (2 + 2 * (size_t)elem_n);
  const size_t n_doubles = 12 * cells + 2 * (size_t)ns1 + box_n + hist_n + (size_t)N + n_fac;
  const size_t bytes = n_doubles * sizeof(double) + (size_t)ns1 * (sizeof(long) + sizeof(int));
  // The workspace is kept for the next call and released with the simulation.
  if (adj_ws_bytes < bytes) {
    if (adj_ws) {
      C3(cudaStreamSynchronize(stream));
      cudaFree(adj_ws);
      adj_ws = nullptr;
      adj_ws_bytes = 0;
    }
    if (cudaMalloc(&adj_ws, bytes) != cudaSuccess) {
      cudaGetLastError();
      adj_ws = nullptr;
      return fail(CRP_ERR_ALLOC, "adjoint: device memory");
    }
    adj_ws_bytes = bytes;
  }
  char* buf = static_cast<char*>(adj_ws);
  struct Drain {  // on every return: the queued work has finished
    cudaStream_t st;
    ~Drain() { cudaStreamSynchronize(st); }
  } guard{stream};
  double* base = reinterpret_cast<double*>(buf);
  d3::Adj3 fr[2];
  for (int s = 0; s < 2; s++) {
    double* b = base + (size_t)s * 6 * cells;
    fr[s] = d3::Adj3{b, b + cells, b + 2 * cells, b + 3 * cells, b + 4 * cells, b + 5 * cells};
  }
  double* gA = base + 12 * cells;
  double* gP = gA + ns1;
  double* d_w = gP + ns1;
  double* hist = d_w + box_n;
  double* d_Jn = hist + hist_n;
  double* d_env = d_Jn + N;
  double* d_sn = d_env + 2 * d3::kElemBatch;
  const d3::SourceFactors fac{d_env, d_sn, d_sn + (size_t)d3::kElemBatch * elem_n};
  long* d_cells = reinterpret_cast<long*>(base + n_doubles);
  int* d_el = reinterpret_cast<int*>(d_cells + ns1);
  C3(cudaMemsetAsync(buf, 0, n_doubles * sizeof(double), stream));
  C3(cudaMemcpyAsync(d_w, w.data(), sizeof(double) * box_n, cudaMemcpyHostToDevice, stream));
  if (ns > 0) {
    C3(cudaMemcpyAsync(d_cells, src_list.data(), sizeof(long) * ns, cudaMemcpyHostToDevice, stream));
    C3(cudaMemcpyAsync(d_el, src_elem.data(), sizeof(int) * ns, cudaMemcpyHostToDevice, stream));
  }
  const d3::Box3 box{lo[0], lo[1], lo[2], bx, by, bz, d_w};
  const int rb = (int)((box_n + 255) / 256);
  // Forward, recording the focal p0 after every step.
  std::vector<double> times((size_t)N + 1);
  times[0] = tstep;
  elem_next = elem_made = 0;
  for (int n = 1; n <= N; n++) {
    const bool plain = plain_ok();
    crp_status st = plain ? queue_plain(N - n) : step_once();
    if (plain && st == CRP_OK && n == N) st = finish_plain();
    if (st != CRP_OK) return st;
    double* out = hist + (size_t)(n - 1) * box_n;
    if (mixed)
      d3::adj3_record<F32c><<<rb, 256, 0, stream>>>(f, view<F32c>(px[cur_p]), view<F32c>(py[cur_p]),
                                                      view<F32c>(pz[cur_p]), box, out);
    else
      d3::adj3_record<F64><<<rb, 256, 0, stream>>>(f, view<F64>(px[cur_p]), view<F64>(py[cur_p]),
                                                     view<F64>(pz[cur_p]), box, out);
    C3(cudaGetLastError());
    launches++;
    times[n] = tstep;
  }
  // Objective.
  d3::adj3_objective<<<N, 256, 0, stream>>>(box, hist, d_Jn);
  C3(cudaGetLastError());
  std::vector<double> Jn(N);
  C3(cudaMemcpyAsync(Jn.data(), d_Jn, sizeof(double) * N, cudaMemcpyDeviceToHost, stream));
  C3(cudaStreamSynchronize(stream));
  double Jsum = 0.0;
  for (int n = 0; n < N; n++) Jsum += Jn[n];
  if (J) *J = g.dt * Jsum;
  // Reverse sweep: reverse step n reads frame set s and writes set s ^ 1.
  const int sx = (f.X + d3::kCols3 - 1) / d3::kCols3, sy = (f.Y + d3::kRows3 - 1) / d3::kRows3;
  const int planes = march3_planes(g.f.Z, (long)sx * sy, sms);
  const dim3 sblk(32, d3::kRows3), sgrid(sx, sy, (f.Z + planes - 1) / planes);
  const int sb = (ns + 63) / 64;
  const double two_dt = 2.0 * g.dt;
  d3::adj3_force<<<rb, 256, 0, stream>>>(f, fr[0], box, hist + (size_t)(N - 1) * box_n, two_dt);
  launches++;
  int s = 0;
  for (int n = N; n >= 1; n--, s ^= 1) {
    if (ns > 0) {
      const int q = (N - n) % d3::kElemBatch;
      if (q == 0) {
        d3::ElemTimes et{};
        const int m = std::min(n, d3::kElemBatch);
        for (int r = 0; r < m; r++) et.t[r] = times[n - r];
        const dim3 grid(elem_n / d3::kBeginThreads3 + 1, m);
        d3::adj3_factors<<<grid, d3::kBeginThreads3, 0, stream>>>(g, et, elem_n, fac);
        launches++;
      }
      const d3::SourceFactors t{fac.env + 2 * q, fac.sn + (size_t)q * elem_n, fac.cs + (size_t)q * elem_n};
      d3::adj3_source<<<sb, 64, 0, stream>>>(g, fr[s], d_cells, d_el, ns, t, gA, gP);
      launches++;
    }
    const double* p0 = n >= 2 ? hist + (size_t)(n - 2) * box_n : nullptr;
    d3::adj3_march<<<sgrid, sblk, 0, stream>>>(g, fr[s], fr[s ^ 1], box, p0, two_dt, planes);
    C3(cudaGetLastError());
    launches++;
  }
  if (elem_n > 0 && ns > 0) {
    std::vector<double> ca(ns), cp(ns);
    C3(cudaMemcpyAsync(ca.data(), gA, sizeof(double) * ns, cudaMemcpyDeviceToHost, stream));
    C3(cudaMemcpyAsync(cp.data(), gP, sizeof(double) * ns, cudaMemcpyDeviceToHost, stream));
    C3(cudaStreamSynchronize(stream));
    std::vector<double> sa(elem_n, 0.0), sp(elem_n, 0.0);
    for (int c = 0; c < ns; c++) {
      sa[src_elem[c]] += ca[c];
      sp[src_elem[c]] += cp[c];
    }
    if (grad_amp) std::copy(sa.begin(), sa.end(), grad_amp);
    if (grad_phase) std::copy(sp.begin(), sp.end(), grad_phase);
  } else {
    C3(cudaStreamSynchronize(stream));
    if (grad_amp) std::fill(grad_amp, grad_amp + elem_n, 0.0);
    if (grad_phase) std::fill(grad_phase, grad_phase + elem_n, 0.0);
  }
  stats.kernel_launches = launches;
  return CRP_OK;
}

crp_status Sim3Impl::read_field(crp_field w, double* host) {
  const d3::Frame3& f = g.f;
  void* buf = nullptr;
  int ilo = 0, jlo = 0, klo = 0, ihi = f.X + 1, jhi = f.Y + 1, khi = f.Z + 1;
  int kind = 0;  // 0 velocity/pressure storage, 1 void-fraction storage, 2 p0 = px + py + pz
  switch (w) {
    case CRP_FIELD_P0: kind = 2; break;
    case CRP_FIELD_PX: buf = px[cur_p]; break;
    case CRP_FIELD_PY: buf = py[cur_p]; break;
    case CRP_FIELD_PZ: buf = pz[cur_p]; break;
    case CRP_FIELD_VX: buf = vx[cur_v], ilo = -1; break;
    case CRP_FIELD_VY: buf = vy[cur_v], jlo = -1; break;
    case CRP_FIELD_VZ: buf = vz[cur_v], klo = -1; break;
    case CRP_FIELD_FG: buf = fg[fg_a], kind = 1; break;
    case CRP_FIELD_FGN: buf = fg[fg_b], kind = 1; break;
    case CRP_FIELD_FGM: buf = fg[fg_c], kind = 1; break;
    case CRP_FIELD_RHO_M: buf = fg[fg_a], kind = 3; break;
    default: return fail(CRP_ERR_UNSUPPORTED, "field not available on 3-D grids");
  }
  const int nx = ihi - ilo + 1, ny = jhi - jlo + 1, nz = khi - klo + 1;
  d3::read3<<<(nx * ny * nz + 255) / 256, 256, 0, stream>>>(
      f, kind, mixed ? 1 : 0, buf, px[cur_p], py[cur_p], pz[cur_p], ilo, jlo, klo, nx, ny, nz, g.rho_inf,
      stats.steps == 0 ? 1 : 0, scratch);
  C3(cudaGetLastError());
  C3(cudaMemcpyAsync(host, scratch, sizeof(double) * nx * ny * nz, cudaMemcpyDeviceToHost, stream));
  C3(cudaStreamSynchronize(stream));
  return CRP_OK;
}

crp_status Sim3Impl::read_bubbles(crp_bubble_field w, double* host) {
  const int n = bub.n;
  if (n == 0) return CRP_OK;
  const double* src = nullptr;
  const int* isrc = nullptr;
  switch (w) {
    case CRP_BUB_X: src = bub.x; break;
    case CRP_BUB_Y: src = bub.y; break;
    case CRP_BUB_Z: src = bub.z; break;
    case CRP_BUB_R_T: src = bub.R_t; break;
    case CRP_BUB_R_P: src = bub.R_p; break;
    case CRP_BUB_R_N: src = bub.R_n; break;
    case CRP_BUB_D1R: src = bub.d1_R_p; break;
    case CRP_BUB_PG: src = bub.PG_p; break;
    case CRP_BUB_PL_P: src = bub.PL_p; break;
    case CRP_BUB_PL_N: src = bub.PL_n; break;
    case CRP_BUB_PL_M: src = bub.PL_m; break;
    case CRP_BUB_DT: src = bub.dt; break;
    case CRP_BUB_RE: src = bub.re; break;
    case CRP_BUB_Q_B: src = bub.Q_B; break;
    case CRP_BUB_N_B: src = bub.n_B; break;
    case CRP_BUB_R0: src = bub.R0; break;
    case CRP_BUB_VX: src = bub.vbx; break;
    case CRP_BUB_VY: src = bub.vby; break;
    case CRP_BUB_VZ: src = bub.vbz; break;
    case CRP_BUB_IBM_X: isrc = bub.ibmx; break;
    case CRP_BUB_IBM_Y: isrc = bub.ibmy; break;
    case CRP_BUB_IBM_Z: isrc = bub.ibmz; break;
    case CRP_BUB_IBN_X: isrc = bub.ibnx; break;
    case CRP_BUB_IBN_Y: isrc = bub.ibny; break;
    case CRP_BUB_IBN_Z: isrc = bub.ibnz; break;
    case CRP_BUB_SUBSTEPS: isrc = bub.nsub; break;
    default: return fail(CRP_ERR_INVALID, "unknown bubble field");
  }
  if (src) {
    C3(cudaMemcpyAsync(host, src, sizeof(double) * n, cudaMemcpyDeviceToHost, stream));
    C3(cudaStreamSynchronize(stream));
    return CRP_OK;
  }
  std::vector<int> tmp(n);
  C3(cudaMemcpyAsync(tmp.data(), isrc, sizeof(int) * n, cudaMemcpyDeviceToHost, stream));
  C3(cudaStreamSynchronize(stream));
  for (int k = 0; k < n; k++) host[k] = (double)tmp[k];
  return CRP_OK;
}

crp_status Sim3Impl::set_elements(int n, const double* amp, const double* phase) {
  if (n != elem_n || n <= 0 || !amp || !phase) return fail(CRP_ERR_INVALID, "element count mismatch");
  std::vector<double> v(amp, amp + n);
  v.insert(v.end(), phase, phase + n);
  C3(cudaMemcpyAsync(d_elem, v.data(), sizeof(double) * v.size(), cudaMemcpyHostToDevice, stream));
  C3(cudaStreamSynchronize(stream));
  return CRP_OK;
}

// C-ABI glue used by sim.cu's entry points.
crp_status sim3_create(const crp_config* cfg, const crp_bubbles_in* bubbles, void* stream, Sim3Impl** out,
                       std::string* err) {
  Sim3Impl* s = new (std::nothrow) Sim3Impl();
  if (!s) return CRP_ERR_ALLOC;
  const crp_status st = s->create(*cfg, bubbles, stream);
  if (st != CRP_OK) {
    if (err) *err = s->err;
    delete s;
    return st;
  }
  *out = s;
  return CRP_OK;
}
void sim3_destroy(Sim3Impl* s) { delete s; }
crp_status sim3_step(Sim3Impl* s, int n) {
  s->elem_next = s->elem_made = 0;
  for (int k = 0; k < n; k++) {
    const bool plain = s->plain_ok();
    const crp_status st = plain ? s->queue_plain(n - k - 1) : s->step_once();
    if (st != CRP_OK) return st;
    if (plain && k == n - 1) return s->finish_plain();
  }
  return CRP_OK;
}
crp_status sim3_read_field(Sim3Impl* s, crp_field w, double* host) { return s->read_field(w, host); }
crp_status sim3_read_bubbles(Sim3Impl* s, crp_bubble_field w, double* host) { return s->read_bubbles(w, host); }
crp_status sim3_set_elements(Sim3Impl* s, int n, const double* amp, const double* phase) {
  return s->set_elements(n, amp, phase);
}
void sim3_dims(const Sim3Impl* s, crp_dims3* d) {
  d->nx = s->g.f.X + 2;
  d->ny = s->g.f.Y + 2;
  d->nz = s->g.f.Z + 2;
  d->num_bubbles = s->bub.n;
  d->dx = s->g.dx;
  d->dy = s->g.dy;
  d->dz = s->g.dz;
  d->dt = s->g.dt;
  d->source_cells = s->src_cells;
}
const crp_stats& sim3_stats(const Sim3Impl* s) { return s->stats; }
const char* sim3_error(const Sim3Impl* s) { return s->err.c_str(); }
crp_status sim3_set_profiling(Sim3Impl* s, int on) { return s->set_profiling(on != 0); }
void* sim3_stream(Sim3Impl* s) { return (void*)s->stream; }

// Snapshots: the device pool, and the host-side step state beside it.
struct HostState3 {
  int cur_v, cur_p, fg_a, fg_b, fg_c, bins_stale;
  double tstep, tstepx, t_prev;
  int supp[3][6];
  int64_t coupling, reach[3];
  crp_stats stats;
  d3::Scalars3 hsc;
};
size_t sim3_state_bytes(const Sim3Impl* s) { return s->pool_bytes; }
crp_status sim3_save_state(Sim3Impl* s, void* blob, std::vector<unsigned char>& host) {
  if (cudaMemcpyAsync(blob, s->pool, s->pool_bytes, cudaMemcpyDeviceToDevice, s->stream) != cudaSuccess ||
      cudaStreamSynchronize(s->stream) != cudaSuccess)
    return s->fail(CRP_ERR_CUDA, "state: device copy");
  HostState3 h{};
  h.cur_v = s->cur_v, h.cur_p = s->cur_p, h.fg_a = s->fg_a, h.fg_b = s->fg_b, h.fg_c = s->fg_c;
  h.bins_stale = s->bins_stale ? 1 : 0;
  h.tstep = s->tstep, h.tstepx = s->tstepx, h.t_prev = s->t_prev;
  std::memcpy(h.supp, s->supp, sizeof(h.supp));
  h.stats = s->stats;
  h.hsc = *s->h_sc;
  h.coupling = s->coupling;
  std::memcpy(h.reach, s->reach, sizeof(h.reach));
  host.resize(sizeof(HostState3));
  std::memcpy(host.data(), &h, sizeof(HostState3));
  return CRP_OK;
}
crp_status sim3_load_state(Sim3Impl* s, const void* blob, const std::vector<unsigned char>& host) {
  if (host.size() != sizeof(HostState3)) return s->fail(CRP_ERR_INVALID, "state: host part of the wrong size");
  HostState3 h;
  std::memcpy(&h, host.data(), sizeof(HostState3));
  if (cudaMemcpyAsync(s->pool, blob, s->pool_bytes, cudaMemcpyDeviceToDevice, s->stream) != cudaSuccess ||
      cudaStreamSynchronize(s->stream) != cudaSuccess)
    return s->fail(CRP_ERR_CUDA, "state: device copy");
  s->cur_v = h.cur_v, s->cur_p = h.cur_p, s->fg_a = h.fg_a, s->fg_b = h.fg_b, s->fg_c = h.fg_c;
  s->bins_stale = h.bins_stale != 0;
  s->tstep = h.tstep, s->tstepx = h.tstepx, s->t_prev = h.t_prev;
  std::memcpy(s->supp, h.supp, sizeof(h.supp));
  s->coupling = h.coupling;
  std::memcpy(s->reach, h.reach, sizeof(s->reach));
  const crp_stats keep = s->stats;
  s->stats = h.stats;
  s->stats.kernel_launches = keep.kernel_launches;
  s->stats.fdtd_launches = keep.fdtd_launches;
  s->stats.rp_launches = keep.rp_launches;
  s->stats.couple_launches = keep.couple_launches;
  s->stats.ms_fdtd = keep.ms_fdtd, s->stats.ms_rp = keep.ms_rp, s->stats.ms_couple = keep.ms_couple;
  s->stats.ms_other = keep.ms_other;
  *s->h_sc = h.hsc;
  return CRP_OK;
}
crp_status sim3_set_tuning(Sim3Impl* s, const crp_tuning* t) {
  if (t->fdtd_rows != 4 && t->fdtd_rows != 8 && t->fdtd_rows != 16)
    return s->fail(CRP_ERR_INVALID, "tuning: fdtd_rows must be 4, 8 or 16");
  if (t->rp_blocks < 0) return s->fail(CRP_ERR_INVALID, "tuning: rp_blocks must be >= 0");
  s->rp_blocks_req = t->rp_blocks;
  s->rp_grid = t->rp_blocks > 0 ? std::min(t->rp_blocks, s->rp_grid_full) : s->rp_grid_full;
  return CRP_OK;
}
crp_status sim3_adjoint(Sim3Impl* s, const crp_objective* obj, double* J, double* grad_amp, double* grad_phase) {
  return s->adjoint(obj, J, grad_amp, grad_phase);
}
void sim3_get_tuning(const Sim3Impl* s, crp_tuning* t) {
  t->fdtd_rows = 8;
  t->rp_blocks = s->rp_blocks_req;
  t->rp_blocks_max = s->rp_grid_full;
}
int sim3_device(const Sim3Impl* s) { return s->device; }

}  // namespace crp
