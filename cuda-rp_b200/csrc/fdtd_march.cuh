// One mixture step of the 2-D grid, fused: void-fraction prediction
// (store_variables, src/bubble_CUDA.cu:1160-1162), VelocityKernel with
// VelocityBoundaryKernel's faces (inc/bubble_CUDA_kernel.cuh:658-798),
// MixturePressureKernel with the predicted void fraction (:816-867) and the
// residual of calculate_pressure_field.
//
// A warp covers 64 columns, two adjacent ones per lane (16-byte accesses), and
// marches up a chunk of rows.  The row below stays in registers; the neighbours to
// the left and right are read again by the lane that needs them (the same cache
// lines) and the west face is formed twice, so that no lane waits for another.
// The next row's values are loaded before a row is computed.
//
// The void fraction takes part only where it can be nonzero: outside the support
// of the last three steps (FdtdArgs::supp) f_g, f_gn and f_gm are zero, so are the
// prediction and the rate term, and the density is rho_inf.  Chunks whose cells
// and neighbours lie outside move 64 bytes per cell instead of 96 and divide by
// nothing; bubble-free simulations have no others.
//
// Bound by the latency of its loads at 16 warps per SM (128 registers) and by the
// last, partly filled wave; cold, 1001 x 1531 without bubbles takes 23.8 us (64 bytes
// per cell: 4.1 TB/s), 41.3 before with 30 cells per warp staged through shared
// memory and 96 bytes per cell; 48 x 96 8.8 us, 19.6 before.
#pragma once

namespace crp {

constexpr int kMarchWarps = 4;  // warps per block, on consecutive chunks of one strip (shared rows hit L1)
constexpr int kMarchCols = 64;  // columns of a warp

// Resident blocks per SM the register budget is set for (128 registers): measured
// on 1001 x 1531 without bubbles and 1024 x 2048 with (us per pass): 4 blocks 26.0 and
// 40.1, 5 blocks (96 registers, more spilled) 29.4 and 43.1, 3 blocks 29.0 and 43.4.
constexpr int kMarchMinBlocks = 4;

// Where the pass leaves p0 of the previous step on the cells [i0, i0 + w) x [j0, j0 + h)
// (the focal history of the adjoint: 3 us per step less than a launch of its own).
struct FocalRecord {
  int i0, j0, w, h;
  double* out;  // null: nowhere
};

struct MarchRow {
  double2 x, y;           // px, py of the lane's two columns
  double xl, yl, xr, yr;  // and of the columns to the left and right
};

// Three forms: kPlain away from the x PML, the first and last row, the source row
// and any void fraction, of which it knows nothing; kEdges without void fraction;
// kVoid for everything.  Lane columns i and i + 1 (i odd, i <= X), rows j0..j1.
enum MarchForm { kPlain = 0, kEdges = 1, kVoid = 2 };
template <typename P, int FORM, bool REC>
__device__ __forceinline__ unsigned long long march_chunk(const GridParams& g, const FdtdArgs<P>& a,
                                                          const FocalRecord& rec, int i, int j0, int j1) {
  constexpr bool GEN = FORM >= kEdges, VOID = FORM == kVoid;
  using G = typename P::G;
  const Frame& f = g.f;
  const int X = f.X, Y = f.Y;
  const bool two = i + 1 <= X;
  const bool src_rows = GEN && g.source_row > 0 && src_pressure(g);
  const unsigned pitch = (unsigned)f.pitch;
  auto load = [&](unsigned k) -> MarchRow {
    MarchRow r;
    r.x = a.pnx.get2(k);
    r.y = a.pny.get2(k);
    r.xl = a.pnx.get(k - 1);
    r.yl = a.pny.get(k - 1);
    r.xr = a.pnx.get(k + 2);
    r.yr = a.pny.get(k + 2);
    return r;
  };
  // p0 of columns i - 1 .. i + 2 of an interior row j, with the boundary values of
  // MixtureBoundaryPressureKernel (p0_at): the source row, then the x ghost columns.
  auto pressures = [&](const MarchRow& r, int j, double* q) {
    q[0] = r.xl + r.yl;
    q[1] = r.x.x + r.y.x;
    q[2] = r.x.y + r.y.y;
    q[3] = r.xr + r.yr;
    if (src_rows && j == g.source_row) {
      q[0] = a.src.p_prev[max(i - 1, 1)];
      q[1] = a.src.p_prev[i];
      q[2] = a.src.p_prev[min(i + 1, X)];
      q[3] = a.src.p_prev[min(i + 2, X)];
    }
    if (i == 1) q[0] = g.pml_x0 ? 0.0 : q[1];
    if (i == X) q[2] = g.pml_x1 ? 0.0 : q[1];
    if (i + 1 == X) q[3] = g.pml_x1 ? 0.0 : q[2];
  };
  auto rho_of = [&](double fa) -> double { return a.rho_const ? g.rho_inf : (1.0 - fa) * g.rho_inf; };
  // dt / mean(rho) of a face, the same for both cells beside it and for every chunk:
  // dt_rho, the plain forms' value, where the mean is rho_inf (the quotient's last bit can
  // differ from it).
  auto face_factor = [&](double ra, double rb) -> double {
    const double m = (ra + rb) * 0.5, q = quotient(g.dt, m);
    return m == g.rho_inf ? g.dt_rho : q;
  };
  auto predict = [&](unsigned k) {  // a ghost cell's prediction
    a.fgC.put(k, G::stored(3.0 * a.fgA.get(k) - 3.0 * a.fgB.get(k) + a.fgC.get(k)));
  };
  auto predict_row = [&](unsigned k) {  // a ghost row's
    if (i == 1) predict(k - 1);
    predict(k);
    predict(k + 1);
    if (i + 1 == X) predict(k + 2);
  };
  // North face jf of column i + c after the y sections of VelocityBoundaryKernel
  // (:734-798): y0 wall or source, [ext] source row, y1 wall.  pre receives the y0
  // face before its source overwrites it (mirrored into row -1).
  auto vy_bounds = [&](int jf, int c, double v, double& pre) -> double {
    if (jf == 0 && !g.pml_y0) {
      if (!src_pressure(g)) v = 0.0;
      pre = v;
      if (g.source_row == 0 && src_velocity(g)) v = a.src.v[min(i + c, X)];
    }
    if (g.source_row > 0 && jf == g.source_row && src_velocity(g)) v = a.src.v[min(i + c, X)];
    if (jf == Y && !g.pml_y1) v = 0.0;
    return v;
  };
  unsigned k = (unsigned)j0 * pitch + (unsigned)(i + 1);  // row j0 - 1
  MarchRow cur = load(k);
  const double2 vyb = a.vy_old.get2(k);
  double pb[4], pc[4], rb[2], rc[4], fc[2];
  pressures(cur, j0 - 1, pb);
  if (VOID) {
    const double2 fb = a.fgA.get2(k);
    rb[0] = rho_of(fb.x);
    rb[1] = rho_of(fb.y);
    if (j0 == 1) predict_row(k);
  }
  k += pitch;  // row j0
  cur = load(k);
  pressures(cur, j0, pc);
  if (GEN && j0 == 1) {  // p0 of the y0 ghost row: PML, source, or the mirror of row 1
    const bool src = g.source_row == 0 && src_pressure(g);
#pragma unroll
    for (int c = 1; c < 3; c++)
      pb[c] = g.pml_y0 ? 0.0 : src ? a.src.p_prev[min(i + c - 1, X)] : pc[c];
  }
  if (VOID) {
    const double2 fa = a.fgA.get2(k);
    fc[0] = fa.x;
    fc[1] = fa.y;
    rc[0] = rho_of(a.fgA.get(k - 1));
    rc[1] = rho_of(fa.x);
    rc[2] = rho_of(fa.y);
    rc[3] = rho_of(a.fgA.get(k + 2));
  }
  double vyd[2];
  {
    const double vo[2] = {vyb.x, vyb.y};
    const double fa = g.vay[j0], fb = g.vby[j0];
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const double q = VOID ? face_factor(rb[c], rc[c + 1]) : g.dt_rho;
      vyd[c] = velocity_face_q(g, vo[c], pb[c + 1], pc[c + 1], q, fa, fb);
      if (GEN) {
        double pre = vyd[c];
        vyd[c] = vy_bounds(j0 - 1, c, vyd[c], pre);
        if (j0 == 1 && (c == 0 || two)) {
          a.vy_new.put(f.idx(i + c, 0), vyd[c]);
          if (!g.pml_y0) a.vy_new.put(f.idx(i + c, -1), pre);
        }
      }
    }
  }
  // Metrics of the three x faces and two cells; their PML factors are read per
  // row where there are any.
  double xu[3] = {0.0, 0.0, 0.0}, rxp[2] = {0.0, 0.0};
  if (g.cyl) {
#pragma unroll
    for (int c = 0; c < 3; c++) xu[c] = g.xu[i + c];
    rxp[0] = g.rxp[i];
    rxp[1] = g.rxp[i + 1];
  }
  const bool wall_w = i == 1 && !g.pml_x0;
  const bool wall_m = i == X && !g.pml_x1, wall_e = i + 1 == X && !g.pml_x1;
  MarchRow nxt = load(k + pitch);
  double2 vx2 = a.vx_old.get2(k), vy2 = a.vy_old.get2(k);
  double vxl = a.vx_old.get(k - 1);
  // f_g of the row above, f_gn and f_gm of this row, one row ahead as well.
  double2 fA2, fB2, fC2;
  double fAl, fAr;
  auto load_void = [&](unsigned q) {
    fA2 = a.fgA.get2(q + pitch);
    fAl = a.fgA.get(q + pitch - 1);
    fAr = a.fgA.get(q + pitch + 2);
    fB2 = a.fgB.get2(q);
    fC2 = a.fgC.get2(q);
  };
  if (VOID) load_void(k);
  unsigned long long res = 0ull;  // max |dp0| as a bit pattern (NaN sorts above every number)
#pragma unroll 1
  for (int j = j0; j <= j1; j++, k += pitch) {
    // The values of this row and of p in the next one are here or on their way;
    // those of one row further are requested now.
    const double2 vxo = vx2, vyo = vy2;
    const double vxw = vxl;
    const MarchRow up = nxt;
    if (j < j1) {
      nxt = load(k + 2 * pitch);
      vx2 = a.vx_old.get2(k + pitch);
      vy2 = a.vy_old.get2(k + pitch);
      vxl = a.vx_old.get(k + pitch - 1);
    }
    if (REC && (unsigned)(j - rec.j0) < (unsigned)rec.h) {
#pragma unroll
      for (int c = 0; c < 2; c++)
        if ((unsigned)(i + c - rec.i0) < (unsigned)rec.w) rec.out[(unsigned)(j - rec.j0) * (unsigned)rec.w + (unsigned)(i + c - rec.i0)] = pc[c + 1];
    }
    double pu[4], ru[4], fu[2], fgp[2], h[2] = {0.0, 0.0};
    pressures(up, j + 1, pu);
    if (GEN && j == Y) {  // p0 of the y1 ghost row: PML, or the mirror of row Y
#pragma unroll
      for (int c = 1; c < 3; c++) pu[c] = g.pml_y1 ? 0.0 : pc[c];
    }
    double qx[3] = {g.dt_rho, g.dt_rho, g.dt_rho}, qy[2] = {g.dt_rho, g.dt_rho};
    if (VOID) {
      const double2 fa = fA2, fB = fB2, fC = fC2;
      fu[0] = fa.x;
      fu[1] = fa.y;
      ru[0] = rho_of(fAl);
      ru[1] = rho_of(fa.x);
      ru[2] = rho_of(fa.y);
      ru[3] = rho_of(fAr);
      if (j < j1) load_void(k + pitch);
      fgp[0] = G::stored(3.0 * fc[0] - 3.0 * fB.x + fC.x);
      fgp[1] = G::stored(3.0 * fc[1] - 3.0 * fB.y + fC.y);
      a.fgC.put2(k, fgp[0], fgp[1]);  // the second is the ghost column where i = X
      if (i == 1) predict(k - 1);
      if (i + 1 == X) predict(k + 2);
#pragma unroll
      for (int c = 0; c < 3; c++) qx[c] = face_factor(rc[c], rc[c + 1]);
      qy[0] = face_factor(rc[1], ru[1]);
      qy[1] = face_factor(rc[2], ru[2]);
      // As void_rate_half.
#pragma unroll
      for (int c = 0; c < 2; c++)
        h[c] = 0.5 * quotient(quotient(-(fgp[c] - fc[c]), g.dt), 1.0 - 0.5 * (fgp[c] + fc[c]));
    }
    const double vo[3] = {vxw, vxo.x, vxo.y};
    double fx[3];
#pragma unroll
    for (int c = 0; c < 3; c++)
      fx[c] = velocity_face_q(g, vo[c], pc[c], pc[c + 1], qx[c], GEN ? g.vax[i + c] : 1.0, GEN ? g.vbx[i + c] : 1.0);
    if (wall_w) fx[0] = 0.0;
    if (wall_m) fx[1] = 0.0;
    if (wall_e) fx[2] = 0.0;
    const double vyv[2] = {vyo.x, vyo.y};
    double vyu[2], nx[2], ny[2];
    const double vay = g.vay[j + 1], vby = g.vby[j + 1], pay = g.pay[j], pby = g.pby[j];
#pragma unroll
    for (int c = 0; c < 2; c++) {
      vyu[c] = velocity_face_q(g, vyv[c], pc[c + 1], pu[c + 1], qy[c], vay, vby);
      if (GEN) {
        double pre;
        vyu[c] = vy_bounds(j, c, vyu[c], pre);
      }
      const double s1x = g.cyl ? fma(xu[c + 1], fx[c + 1], -__dmul_rn(xu[c], fx[c])) * g.rdx * rxp[c]
                               : (-fx[c] + fx[c + 1]) * g.rdx;
      const double s1y = (-vyd[c] + vyu[c]) * g.rdy;
      const double px = c ? cur.x.y : cur.x.x, py = c ? cur.y.y : cur.y.x;
      nx[c] = pressure_component(g, px, GEN ? g.pax[i + c] : 1.0, GEN ? g.pbx[i + c] : 1.0, s1x, h[c]);
      ny[c] = pressure_component(g, py, pay, pby, s1y, h[c]);
      double p0new = nx[c] + ny[c];
      if (src_rows && j == g.source_row) p0new = a.src.p_cur[min(i + c, X)];
      if (c == 0 || two) res = max(res, (unsigned long long)__double_as_longlong(fabs(pc[c + 1] - p0new)));
    }
    if (two) {
      a.vx_new.put2(k, fx[1], fx[2]);
      a.vy_new.put2(k, vyu[0], vyu[1]);
      a.px.put2(k, nx[0], nx[1]);
      a.py.put2(k, ny[0], ny[1]);
    } else {
      a.vx_new.put(k, fx[1]);
      a.vy_new.put(k, vyu[0]);
      a.px.put(k, nx[0]);
      a.py.put(k, ny[0]);
    }
    if (i == 1) a.vx_new.put(k - 1, fx[0]);  // the x0 face
    vyd[0] = vyu[0];
    vyd[1] = vyu[1];
    cur = up;
#pragma unroll
    for (int c = 0; c < 4; c++) pc[c] = pu[c];
    if (VOID) {
      fc[0] = fu[0];
      fc[1] = fu[1];
#pragma unroll
      for (int c = 0; c < 4; c++) rc[c] = ru[c];
    }
  }
  if (VOID && j1 == Y) predict_row(k);
  return res;
}

// REC: with the record (only without bubbles).
template <typename P, bool REC>
__global__ void __launch_bounds__(32 * kMarchWarps, kMarchMinBlocks) fdtd_march(const __grid_constant__ GridParams g,
                                                                  const FdtdArgs<P> a, const FocalRecord rec, int rows,
                                                                  int strips) {
  const int X = g.f.X, Y = g.f.Y;
  const int lane = threadIdx.x & 31;
  const int strip = blockIdx.x % strips, chunk = (blockIdx.x / strips) * kMarchWarps + (threadIdx.x >> 5);
  const int i0 = 1 + strip * kMarchCols, i1 = min(X, i0 + kMarchCols - 1), i = i0 + 2 * lane;
  const int j0 = 1 + chunk * rows, j1 = min(Y, j0 + rows - 1);
  if (j0 > Y) return;
  // Whether the warp's cells, widened by one (ghost cells count with the cells
  // beside them), meet a support box.
  bool fg = false;
  if (a.bubbles) {
    const int* s = a.dsupp ? a.dsupp : &a.supp[0][0];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const int b0 = s[4 * q], b1 = s[4 * q + 1], b2 = s[4 * q + 2], b3 = s[4 * q + 3];
      fg = fg || (b0 <= b2 && b1 <= b3 && b0 <= i1 + 1 && b2 >= i0 - 1 && b1 <= j1 + 1 && b3 >= j0 - 1);
    }
  }
  const bool edges = i0 <= g.px0 || i1 >= g.px1 || j0 == 1 || j1 == Y ||
                     (g.source_row >= j0 - 1 && g.source_row <= j1 + 1 && g.source_row > 0);
  unsigned long long res = 0ull;
  if (i <= X) {
    if (!REC && fg)
      res = march_chunk<P, kVoid, false>(g, a, rec, i, j0, j1);
    else if (edges)
      res = march_chunk<P, kEdges, REC>(g, a, rec, i, j0, j1);
    else
      res = march_chunk<P, kPlain, REC>(g, a, rec, i, j0, j1);
  }
  // Warp maximum, one atomic per warp with a nonzero residual.
  for (int o = 16; o > 0; o >>= 1) res = max(res, __shfl_xor_sync(0xffffffffu, res, o));
  if (lane == 0 && res) atomicMax(a.residual, res);
}

}  // namespace crp
