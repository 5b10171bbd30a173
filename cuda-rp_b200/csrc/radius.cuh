// The per-bubble radius solve of the reference scheme shared by the 2-D and
// 3-D paths: the sub-step state of BubbleRadiusKernel and one pass of its
// sub-step loop (inc/bubble_CUDA_kernel.cuh:471-554).
#pragma once
#include "crp_device.cuh"

namespace crp {

// The sub-step comes in two forms of the same scheme:
//   kLean  the thermal model of thermal64, no divisions but reciprocals;
//   kHeat  the reference's operation order with the coth form, kept for runs with the
//          temperature branch.  A resting bubble's heat flux is what the rounding of
//          its gas pressure leaves (the gas pressure has a fixed point at which
//          PG0 R0^3 and PG R^3 differ by rounding), so another order of operations
//          moves the temperature field by up to 1e-8 before the burst arrives; with
//          the order kept it is reproduced to the bit.
enum RadiusForm { kLean = 0, kHeat = 1 };

// Per-bubble constants of the lean form: the mixed path (T = float) also keeps
// the FP32 thermal model's.
template <typename T>
struct RadiusConst {
  BubbleConst c;
};
template <>
struct RadiusConst<float> {
  BubbleConst c;
  double R0;
  ThermalConst<float> f;
};
template <typename T, int FORM>
struct RadiusConstOf {
  using type = RadiusConst<T>;
};
template <typename T>
struct RadiusConstOf<T, kHeat> {
  using type = BubbleR0;
};

// Per-bubble state of BubbleRadiusKernel (inc/bubble_CUDA_kernel.cuh:471-554)
// while its sub-steps run.  T: type of the thermal model near equilibrium.
template <typename T, int FORM>
struct RpState {
  double Rt, Rp, Rn, d1Rp, PGp, dtL, remain, time, PC0, PC1, PC2, heat, vis, re_n;
  typename RadiusConstOf<T, FORM>::type r;
  int count;
};
template <typename T, int FORM>
__device__ __forceinline__ void radius_const(const BubbleParams& b, double R0, RpState<T, FORM>& s) {
  if constexpr (FORM == kHeat) {
    s.r = bubble_r0(b, R0);
  } else {
    s.r.c = bubble_const(b, R0);
    if constexpr (sizeof(T) == sizeof(float)) {
      s.r.R0 = R0;
      s.r.f = thermal_const32(b, bubble_r0(b, R0));
    }
  }
}

// Relative radius excursion |R/R0 - 1| above which the mixed path evaluates
// the thermal model in FP64: FP32 is accurate for the small oscillations of a
// quiet bubble, and its rounding is amplified once the bubble is driven.
constexpr double kThermalFp64Excursion = 1.0e-3;

// ---- kHeat ------------------------------------------------------------------
// One pass of the sub-step loop of BubbleRadiusKernel (:506-539).  T is the
// real type of the thermal model (omega_N, alpha_N, Lp_N); everything else is FP64.
template <typename T, typename STATE>
__device__ __forceinline__ void thermal_model(const BubbleParams& bp, const STATE& s, double PGn, double& omega,
                                              C64& lp) {
  Cx<T> alpha_t;
  ThermalConst<T> c;
  if constexpr (sizeof(T) == sizeof(double))
    c = thermal_const64(bp, s.r);
  else
    c = thermal_const32(bp, s.r);
  omega = (double)omega_n<T>(alpha_t, (T)PGn, (T)s.Rn, c);
  const Cx<T> lp_t = lp_n<T>(alpha_t, (T)s.Rn, c.cut2);
  lp = C64{(double)lp_t.re, (double)lp_t.im};
}

template <typename T>
__device__ __forceinline__ void rp_substep_heat(const BubbleParams& bp, RpState<T, kHeat>& s) {
  const double PGn = s.PGp;
  const double PL = s.PC2 * s.time * s.time + s.PC1 * s.time + s.PC0;
  rp_substep(s.Rt, s.Rp, s.Rn, s.d1Rp, PGn, PL, s.dtL, s.remain, bp);
  s.time = s.time + s.dtL;
  double omega;
  C64 lp;
  if (sizeof(T) == sizeof(double) || fabs(s.Rn - s.r.R0) > kThermalFp64Excursion * s.r.R0)
    thermal_model<double>(bp, s, PGn, omega, lp);
  else
    thermal_model<T>(bp, s, PGn, omega, lp);
  const double den = lp.re * lp.re + lp.im * lp.im;
  const double inv_wdt = 1.0 / (omega * s.dtL);
  s.PGp = gas_pressure(PGn, s.Rp, s.Rn, inv_wdt, s.dtL, den, lp, bp, s.r);
  const double inv_den = 1.0 / den;  // for the heat flux only, off the chain to the next sub-step
  const double Rp = s.Rp, Rn = s.Rn, PGp = s.PGp;
  const double s0 = 0.5 * (Rp + Rn);
  const double s1 = inv_den * s.r.T0_PG0R03;
  const double dTdr = lp.re * s1 * (s.r.PG0 * s.r.R03 - 0.5 * (PGp + PGn) * s0 * s0 * s0) +
                      lp.im * s1 * (PGp * Rp * Rp * Rp - PGn * Rn * Rn * Rn) * inv_wdt;
  s.heat -= 4.0 * bp.pi * Rp * Rp * bp.K0 * dTdr * s.dtL;
  // 4 pi Rp^2 (4 mu d1Rp / Rp) d1Rp dt, with Rp^2 / Rp cancelled.
  s.vis += 4.0 * bp.pi * Rp * 4.0 * bp.mu * s.d1Rp * s.d1Rp * s.dtL;
  s.count++;
}

// ---- kLean ------------------------------------------------------------------
// The FP32 thermal model of the mixed path near equilibrium.
__device__ __forceinline__ Thermal thermal32(const ThermalConst<float>& c, double PG, double Rb) {
  Cx<float> alpha;
  const float omega = omega_n<float>(alpha, (float)PG, (float)Rb, c);
  const Cx<float> lp = lp_n<float>(alpha, (float)Rb, c.cut2);
  const double lr = lp.re, li = lp.im;
  return {(double)omega, lr, li, lr * lr + li * li};
}

// a x + b y with every operation rounded.
__device__ __forceinline__ double weighted(double a, double x, double b, double y) {
  return __dadd_rn(__dmul_rn(a, x), __dmul_rn(b, y));
}

// One pass of the sub-step loop of BubbleRadiusKernel (:506-539):
// solveRayleighPlesset (:227-260), one variable sub-step of the three-level
// scheme; the thermal model at the old radius; solvePG (:326-340), with c1, c2, c3
// and the numerator multiplied by R omega |Lp|^2, so that Lp and the time step enter
// without divisions of their own and the gas pressure costs one reciprocal; and
// the heat flux (:521-527).
//
// Bound by the FP64 pipe in the quiet phase (63 % busy; the launch over 262,144
// bubbles of 10 sub-steps takes 77 us, 178 us with the coth form) and by the latency of
// this chain once a few bubbles are stiff.  Cycles per sub-step of one warp alone, for
// w < 32, between and above 760: quiet instance 1,330, 1,710 and 1,520; TIGHT 1,250, 1,420
// and 1,360; the coth form 4,620.
//
// TIGHT: for launches that end with the chains of a few stiff bubbles.  The radius
// update runs inside the thermal model's rounds, without branches of its own, and the
// rounds are unrolled; the results are the same to the bit (every multiply-add is
// written out, so that both are rounded alike).
template <bool TIGHT, typename T>
__device__ __forceinline__ void rp_substep_lean(const BubbleParams& b, RpState<T, kLean>& s) {
  const double eps = 2.22044604925031308e-016;
  const double PGn = s.PGp;
  const double PL = fma(s.PC2 * s.time, s.time, fma(s.PC1, s.time, s.PC0));
  const double Rm = s.Rn, Rn = s.Rp, d1n = s.d1Rp;
  const double inv_Rn = recip(Rn);
  const double dtm = s.dtL;
  double dtp, Rp, d1, last;
  auto radius = [&]() {
    // The velocity and acceleration limits, 0.01 Rn / |d1R| and 0.1 Rn / sqrt(|acc|)
    // (:238-241): each quotient is formed only where it is the smaller step, decided
    // on the products (the squares for the second), so a quiet sub-step divides by
    // neither.  An infinite velocity or acceleration makes the quotient NaN (recip,
    // rsqrt_pos) and with it the step and the remaining time: the solve stops as failed
    // (rp_failed) where the reference takes steps of 0 up to the cap.
    const double net = fma(-(4.0 * b.mu * inv_Rn), d1n, fma(-2.0 * b.sig, inv_Rn, PGn - PL));
    const double acc = fma(net, b.inv_rho, -__dmul_rn(1.5 * d1n, d1n));
    dtp = smaller(1.01 * dtm, b.dt0);
    const double ad = fabs(d1n), aa = fabs(acc), lim = 0.1 * Rn;
    if (TIGHT) {
      const double tv = 0.01 * Rn * recip(ad), ta = lim * rsqrt_pos(aa);
      dtp = ad > eps && 0.01 * Rn < dtp * ad ? limited(tv, dtp) : dtp;
      dtp = aa > eps && lim * lim < dtp * dtp * aa ? limited(ta, dtp) : dtp;
    } else {
      if (ad > eps && 0.01 * Rn < dtp * ad) dtp = limited(0.01 * Rn * recip(ad), dtp);
      if (aa > eps && lim * lim < dtp * dtp * aa) dtp = limited(lim * rsqrt_pos(aa), dtp);
    }
    // q and 1 + q round as the reference's do: the rounding of 1 + q is the same at
    // every sub-step of a constant growth and acts on R as a small force, 1e-9 of a
    // driven bubble's radius after 1000 mixture steps.  So do the products of the
    // velocity's difference, in which the radii cancel.
    const double sum = dtm + dtp;
    const double q = quotient(dtp, dtm);
    const double inv3 = recip(dtm * dtp * sum);
    const double tm2 = __dmul_rn(dtm, dtm), tp2 = __dmul_rn(dtp, dtp);  // their difference 0 at equal steps
    Rp = fma(dtp * inv_Rn, 0.5 * sum * acc, fma(1.0 + q, Rn, -__dmul_rn(q, Rm)));
    d1 = fma(__dadd_rn(weighted(tm2, Rp, tp2 - tm2, Rn), -__dmul_rn(tp2, Rm)), inv3, __dmul_rn(dtp * inv_Rn, acc));
    s.Rt = Rp;
    last = dtp;
    if (TIGHT) {
      const double rem = s.remain, qr = quotient(rem, dtm);
      const double Rl = fma(rem * inv_Rn, 0.5 * (dtm + rem) * acc, fma(1.0 + qr, Rn, -__dmul_rn(qr, Rm)));
      if (dtp >= rem) last = rem, s.Rt = Rl;
    } else if (dtp >= s.remain) {
      last = s.remain;
      const double qr = quotient(last, dtm);
      s.Rt = fma(last * inv_Rn, 0.5 * (dtm + last) * acc, fma(1.0 + qr, Rn, -__dmul_rn(qr, Rm)));
    }
  };
  Thermal th;
  if constexpr (sizeof(T) == sizeof(float)) {
    if (fabs(Rn - s.r.R0) > kThermalFp64Excursion * s.r.R0)
      th = thermal64<false>(b, s.r.c.pgr, Rn, inv_Rn, [] {});
    else
      th = thermal32(s.r.f, PGn, Rn);
    radius();
  } else if constexpr (TIGHT) {
    th = thermal64<true>(b, s.r.c.pgr, Rn, inv_Rn, radius);
  } else {
    th = thermal64<false>(b, s.r.c.pgr, Rn, inv_Rn, [] {});
    radius();
  }
  s.remain -= last;
  s.Rn = Rn;
  s.Rp = Rp;
  s.d1Rp = d1;
  s.dtL = dtp;
  s.time = s.time + dtp;
  s.count++;
  // Gas pressure.
  const double k0 = b.k0g * s.r.c.tpgr;  // 3 (gam - 1) K0 T0 / (PG0 R0^3)
  const double R = 0.5 * (Rp + Rn), R3 = R * R * R;
  const double Rp3 = Rp * Rp * Rp, Rn3 = Rn * Rn * Rn;
  const double wd = th.omega * th.den;
  const double wh = th.omega * dtp * th.lr;
  const double gd = Rp - Rn, gc = 0.5 * b.th_g3;
  const double a3 = 0.5 * k0 * wh * R3;
  const double wn = k0 * th.li;
  const double c1 = fma(-wn, Rp3, fma(wd, fma(gc, gd, R), a3));
  const double c2 = fma(-wn, Rn3, fma(wd, fma(-gc, gd, R), -a3));
  const double PG = fma(c2, PGn, __dmul_rn(k0 * wh, s.r.c.pgr)) * recip(c1);
  s.PGp = PG;
  // Heat flux (off the chain to the next sub-step) and viscous work:
  // 4 pi Rp^2 (4 mu d1R / Rp) d1R dt, with Rp^2 / Rp cancelled.
  const double hx = fma(wh, fma(-0.5 * (PG + PGn), R3, s.r.c.pgr),
                        __dmul_rn(th.li, fma(PG, Rp3, -__dmul_rn(PGn, Rn3))));
  s.heat = fma(-(4.0 * b.pi * b.K0 * Rp * Rp), s.r.c.tpgr * hx * recip(wd), s.heat);
  s.vis = fma(16.0 * b.pi * b.mu * Rp * d1, d1 * dtp, s.vis);
}

// Whether a solve goes on, and whether one that does not was left unfinished: at the
// cap, or with no step left (a remaining time of NaN).
template <typename STATE>
__device__ __forceinline__ bool rp_more(const BubbleParams& b, const STATE& s) {
  return s.remain > 0.0 && s.count < b.step_cap;
}
template <typename STATE>
__device__ __forceinline__ bool rp_failed(const STATE& s) {
  return !(s.remain <= 0.0);
}

template <bool TIGHT, typename T, int FORM>
__device__ __forceinline__ void rp_substep_full(const BubbleParams& b, RpState<T, FORM>& s) {
  if constexpr (FORM == kHeat)
    rp_substep_heat<T>(b, s);
  else
    rp_substep_lean<TIGHT, T>(b, s);
}

}  // namespace crp
