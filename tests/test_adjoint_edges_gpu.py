"""The reverse sweeps of crp_adjoint at the edges of their tiling (64 columns per warp,
two per lane, chunks of rows or planes, source tables of 32 steps): the gradient
against difference formulas of J that are exact up to rounding.  J is quadratic in an
element's amplitude, and a trigonometric polynomial of degree 2 in its phase:
with o(x) = (J(phase + x) - J(phase - x)) / 2 = b1 sin x + b2 sin 2x the derivative is
b1 + 2 b2, b1 = o(pi / 2), b2 = o(pi / 4) - b1 / sqrt(2).  J itself is a sum of squares
after at most 75 linear steps (relative rounding below 1e-13), so the two sides agree
within 1e-11 of the largest J that enters."""
import numpy as np
import pytest

import crp
from test_fdtd3_edges_gpu import grid
from test_fdtd_edges_gpu import config

pytestmark = pytest.mark.gpu

TOL = 1e-11


def check(run, amp, phase):
    _, ga, gp = run(amp, phase, True)
    J = []

    def at(e, da, dp):
        a, p = amp.copy(), phase.copy()
        a[e] += da
        p[e] += dp
        J.append(run(a, p, False)[0])
        return J[-1]

    odd = lambda e, x: 0.5 * (at(e, 0.0, x) - at(e, 0.0, -x))
    n = len(amp)
    fa = np.array([(at(e, 0.5, 0.0) - at(e, -0.5, 0.0)) for e in range(n)])
    b1 = np.array([odd(e, np.pi / 2) for e in range(n)])
    fp = b1 + 2.0 * (np.array([odd(e, np.pi / 4) for e in range(n)]) - b1 / np.sqrt(2.0))
    scale = max(J)
    assert scale > 0 and np.abs(ga).max() > 1e-3 * scale
    assert np.abs(ga - fa).max() <= TOL * scale, (ga, fa)
    assert np.abs(gp - fp).max() <= TOL * scale, (gp, fp)


PLANAR = {
    "5x7_walls": dict(x=5, y=7, pml_x1=0, pml_y1=0, tr_cylindrical=0),
    "63x17": dict(x=63, y=17),
    "64x16_row5": dict(x=64, y=16, pml_y0=1, ext_source_row=5),
    "65x33_row4": dict(x=65, y=33, pml_y0=1, pml_x0=1, ext_source_row=4),
    "66x41_plane": dict(x=66, y=41, tr_focused_p=0, tr_plane_p=1, pml_y1=0),
    "129x20_row1_mixed": dict(x=129, y=20, ext_source_row=1, pml_x1=0, ext_precision=1),
}


@pytest.mark.parametrize("name", list(PLANAR))
@pytest.mark.parametrize("steps", [33, 75])
def test_planar(name, steps):
    over = dict(PLANAR[name])
    cfg = config(over.pop("x"), over.pop("y"), ext_elements=3, **over)

    def run(amp, phase, grads):
        with crp.Sim(cfg) as sim:
            sim.set_source_elements(amp, phase)
            # A focal disk over the whole grid: every cell's objective term counts.
            return sim.adjoint(steps, 2e-2, 3 if grads else 0)

    if cfg.ext_precision == 1:  # 32-bit storage of the forward fields: J is quadratic to 1e-6 only
        amp, phase = np.array([0.9, 1.2, 1.0]), np.array([0.3, -0.4, 0.0])
        ref = config(129, 20, ext_elements=3, **{**over, "ext_precision": 0})
        _, ga, gp = run(amp, phase, True)
        with crp.Sim(ref) as sim:
            sim.set_source_elements(amp, phase)
            J, ra, rp = sim.adjoint(steps, 2e-2, 3)
        assert max(np.abs(ga - ra).max(), np.abs(gp - rp).max()) <= 1e-5 * J
        return
    check(run, np.array([0.9, 1.2, 1.0]), np.array([0.3, -0.4, 0.0]))


@pytest.mark.parametrize("shape", [(13, 11, 12), (20, 17, 33), (65, 16, 18), (66, 15, 13)])
def test_3d(shape):
    cfg = grid(*shape, elems=3)

    def run(amp, phase, grads):
        with crp.Sim(cfg) as sim:
            sim.set_source_elements(amp, phase)
            return sim.adjoint(40, 2e-2, 3 if grads else 0)

    check(run, np.array([0.9, 1.2, 1.0]), np.array([0.3, -0.4, 2.0]))
