"""The void-fraction forms of the FDTD passes where there is none: cells whose density
is rho_inf take the velocity update with dt / rho_inf as the plain forms do, to the bit.

dt and rho_inf are a pair whose quotient lies 2^-54 of a unit from the middle of two
doubles, where a quotient by way of a rounded reciprocal is one unit off.  A
population with so small a weight that 1 - f_g is 1 leaves the pressure as without
bubbles: f_g's own terms are below 1e-200.  Compared are values above 1e-6 of the
largest; at the foot of the wave, beside exact zeros, those terms decide ties."""
import numpy as np
import pytest

import _bind as B
import crp
from test_cart3d import cart3d_small

pytestmark = pytest.mark.gpu

RHO = float.fromhex("0x1.ff01e0e42ff97p+9")
CFL = float.fromhex("0x1.78aa5f48378f7p-2")
H, C = 2.0**-13, 1024.0
QUOTIENT = float.fromhex("0x1.7965afa8847edp-35")


def compare(cfg, pos, steps, fields):
    n = len(pos)
    assert cfg.sim_cfl * H / C / RHO == QUOTIENT
    out = []
    for bubbles in (False, True):
        cfg.bub_enable = 1 if bubbles else 0
        z = np.ascontiguousarray(pos[:, 2]) if pos.shape[1] == 3 else None
        b = crp.Bubbles(np.ascontiguousarray(pos[:, 0]), np.ascontiguousarray(pos[:, 1]), np.full(n, 3e-6),
                        np.full(n, 1e-250), z)
        with crp.Sim(cfg, b if bubbles else None) as sim:
            sim.step(steps)
            out.append([sim.field(f) for f in fields])
            if bubbles:
                fg = sim.field("f_g")
                assert 0.0 < np.abs(fg).max() < 1e-200
    for f, a, b in zip(fields, *out):
        seen = np.abs(a) > 1e-6 * np.abs(a).max()
        assert seen.sum() > 500
        assert np.array_equal(a[seen], b[seen]), (f, np.abs(a - b).max() / np.abs(a).max())


def test_axisymmetric():
    cfg = B.small_config(dbg_T=0, tr_amp=0.05, sim_cfl=CFL, grid_x=70, grid_y=96, grid_lx=70 * H, grid_ly=96 * H,
                         ext_c_inf=C, ext_rho_inf=RHO, tr_box_size=0.0)
    pos = np.array([(x, y) for x in (3.3, 20.2, 41.7) for y in (5.4, 17.1, 31.8)]) * H
    compare(cfg, pos, 60, ("p0", "vx", "vy"))


def test_three_dimensional():
    cfg = cart3d_small(40, h=H, sim_cfl=CFL, ext_c_inf=C, ext_rho_inf=RHO, tr_amp=0.05e6 / (RHO * C))
    pos = np.array([(x, y, z) for x in (15.3, 22.2) for y in (16.4, 24.1) for z in (12.3, 20.4)]) * H
    compare(cfg, pos, 40, ("p0", "vx", "vy", "vz"))
