"""Tiles of the 3-D grid that bubbles have left while their void fraction lives on.

Three bubbles start 0.05 cells inside a face of a 32 x 8 x 8 tile, in a light, slow
medium whose source pushes them across it within the first ten steps.  The source is
on for one step in three or four (its period is one step, so its sine is sampled at
one phase), and the Picard tolerance lies between its jumps and the rest of the field:
the loop runs on two steps of every three or four.  The steps without it extrapolate
the void fraction, so what the bubbles left behind in the tile stays (steps of every
three) or grows threefold a time (of every four) although no coupling puts anything
there.  FP64 parity tolerance of the 3-D tests; the largest value left behind at the
end is checked on the oracle's side."""
import numpy as np
import pytest

import _bind as B
import crp
from test_cart3d import cart3d_small

pytestmark = pytest.mark.gpu

TOL = 1e-9
H = 2e-4
FG = ("f_g", "f_gn", "f_gm")


def case(off, tol):
    c, rho = 400.0, 1.2
    cfg = cart3d_small(grid_x=40, grid_y=24, ext_grid_z=24, grid_lx=40 * H, grid_ly=24 * H, ext_grid_lz=24 * H,
                       pml_grid_number=3, ext_array_radius=7.7 * H, ext_array_elements=1, ext_rho_inf=rho, ext_c_inf=c,
                       tr_freq=c / (0.4 * H) / 1.0001, tr_on_wave=1, tr_off_wave=off, ext_ramp_cycles=0.0,
                       tr_amp=2e4 / (rho * c), ext_picard_tol=tol, bub_enable=1)
    pos = np.array([(17.3, 6.55, 5.2), (20.2, 6.55, 4.8), (22.7, 6.55, 5.4)]) * H
    bub = crp.Bubbles(pos[:, 0].copy(), pos[:, 1].copy(), np.full(3, 2e-5), np.full(3, 1e-3), pos[:, 2].copy())
    return cfg, bub


def tile(a):
    """The tile of cells 0..31 x 8..15 x 0..7 of a field [z][y][x]."""
    return a[0:8, 8:16, 0:32]


@pytest.mark.parametrize("off,tol,steps,left", [
    (2, 0.15, 60, 5e-9),    # the loop runs on two steps of three
    (3, 0.15, 42, 2.9e-4),  # on two of four
    (2, 1e-3, 60, 0.0),     # on every step: nothing is left behind
])
def test_void_fraction_outlives_its_bubbles(off, tol, steps, left):
    cfg, bub = case(off, tol)
    cpu = B.OracleSim3(cfg, bub)
    one = np.ones(1), np.full(1, 0.5 * np.pi)
    cpu.set_source_elements(*one)
    with crp.Sim(cfg, bub) as gpu:
        gpu.set_source_elements(*one)
        last = 0
        for k in range(0, steps, 6):
            gpu.step(6)
            for s in range(k, k + 6):
                cpu.step(1)
                if (cpu.bubbles("ibn_y") >= 7).any():
                    last = s + 1
            for f in FG + ("p0", "vx", "vy", "vz"):
                b = cpu.field(f)
                assert np.abs(gpu.field(f) - b).max() <= TOL * np.abs(b).max(), (k + 6, f)
        assert gpu.stats().picard_total == cpu.stats().picard_total
    assert 6 <= last <= 12  # the last step that had a bubble in the tile
    most = max(np.abs(tile(cpu.field(f))).max() for f in FG)
    assert most >= left if left else most == 0.0
