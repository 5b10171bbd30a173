"""The FDTD pass against the oracle at the edges of its tiling (64 columns per
warp, two per lane, chunks of a few rows): odd and even widths around a warp's,
row remainders, source rows on and beside chunk borders, walls and PML on every
side, bubble-free runs queued in batches of steps, and bubbles whose support box
ends beside a strip.  FP64 parity tolerance."""
import numpy as np
import pytest

import _bind as B
import crp
from test_parity_gpu import TOL_FP64, _compare

pytestmark = pytest.mark.gpu

H = 1e-4


def config(x, y, **over):
    base = dict(grid_x=x, grid_y=y, grid_lx=x * H, grid_ly=y * H, pml_grid_number=3, tr_focal_dist=0.7 * y * H,
                tr_box_size=0.0, bub_enable=0, tr_amp=0.05, dbg_T=0)
    base.update(over)
    return B.small_config(**base)


PLAIN = {
    "2x3": dict(x=2, y=3, pml_x1=0, pml_y1=0),
    "5x7_walls": dict(x=5, y=7, pml_x1=0, pml_y1=0, tr_cylindrical=0),
    "63x17": dict(x=63, y=17),
    "64x16_row5": dict(x=64, y=16, pml_y0=1, ext_source_row=5),
    "65x33_row4": dict(x=65, y=33, pml_y0=1, pml_x0=1, ext_source_row=4),
    "66x65_last_row": dict(x=66, y=65, ext_source_row=65, pml_y1=0),
    "127x9_row1": dict(x=127, y=9, ext_source_row=1, pml_x1=0),
    "128x40_plane_v": dict(x=128, y=40, tr_focused_p=0, tr_plane_v=1, pml_y0=1, ext_source_row=8),
    "129x40_focus_v": dict(x=129, y=40, tr_focused_p=0, tr_focused_v=1, pml_y1=0),
    "200x150_mixed": dict(x=200, y=150, pml_y0=1, pml_x0=1, ext_source_row=6, ext_precision=1),
}


@pytest.mark.parametrize("name", list(PLAIN))
def test_without_bubbles(name):
    over = dict(PLAIN[name])
    cfg = config(over.pop("x"), over.pop("y"), **over)
    tol = 1e-9 if cfg.ext_precision == 0 else 1e-6
    cpu = B.OracleSim(cfg)
    with crp.Sim(cfg) as gpu:
        for n in (1, 1, 37, 32, 2):  # across the batches of queued steps
            gpu.step(n)
            cpu.step(n)
            _compare(gpu, cpu, tol)
        assert gpu.stats().steps == 73 and abs(gpu.stats().time - cpu.stats().time) <= 1e-15 * cpu.stats().time


BUBBLES = {
    "ends_at_64": dict(x=130, y=40, cells=(58, 64, 10, 14)),
    "starts_at_65": dict(x=130, y=41, cells=(65, 70, 16, 17)),
    "last_column": dict(x=65, y=24, cells=(60, 65, 20, 24), pml_x1=0, pml_y1=0),
    "axis_and_first_row": dict(x=40, y=24, cells=(1, 3, 1, 4), tr_amp=0.01),
    "everywhere": dict(x=33, y=19, cells=(1, 33, 1, 19), tr_cylindrical=0, tr_amp=0.01),
    "source_row_mixed": dict(x=70, y=30, cells=(10, 20, 3, 9), pml_y0=1, ext_source_row=6, ext_precision=1, tr_amp=0.01),
}


@pytest.mark.parametrize("name", list(BUBBLES))
def test_with_bubbles(name):
    over = dict(BUBBLES[name])
    i0, i1, j0, j1 = over.pop("cells")
    cfg = config(over.pop("x"), over.pop("y"), bub_enable=1, **over)
    rng = np.random.default_rng(2)
    n = 60
    x = H * (i0 - 1 + 0.1 + (i1 - i0 + 0.8) * rng.random(n))
    y = H * (j0 - 1 + 0.1 + (j1 - j0 + 0.8) * rng.random(n))
    bub = crp.Bubbles(x, y, 3e-6 * np.exp(0.2 * rng.standard_normal(n)), np.ones(n))
    tol = 1e-9 if cfg.ext_precision == 0 else 1e-6
    cpu = B.OracleSim(cfg, bub)
    with crp.Sim(cfg, bub) as gpu:
        # At the end of the run, and the quantities that are no rounding noise
        # there (the burst is still short of some bubbles).
        for steps in (2, 6, 52):
            gpu.step(steps)
            cpu.step(steps)
        for k in ("p0", "vx", "vy", "f_g"):
            b = cpu.field(k)
            assert np.abs(gpu.field(k) - b).max() <= tol * np.abs(b).max(), k
        if cfg.ext_precision == 0:
            for k in ("R_t", "PG_p"):
                b = cpu.bubbles(k)
                assert np.abs(gpu.bubbles(k) - b).max() <= tol * np.abs(b).max(), k
            assert np.array_equal(gpu.bubbles("ibn_x"), cpu.bubbles("ibn_x"))
