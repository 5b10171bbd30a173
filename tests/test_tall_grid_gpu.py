"""Read-back of a grid with more rows than 8 times the largest launch extent."""
import numpy as np
import pytest

import _bind as B
import crp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_fields_of_a_tall_grid(precision):
    Y = 600000
    cfg = B.small_config(grid_x=8, grid_y=Y, grid_lx=8e-4, grid_ly=Y * 1e-4, pml_grid_number=3, bub_enable=0, dbg_T=0,
                         tr_focused_p=0, tr_plane_p=1, ext_precision=precision)
    cpu = B.OracleSim(cfg)
    with crp.Sim(cfg) as gpu:
        t = gpu.tuning
        t.fdtd_rows = 16
        gpu.tuning = t
        gpu.step(4)
        cpu.step(4)
        for f in ("vx", "vy", "f_g", "rho_m"):
            a, b = gpu.field(f), cpu.field(f)
            assert a.shape == b.shape
            assert np.abs(a - b).max() <= (1e-9 if precision == 0 else 1e-7) * max(np.abs(b).max(), 1e-12), f
        assert np.abs(gpu.field("vy")).max() > 1e-6 and np.all(gpu.field("rho_m")[-1] == cfg.ext_rho_inf)
