"""The 3-D FDTD pass against the 3-D oracle at the edges of its tiling (64 columns
per warp, two per lane, 8 rows per block, chunks of planes): odd and even extents
per axis, bubble-free runs queued in batches of steps, clouds smaller than a tile and
over most of the grid.  FP64 parity tolerance of the 3-D tests."""
import numpy as np
import pytest

import _bind as B
import crp
from test_cart3d import cart3d_small

pytestmark = pytest.mark.gpu

TOL = 1e-9


def grid(x, y, z, **over):
    return cart3d_small(grid_x=x, grid_y=y, ext_grid_z=z, grid_lx=x * 2e-4, grid_ly=y * 2e-4, ext_grid_lz=z * 2e-4,
                        pml_grid_number=3, ext_array_radius=(min(x, y, z) / 2 - 4.3) * 2e-4, **over)


def same(gpu, cpu, names):
    for k in names:
        b = cpu.field(k)
        assert np.abs(gpu.field(k) - b).max() <= TOL * max(np.abs(b).max(), 1e-9), k


@pytest.mark.parametrize("shape", [(12, 12, 12), (13, 9, 17), (63, 16, 11), (64, 17, 33), (65, 15, 16), (66, 24, 40),
                                   (129, 10, 13)])
def test_without_bubbles(shape):
    cfg = grid(*shape)
    cpu = B.OracleSim3(cfg)
    with crp.Sim(cfg) as gpu:
        for n in (1, 2, 35, 2):  # across the batches of queued steps
            gpu.step(n)
            cpu.step(n)
        same(gpu, cpu, ("p0", "vx", "vy", "vz", "pz"))
        assert gpu.stats().steps == 40 and abs(gpu.stats().residual_last - cpu.stats().residual_last) <= 1e-9 * max(
            cpu.stats().residual_last, 1e-30)


@pytest.mark.parametrize("shape,cloud,shape_kind", [((40, 22, 26), 3e-4, 1), ((67, 20, 20), 1e-3, 1),
                                                    ((33, 33, 35), 2.4e-3, 2)])
def test_with_a_cloud(shape, cloud, shape_kind):
    cfg = grid(*shape, bubbles=200, ext_cloud_r=cloud, ext_cloud_shape=shape_kind, tr_amp=0.05e6 / (998 * 1482))
    bub = crp.seed_bubbles3(cfg)
    half = 1e-4
    for a, n in ((bub.x, shape[0]), (bub.y, shape[1]), (bub.z, shape[2])):
        np.clip(a, half, n * 2e-4 - half, out=a)
    cpu = B.OracleSim3(cfg, bub)
    with crp.Sim(cfg, bub) as gpu:
        for n in (3, 27):
            gpu.step(n)
            cpu.step(n)
        same(gpu, cpu, ("p0", "vx", "vy", "vz", "f_g"))
        assert np.array_equal(gpu.bubbles("ibn_x"), cpu.bubbles("ibn_x"))
        r = cpu.bubbles("R_t")
        assert np.abs(gpu.bubbles("R_t") - r).max() <= TOL * r.max()


def test_steps_without_coupling():
    """A Picard tolerance so loose that the loop runs on some steps only: the void
    fraction is extrapolated over gaps of up to 20 steps in between."""
    cfg = grid(40, 22, 26, bubbles=200, ext_cloud_r=6e-4, ext_cloud_shape=1, tr_amp=0.02e6 / (998 * 1482),
               ext_picard_tol=0.2, tr_on_wave=1, ext_ramp_cycles=0)
    bub = crp.seed_bubbles3(cfg)
    cpu = B.OracleSim3(cfg, bub)
    with crp.Sim(cfg, bub) as gpu:
        for n in (20, 30, 15, 35):
            gpu.step(n)
            cpu.step(n)
            same(gpu, cpu, ("p0", "vx", "f_g", "f_gn", "f_gm"))
            assert gpu.stats().picard_total == cpu.stats().picard_total
        assert 20 < cpu.stats().picard_total < 130
