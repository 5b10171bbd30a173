"""The lean form of the radius solve (reference scheme, no temperature branch): its
reciprocals and roots against 64-bit mantissas, the thermal model's three ranges
against the oracle, and the 3-D kernel for launches that wait for stiff bubbles."""
import ctypes
import os

import numpy as np
import pytest

import _bind as B
import crp
from test_cart3d import cart3d_small
from test_thermal_ranges_gpu import CASES

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# Largest relative errors, in units of 2^-53.  Each ends with one rounding (1 unit); the
# seed's error of 2^-20 leaves 2^-60.  The residual that the roots' step corrects by
# carries one rounding at half weight (rsqrt, sqrt) or three at a quarter (rroot4).
BOUNDS = {"recip": 1.01, "quotient": 1.01, "rsqrt_pos": 1.51, "sqrt_pos": 1.51, "rroot4_pos": 1.76}


@pytest.mark.parametrize("lo,hi", [(0.5, 4.0), (1e-12, 1e-3), (1e-40, 1e40)])
def test_reciprocals_and_roots(lo, hi):
    lib = ctypes.CDLL(os.path.join(ROOT, "cuda-rp_b200", "build", "libunits.so"))
    rng = np.random.default_rng(11)
    n = 1 << 21
    a, b = (np.exp(rng.uniform(np.log(lo), np.log(hi), n)) for _ in range(2))
    out = np.empty((8, n))
    p = lambda x: x.ctypes.data_as(ctypes.c_void_p)
    assert lib.units_helpers(n, p(a), p(b), p(out)) == 0
    L = np.longdouble
    x, r = b.astype(L), out[:5].astype(L)
    root = np.sqrt(x)
    rel = {"recip": r[0] * x, "quotient": r[1] * x / a.astype(L), "rsqrt_pos": r[2] * root, "sqrt_pos": r[3] / root,
           "rroot4_pos": r[4] * np.sqrt(root)}
    err = {k: float(np.abs(v - 1).max()) * 2.0**53 for k, v in rel.items()}
    print(err)
    assert all(err[k] <= BOUNDS[k] for k in err), err
    assert np.array_equal(out[1], out[6])  # quotients as divisions (ties of the last bit are rarer than 1 in 1e9)


@pytest.mark.parametrize("name", list(CASES))
def test_thermal_ranges(name):
    """As test_thermal_range_matches_oracle, whose runs have the temperature branch on
    and so the coth form: here thermal64.  The same FP64 parity tolerance."""
    r0 = CASES[name]
    n = len(r0)
    cfg = B.small_config(tr_amp=0.07, dbg_T=0)
    rng = np.random.default_rng(3)
    bub = crp.Bubbles(1e-4 + 1.5e-3 * rng.random(n), 4e-4 + 8e-4 * rng.random(n), r0, 1e-18 / r0**3)
    cpu = B.OracleSim(cfg, bub)
    cpu.step(120)
    with crp.Sim(cfg, bub) as gpu:
        gpu.step(120)
        errs = {k: float(np.max(np.abs(gpu.bubbles(k) / cpu.bubbles(k) - 1.0))) for k in ("R_t", "PG_p")}
        p = cpu.field("p0")
        errs["p0"] = float(np.max(np.abs(gpu.field("p0") - p)) / np.max(np.abs(p)))
    assert np.max(np.abs(cpu.bubbles("R_t") / r0 - 1.0)) > 1e-7
    assert max(errs.values()) < 1e-9, errs


def test_stiff_bubbles_in_3d():
    """A cloud that collapses (2,415 sub-steps in one step): the launches after it take
    the kernel for stiff bubbles.  A relative change of R0 by 3e-15 moves the oracle's
    radii by 6e-11 and its pressure by 1e-11 over these steps."""
    cfg = cart3d_small(24, bubbles=60, pml_grid_number=4, ext_array_radius=7.3 * 2e-4, ext_cloud_r=3e-4,
                       tr_amp=0.5e6 / (998 * 1482), ext_n_b=0.1)
    bub = B.oracle_seed_bubbles3(cfg)
    cpu = B.OracleSim3(cfg, bub)
    with crp.Sim(cfg, bub) as gpu:
        for _ in range(6):
            gpu.step(8)
            cpu.step(8)
            r, p = cpu.bubbles("R_t"), cpu.field("p0")
            assert np.abs(gpu.bubbles("R_t") / r - 1.0).max() < 1e-9
            assert np.abs(gpu.field("p0") - p).max() < 1e-9 * np.abs(p).max()
        assert gpu.stats().rp_substeps_max > 1000 and gpu.stats().picard_total == cpu.stats().picard_total
