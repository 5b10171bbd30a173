"""The thermal model's three ranges on the GPU against the oracle: bubbles whose
alpha_N argument (w = 2 s^2, about 1.6 per micrometre of rest radius here) lies
below 32, between 32 and 760, above 760, and on both sides of the two limits
while they oscillate.

Tolerance: the FP64 parity tolerance 1e-9.  Both sides evaluate the model within
a few 1e-15 for these radii (the oracle's coth form loses at most 1e-12 of
Im Lp at 1 um), and 120 steps of a 0.1 MPa drive amplify that by far less than 1e3."""
import numpy as np
import pytest

import _bind as B
import crp

pytestmark = pytest.mark.gpu

TOL = 1e-9


def radii(lo, hi, n=40):
    return np.geomspace(lo, hi, n)


CASES = {
    "small": radii(1e-6, 1.5e-5),
    "limit_32": radii(1.8e-5, 2.4e-5),
    "middle": radii(2.5e-5, 4e-4),
    "limit_760": radii(4.2e-4, 5.6e-4),
    "large": radii(6e-4, 2e-3),
    "one": np.array([4.75e-4]),
}


@pytest.mark.parametrize("scheme", [0, 1])
@pytest.mark.parametrize("name", list(CASES))
def test_thermal_range_matches_oracle(name, scheme):
    r0 = CASES[name]
    n = len(r0)
    cfg = B.small_config(tr_amp=0.07, ext_rp_scheme=scheme)
    rng = np.random.default_rng(3)
    bub = crp.Bubbles(1e-4 + 1.5e-3 * rng.random(n), 4e-4 + 8e-4 * rng.random(n), r0, 1e-18 / r0**3)
    cpu = B.OracleSim(cfg, bub)
    cpu.step(120)
    with crp.Sim(cfg, bub) as gpu:
        gpu.step(120)
        errs = {k: float(np.max(np.abs(gpu.bubbles(k) / cpu.bubbles(k) - 1.0))) for k in ("R_t", "PG_p")}
        p = cpu.field("p0")
        errs["p0"] = float(np.max(np.abs(gpu.field("p0") - p)) / np.max(np.abs(p)))
    print(name, scheme, errs)
    assert np.max(np.abs(cpu.bubbles("R_t") / r0 - 1.0)) > 1e-7  # the burst has reached the bubbles
    assert max(errs.values()) < TOL, errs


@pytest.mark.parametrize("precision", [0, 1])
def test_stiff_launches_round_as_quiet_ones(precision):
    """A cloud that starts to collapse (1,468 sub-steps): host-driven steps take the
    radius kernel for stiff launches once a bubble has needed 150 sub-steps, graph
    steps the quiet one throughout; bit for bit the same."""
    out = []
    for graphs in (0, 1):
        cfg = B.small_config(tr_amp=0.2, dbg_T=0, ext_bubble_count=120, ext_bubble_seed=3, ext_r0_sigma_ln=0.3,
                             ext_cloud_r=8e-4, ext_cloud_h=2e-3, ext_n_b=1.0, bub_R0=3e-6, ext_precision=precision,
                             ext_graphs=graphs)
        bub = crp.seed_bubbles(cfg)
        with crp.Sim(cfg, bub) as gpu:
            gpu.step(290)
            gpu.step(25)
            assert gpu.stats().rp_substeps_max > 1000
            out.append([gpu.field(k) for k in ("p0", "vx", "f_g")] + [gpu.bubbles(k) for k in ("R_t", "PG_p", "Q_B")])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
