"""Radius sub-steps whose acceleration or velocity is infinite: the step limits of
solveRayleighPlesset leave no step, and the solve ends as failed (the caller's
sub-step error) in every form, as with the reference's steps of 0 up to the cap; one
of NaN has no limit in the reference and runs to its end."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CAP = 50


@pytest.mark.parametrize("form", [0, 1, 2, 3])
def test_no_step_left_is_a_failed_solve(form):
    lib = ctypes.CDLL(os.path.join(ROOT, "cuda-rp_b200", "build", "libunits.so"))
    inf, nan = np.inf, np.nan
    #       pressure, velocity, fails
    rows = [(0.0, 0.0, 0), (1e4, -1.0, 0), (nan, 0.0, 0), (0.0, nan, 0),
            (inf, 0.0, 1), (-inf, 0.0, 1), (0.0, inf, 1), (0.0, -inf, 1), (inf, -inf, 1), (-inf, inf, 1),
            (1e300, 0.0, 1), (0.0, 1e200, 1)]
    a = np.array([r[:2] for r in rows])
    pl, v = np.ascontiguousarray(a[:, 0]), np.ascontiguousarray(a[:, 1])
    out = np.full((len(rows), 2), -1, dtype=np.int32)
    p = lambda x: x.ctypes.data_as(ctypes.c_void_p)
    assert lib.units_solve(form, CAP, len(rows), p(pl), p(v), p(out)) == 0
    assert out[:, 0].tolist() == [r[2] for r in rows]
    assert out[0, 1] == 10 and out[:, 1].max() <= CAP
