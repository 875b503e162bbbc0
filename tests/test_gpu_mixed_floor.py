"""The mixed form on the benchmark's batch, whose Coulomb-dominated points end at the rounding floor: a step that stays
inexact in double-double is finished in FP64, not taken for the floor."""
import numpy as np
import pytest

from helpers import gpu_solver
from test_gpu_solve import gpu_solution

pytestmark = pytest.mark.gpu


def test_mixed_form_is_within_its_bound_on_the_whole_batch(synthetic_xs):
    """4096 points, 128 B-splines, l_max 2, e-e on: every point's EDF is within 1e-8 of the plain FP64 form's, the
    bound that the benchmark states for the mixed form."""
    from boltzmann_gb300.workloads import batch_parameters
    P = 4096
    prm = batch_parameters(P, 20261203)
    out = {}
    for prec in ("mixed", "fp64"):
        s, args = gpu_solver(synthetic_xs, 128, 2, True, P, prec)
        f, q = gpu_solution(s, args, prm, True, P)
        assert np.all(np.asarray(q["status"]) <= 1)
        out[prec] = np.asarray(f)
    err = np.linalg.norm(out["mixed"] - out["fp64"], axis=0) / np.linalg.norm(out["fp64"], axis=0)
    assert err.shape == (P,) and np.max(err) <= 1e-8, (np.argsort(err)[-3:], np.sort(err)[-3:])
