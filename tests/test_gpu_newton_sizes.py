"""Newton-step kernels at the sizes where their layout changes: spline counts around a warp's
multiples, one to many points (a point's splines are split over a cluster's CTAs when few points
run; several points share a CTA when many do), every mode count.

The way the work is split is not allowed to enter a point's arithmetic, so a point's solution is
the same to the last bit however many points are solved with it, in both forms.
"""
import numpy as np
import pytest

from helpers import gpu_solver
from test_gpu_solve import gpu_solution

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_sp,l_max", [(16, 1), (31, 2), (49, 3), (65, 1), (100, 2)])
def test_point_does_not_depend_on_the_batch(synthetic_xs, n_sp, l_max, precision):
    from boltzmann_gb300.workloads import batch_parameters
    sizes = (1, 2, 11, 330)
    prm = batch_parameters(sizes[-1], 77)
    ref = None
    for P in reversed(sizes):
        s, args = gpu_solver(synthetic_xs, n_sp, l_max, True, P, precision)
        sub = {k: (v[..., :P] if np.ndim(v) > 1 else v[:P]) for k, v in prm.items() if np.ndim(v)}
        ff, q = gpu_solution(s, args, sub, True, P)
        ff, st = np.asarray(ff), np.asarray(q["status"])
        assert np.all(np.isfinite(ff[:, st <= 1])) and np.mean(st <= 1) > 0.5
        if ref is None:
            ref = ff, st
        # coarse grids leave some points unconverged: they too end alike
        np.testing.assert_array_equal(st, ref[1][:P], err_msg="%d points" % P)
        np.testing.assert_array_equal(ff, ref[0][:, :P], err_msg="%d points" % P)


@pytest.mark.parametrize("n_sp,l_max", [(20, 1), (47, 2)])
def test_coefficients_of_several_points_per_cta(synthetic_xs, n_sp, l_max):
    """From 608 points on, the e-e coefficients of two or four points are formed by one CTA (an odd
    count leaves its last group partly empty): the same bits as for two points."""
    from boltzmann_gb300.workloads import batch_parameters
    prm = batch_parameters(2501, 78)
    out = []
    for P in (2, 701, 2501):
        s, args = gpu_solver(synthetic_xs, n_sp, l_max, True, P, "mixed")
        sub = {k: (v[..., :P] if np.ndim(v) > 1 else v[:P]) for k, v in prm.items() if np.ndim(v)}
        ff, q = gpu_solution(s, args, sub, True, P)
        out.append((np.asarray(ff), np.asarray(q["status"])))
    for ff, st in out[:-1]:
        np.testing.assert_array_equal(st, out[-1][1][:len(st)])
        np.testing.assert_array_equal(ff, out[-1][0][:, :ff.shape[1]])
    assert np.mean(out[-1][1] <= 1) > 0.5
