"""The finite-volume operator and op-split step off the fixture's sizes: odd line lengths (remainders
of the kernels' tiles), stencils of two to five points (the last takes the general sweeps), fields of both signs and
zero, both x-rows that fit in shared memory with few and with many rows, and a NaN. Against the dense
oracle (oracle/bte1d_fvm_oracle.py). Tolerance 1e-12 of the largest value, as for the fixtures."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(synthetic_xs, Np, Nr, Nvt, orders):
    from helpers import FVM_IMPLICIT_PARAMS
    from boltzmann_gb300.bte_1d3v_fvm import bte_1d3v_fvm
    pvr, pvt, px = orders
    s = bte_1d3v_fvm(dict(FVM_IMPLICIT_PARAMS, collisions=synthetic_xs, Np=Np, Nr=Nr, Nvt=Nvt, pvr=pvr, pvt=pvt, px=px))
    dt = 1e-3
    s.init(dt)
    rng = np.random.default_rng(Np + Nr)
    E = 3e3 * rng.standard_normal(Np)
    E[Np // 3] = 0.0
    v = s.initial_condition().cpu().numpy() * (1.0 + 0.3 * rng.standard_normal((s.dof_v, Np)))
    return s, E, v, dt


@pytest.mark.parametrize("Np,Nr,Nvt,orders", [(13, 7, 4, (1, 1, 1)), (33, 9, 6, (2, 2, 2)), (64, 12, 8, (3, 3, 3)),
                                              (101, 10, 4, (2, 1, 3)), (31, 9, 10, (4, 4, 4)), (900, 6, 4, (2, 2, 2))])
def test_operator_and_split_step_match_the_oracle(synthetic_xs, Np, Nr, Nvt, orders):
    from oracle import bte1d_fvm_oracle as O
    s, E, v, dt = _setup(synthetic_xs, Np, Nr, Nvt, orders)
    p, gi = s.params, s.grid_info
    vr, vt, x = gi["vr"], gi["vt"], gi["x"]
    cA, ax = s._coef(dt).cA, s._coef(dt).ax
    g = dict(Nr=len(vr), Nvt=len(vt), Nx=Np, pvr=orders[0], pvt=orders[1], px=orders[2], tau=p.tau, qe=p.qe, me=p.me,
             vth=s.bs_vth, L=p.L, vr=vr, vt=vt, n0=p.n0, np0=p.np0, op_col_en=s.op_col.dense(),
             PmatC=s.op_col.inverse_dense(dt * p.tau * p.n0 * p.np0), **s.bands)
    want = O.op_split_step(g, E, v, dt)
    got = s.step_op_split(E, v, None, 0.0, dt).cpu().numpy()
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))
    A_Ep, A_En = O.adv_v_fvm(vr, vt, orders[0], orders[1], s.vmax)
    xs = O.x_shift_bands(vr, vt, x, orders[2], ax, dt)
    want = O.implicit_matvec(g, cA * A_Ep, cA * A_En, xs, E, v, dt)
    got = s.rhs_mvec(E, v, dt).cpu().numpy()
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


def test_nan_reaches_its_column_and_no_call_after(synthetic_xs):
    """A NaN at one value makes every value off the inflow of its x column NaN (the collision terms
    couple all cells and ordinates of a column, also through zero entries of their matrices), and the
    call after it is clean."""
    s, E, v, dt = _setup(synthetic_xs, 37, 9, 6, (2, 2, 2))
    clean = s.rhs_mvec(E, v, dt).cpu().numpy(), s.step_op_split(E, v, None, 0.0, dt).cpu().numpy()
    w = v.copy()
    w[-1, 20] = np.nan
    y = s.rhs_mvec(E, w, dt).cpu().numpy()
    assert np.all(np.isnan(y[:, 20])) and np.all(np.isfinite(y[:, :15]))
    assert np.all(np.isnan(s.step_op_split(E, w, None, 0.0, dt).cpu().numpy()[:, 20]))
    again = s.rhs_mvec(E, v, dt).cpu().numpy(), s.step_op_split(E, v, None, 0.0, dt).cpu().numpy()
    assert np.array_equal(again[0], clean[0]) and np.array_equal(again[1], clean[1])
