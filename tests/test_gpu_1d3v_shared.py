"""What calls on one 1D3V handle may do beside and on top of one another: the operator of the fully implicit
step on one stream while the v-step runs on another, and operators whose output is their input."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(synthetic_xs, Np=65, Nr=15, Nvt=8, lmax=1):
    from boltzmann_gb300.bte_1d3v import bte_1d3v
    b = bte_1d3v(dict(L=2.54e-2, V0=100.0, freq=13.56e6, Tg=300.0, p0=1.0, atol=1e-14, rtol=1e-10, gmres_rsrt=30,
                      gmres_rsrt_iter=20, max_iter=300, Np=Np, Nr=Nr, Nvt=Nvt, lmax=lmax, dt=1e-3, ev_max=80.0,
                      ev_extend=0, sp_order=3, spline_qpts=5, Te=4.0, xspace_type=1, vspace_type=1,
                      collisions=synthetic_xs))
    rng = np.random.default_rng(Np)
    V = b.initial_condition().cpu().numpy() * (1.0 + 0.2 * rng.standard_normal((b.dof_vr * b.dof_vt, Np)))
    return b, 3e3 * rng.standard_normal(Np), V


def test_implicit_operator_beside_the_v_step(synthetic_xs):
    """bte1d_fim_matvec queued on a second stream while bte1d_step_v works on the same handle: both give what they
    give alone."""
    import torch
    b, E, V = _solver(synthetic_xs)
    dt = 1e-3
    Vd, Ed = torch.as_tensor(V, device="cuda"), torch.as_tensor(E, device="cuda")
    alone_m, alone_v = b.fim_mvec(Ed, Vd, dt).clone(), b.step_bte_v(Ed, Vd, None, 0.0, dt).clone()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        with torch.cuda.stream(side):
            got = [b.fim_mvec(Ed, Vd, dt) for _ in range(60)]
        v = b.step_bte_v(Ed, Vd, None, 0.0, dt)
        torch.cuda.synchronize()
        assert all(torch.equal(y, alone_m) for y in got)
        assert torch.equal(v, alone_v)


@pytest.mark.parametrize("Np,Nr,lmax", [(9, 7, 1), (65, 15, 2), (201, 31, 1)])
def test_operators_in_place(synthetic_xs, Np, Nr, lmax):
    """bte1d_lmat and bte1d_fim_matvec with the output on their input: the same bits as into another buffer."""
    import torch
    from boltzmann_gb300 import _lib
    lib = _lib.load()
    b, E, V = _solver(synthetic_xs, Np=Np, Nr=Nr, lmax=lmax)
    Ed, st = torch.as_tensor(E, device="cuda"), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    X = torch.randn((Np, b.dof_v), device="cuda", dtype=torch.float64, generator=torch.Generator(device="cuda").manual_seed(Np))
    for f, x in ((lib.bte1d_lmat, X), (lib.bte1d_fim_matvec, torch.as_tensor(V, device="cuda").contiguous())):
        y, z = torch.empty_like(x), x.clone()
        assert f(b._h, 1e-3, _lib.ptr(Ed), _lib.ptr(x), _lib.ptr(y), st) == 0
        for _ in range(20):
            z.copy_(x)
            assert f(b._h, 1e-3, _lib.ptr(Ed), _lib.ptr(z), _lib.ptr(z), st) == 0
            torch.cuda.synchronize()
            assert torch.equal(z, y)
