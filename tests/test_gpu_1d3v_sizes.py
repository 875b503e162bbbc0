"""The FP64 products of the 1D3V steps (warps of 32 columns x 1 to 12 rows) off the benchmark's sizes:
the general product, the x-advection step, the v-space operator and the fully implicit operator
against dense NumPy at sizes around 32 columns, single rows and several rounds of warps. Tolerance
1e-12 of the largest value (FP64 sums of at most a few hundred terms; the x-step also carries the
conditioning of the radial eigenvectors, 1e-11)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (1, 33, 7), (12, 31, 40), (13, 32, 5), (25, 64, 3), (305, 200, 305),
                                   (700, 97, 9), (64, 3200, 64), (5, 101, 1000)])
def test_gemm_sizes(M, N, K):
    import torch
    from boltzmann_gb300 import _lib
    from boltzmann_gb300.native_kernels import _ptr, _stream
    rng = np.random.default_rng(M + N + K)
    A, B = rng.standard_normal((M, K + 1)), rng.standard_normal((K, N + 2))
    t = lambda a: torch.as_tensor(a, device="cuda")
    out = torch.full((M, N + 3), 7.0, dtype=torch.float64, device="cuda")
    dA, dB = t(A), t(B)
    assert _lib.load().bte_dgemm_nn(M, N, K, _ptr(dA), K + 1, _ptr(dB), N + 2, _ptr(out), N + 3, _stream()) == 0
    y = out.cpu().numpy()
    assert np.all(y[:, N:] == 7.0)
    scale = np.abs(A[:, :K]) @ np.abs(B[:, :N])
    assert np.max(np.abs(y[:, :N] - A[:, :K] @ B[:, :N]) / scale) <= K * 2.3e-16


@pytest.mark.parametrize("Np,Nr,Nvt,lmax", [(9, 7, 2, 1), (32, 8, 4, 2), (33, 11, 6, 1), (65, 16, 8, 2), (131, 9, 4, 3)])
def test_steps_and_operators(synthetic_xs, Np, Nr, Nvt, lmax):
    from boltzmann_gb300.bte_1d3v import bte_1d3v
    p = dict(L=2.54e-2, V0=100.0, freq=13.56e6, Tg=300.0, p0=1.0, atol=1e-14, rtol=1e-10, gmres_rsrt=30,
             gmres_rsrt_iter=20, max_iter=300, Np=Np, Nr=Nr, Nvt=Nvt, lmax=lmax, dt=1e-3, ev_max=80.0, ev_extend=0,
             sp_order=3, spline_qpts=5, Te=4.0, xspace_type=1, vspace_type=1, collisions=synthetic_xs,
             solver_type="fully_implicit")
    b = bte_1d3v(p)
    rng = np.random.default_rng(Np)
    nr, nsh, n = Nr + 1, lmax + 1, b.dof_v
    V = rng.standard_normal((nr, Nvt, Np))
    E = 3e3 * rng.standard_normal(Np)
    dt = 1e-3
    q = b.params
    Cv = q.tau * q.n0 * q.np0 * (b.op_col_en + q.Tg * b.op_col_gT).cpu().numpy()
    Av = q.tau * b.op_adv_v.cpu().numpy()
    X = rng.standard_normal((n, Np))
    want = X - dt * (Cv @ X + E[None, :] * (Av @ X))
    assert _rel(b.lmat_mvec(E, X, dt).cpu().numpy(), want) <= 1e-12
    cth = np.cos(b.xp_vt)
    D = np.repeat(b.Dp[None], Nvt, axis=0)
    flow = np.ones((Nvt, Np))
    for j in range(Nvt):
        D[j, 0 if cth[j] >= 0 else -1] = 0.0
        flow[j, 0 if cth[j] >= 0 else -1] = 0.0
    U = np.einsum("lj,rjx->xrl", b.op_po2sh, V).reshape(Np, n)
    yv = np.einsum("jl,xrl->rjx", b.op_psh2o, (U @ Cv.T + E[:, None] * (U @ Av.T)).reshape(Np, nr, nsh))
    yx = np.einsum("rk,kjx->rjx", b.op_adv_x, np.einsum("jxy,kjy->kjx", D, V)) * cth[:, None]
    want = (V - dt * (yv - yx) * flow).reshape(nr * Nvt, Np)
    assert _rel(b.fim_mvec(E, V.reshape(nr * Nvt, Np), dt).cpu().numpy(), want) <= 1e-12
    W = np.einsum("ik,kjx->ijx", b.op_adv_x_qinv, V) * flow
    for r in range(nr):
        for j in range(Nvt):
            W[r, j] = np.linalg.solve(np.eye(Np) + dt * b.op_adv_x_d[r] * cth[j] * D[j], W[r, j])
    want = np.einsum("ik,kjx->ijx", b.op_adv_x_q, W).reshape(nr * Nvt, Np)
    assert _rel(b.step_bte_x(V.reshape(nr * Nvt, Np), 0.0, dt).cpu().numpy(), want) <= 1e-11
