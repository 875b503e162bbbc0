"""The finite-volume handle at the ends of what it takes: very many lines, and a device without room for
what only makes it faster."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Handle:
    """A handle of the C interface with first-order bands and a random collision operator."""

    def __init__(self, Nr, Nvt, Nx, seed=0):
        from boltzmann_gb300 import _lib
        self.lib, self.shape = _lib.load(), (Nr, Nvt, Nx)
        rng = np.random.default_rng(seed)
        dp = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
        c = lambda a: np.ascontiguousarray(a, dtype=np.float64)
        band = lambda n, s: c(np.stack([np.full(n, s), np.full(n, -s)]))
        self.w = c(rng.uniform(0.5, 1.5, Nvt) / Nvt)
        self.dinv, self.H = c(rng.uniform(0.5, 1.0, Nr)), c(rng.uniform(-0.1, 0.1, (Nr, Nr)))
        self.vt = c(np.linspace(np.pi - 1e-3, 1e-3, Nvt))
        keep = [c(np.linspace(0.5, 5.0, Nr)), self.vt, self.w, c(rng.uniform(0, 1, Nr)), c(np.triu(rng.uniform(0, 1, (Nr, Nr)), 1)),
                band(Nr, 2.0), band(Nr, -2.0), band(Nvt, 0.3), band(Nvt, -0.3), band(Nx, 3.0), band(Nx, -3.0)]
        self.h = C.c_void_p()
        assert self.lib.bte_fvm_create(0, Nr, Nvt, Nx, 2, 2, 2, *[dp(a) for a in keep], C.byref(self.h)) == 0
        self._set = lambda: self.lib.bte_fvm_set_collision_inverse(self.h, dp(self.dinv), dp(self.H))

    def set_inverse(self):
        assert self._set() == 0, self.lib.bte_fvm_last_error()

    def precond(self, cE, ax, step, E, X):
        import torch
        Y = torch.empty_like(X)
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        rc = self.lib.bte_fvm_precond(self.h, cE, ax, step, E.data_ptr(), X.data_ptr(), Y.data_ptr(), st)
        assert rc == 0, self.lib.bte_fvm_last_error()
        torch.cuda.synchronize()
        return Y

    def close(self):
        self.lib.bte_fvm_destroy(self.h)


def test_more_lines_than_a_grid_has_rows():
    """2.2 million (v_r, theta) lines. Without field and drift the sweeps leave the collision solve as it is, and the
    x sweep zeroes the inflow values. Tolerance: the rounding of the moments' sums, Nvt eps of their size."""
    import torch
    Nr, Nvt, Nx = 2, 1_100_000, 2
    f = _Handle(Nr, Nvt, Nx)
    f.set_inverse()
    X = torch.rand((Nr, Nvt, Nx), device="cuda", dtype=torch.float64, generator=torch.Generator(device="cuda").manual_seed(1))
    got = f.precond(0.0, 0.0, 1e-3, torch.zeros(Nx, device="cuda", dtype=torch.float64), X).cpu().numpy()
    f.close()
    x = X.cpu().numpy()
    m = np.einsum("j,rjx->rx", f.w, x)
    want = f.dinv[:, None, None] * x + (f.H @ m)[:, None, :]
    north = f.vt <= 0.5 * np.pi
    want[:, north, 0] = 0.0
    want[:, ~north, Nx - 1] = 0.0
    assert np.max(np.abs(got - want)) <= Nvt * 2.3e-16 * np.max(np.abs(want))


def test_no_room_for_the_sweep_coefficients():
    """A device with less free memory than the sweeps' coefficients take: the handle works all the same, with the
    values of one that has them to 1e-12 of the largest (another order of the same operations)."""
    import torch
    Nr, Nvt, Nx = 64, 16, 4000
    g = torch.Generator(device="cuda").manual_seed(2)
    X = torch.rand((Nr, Nvt, Nx), device="cuda", dtype=torch.float64, generator=g)
    E = torch.randn(Nx, device="cuda", dtype=torch.float64, generator=g)
    a = _Handle(Nr, Nvt, Nx)
    a.set_inverse()
    want = a.precond(0.7, 0.4, 1e-2, E, X)
    a.close()
    b = _Handle(Nr, Nvt, Nx)
    spare = torch.empty(Nr * Nvt * Nx * 8, device="cuda", dtype=torch.uint8)   # the output's, and a little more
    torch.cuda.synchronize()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (128 << 20), device="cuda", dtype=torch.uint8)
    assert torch.cuda.mem_get_info()[0] < 6 * X.numel() * 8
    del spare
    try:
        b.set_inverse()
        got = b.precond(0.7, 0.4, 1e-2, E, X)
    finally:
        del fill
        torch.cuda.empty_cache()
    b.close()
    assert float((got - want).abs().max()) <= 1e-12 * float(want.abs().max())
