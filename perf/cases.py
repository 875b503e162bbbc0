"""Performance cases: the calls a user of the package makes, at the sizes of its own configurations.

A case is a dict of plain values; `prepare` builds what a program holds before the call (solver object,
parameters, state), `run` makes one call through the public classes, `exact` gives the same outputs from dense
linear algebra in 64 bits on the assembled operators that the solver object holds, without the package's kernels.
"""
import math
import os
import types

import numpy as np
import torch

from boltzmann_gb300.bte_0d3v_batched import bte_0d3v_batched, vspace_grid_extension
from boltzmann_gb300.bte_1d3v import bte_1d3v
from boltzmann_gb300.bte_1d3v_fvm import bte_1d3v_fvm
from boltzmann_gb300.workloads import EV_MAX, TE_NORM, batch_parameters, write_synthetic_lxcat

QE, ME, KB, EPS0 = 1.602176634e-19, 9.1093837139e-31, 1.380649e-23, 8.8541878188e-12
C_GAMMA = math.sqrt(2.0 * QE / ME)

# Newton options of the reference's driver, as bench.py and the tests pass them
ATOL, RTOL, MAXIT, ALPHA = 1e-20, 1e-14, 100, (1e-16, 0.5, 1e-4)

# the 1D3V parameter tables of bench.py (200 x points, 64 B-splines, 16 ordinates); a case replaces the sizes
SPECTRAL = dict(L=2.54e-2, V0=100.0, freq=13.56e6, Tg=300.0, p0=1.0, atol=1e-14, rtol=1e-10, gmres_rsrt=30,
                gmres_rsrt_iter=20, max_iter=300, Np=200, Nr=63, Nvt=16, lmax=1, dt=1e-3, ev_max=80.0, ev_extend=0,
                sp_order=3, spline_qpts=5, Te=4.0, xspace_type=1, vspace_type=1)
FVM = dict(L=2.54e-2, V0=100.0, freq=13.56e6, Tg=300.0, p0=1.0, atol=1e-14, rtol=1e-10, gmres_rsrt=30,
           gmres_rsrt_iter=20, Np=200, Nr=63, Nvt=16, lmax=1, dt=1e-3, ev_max=80.0, ev_extend=0, sp_order=3,
           spline_qpts=5, Te=4.0, xspace_type=0, vspace_type=0, adaptive_grid=1, pvr=2, pvt=2, px=2, ic_file="")

# Exponents of the sweeps' ionization degree and of E/N in Td: the benchmark's ranges, as far as 64 bits determine
# the answer on the finest grid. Coulomb-dominated points (higher ionization at a few Td) move by 1e-8 with any change
# of rounding, and above some 200 Td the 80 eV grid no longer holds the distribution: single points there have no
# root that Newton's method reaches.
ION_RANGE, EBYN_RANGE = (-8.0, -4.5), (0.5, 2.3)


def listed():
    return [
        # one operating point of a fluid code's table look-up: the smallest grid of the benchmarks, default precision
        dict(name="point_fp64", kind="steady", n_sp=64, l_max=1, points=1, ee=False, precision="fp64"),
        # a handful of points with electron-electron collisions at the benchmark's grid, default precision
        dict(name="few_ee_fp64", kind="steady", n_sp=128, l_max=2, points=16, ee=True, precision="fp64"),
        # a request of the serving mix (bench.py serves 64 to 256 splines, l_max 1 to 3, 1 to 512 points): odd point count
        dict(name="request_mixed", kind="steady", n_sp=96, l_max=3, points=137, ee=True, precision="mixed"),
        # the benchmark's batch: 4096 points of a parameter sweep, 385 x 385 systems
        dict(name="batch_mixed", kind="steady", n_sp=128, l_max=2, points=4096, ee=True, precision="mixed"),
        # the same sweep without electron-electron collisions in the default precision
        dict(name="batch_fp64", kind="steady", n_sp=64, l_max=1, points=1000, ee=False, precision="fp64"),
        # the finest grid of the serving mix, above the tensor-core factorization's size (N = 769)
        dict(name="fine_mixed", kind="steady", n_sp=256, l_max=2, points=75, ee=True, precision="mixed"),
        # one radio-frequency period of the transient solve
        dict(name="transient_rf", kind="transient", n_sp=64, l_max=1, points=24, steps=40),
        # the 1D3V Strang split step at an odd size, and the benchmark's fully implicit step
        dict(name="strang_odd", kind="spectral", solver="strang", Np=101, Nr=47, Nvt=8, lmax=1),
        dict(name="implicit_spectral", kind="spectral", solver="fully_implicit", Np=200, Nr=63, Nvt=16, lmax=1),
        # the finite-volume 1D3V steps: the op-split step at an odd size, the benchmark's implicit step
        dict(name="split_fvm_odd", kind="fvm", solver="XVTVRC", Np=101, Nr=31, Nvt=8),
        dict(name="implicit_fvm", kind="fvm", solver="fully_implicit", Np=200, Nr=63, Nvt=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steady", "steady", "steady", "steady", "transient", "spectral", "spectral", "fvm", "fvm"])
    if kind == "steady":
        precision = rng.choice(["fp64", "mixed", "mixed"])
        l_max = rng.choice([1, 2, 3])
        n_sp = _log_int(rng, 56, min(256, 768 // (l_max + 1)))
        ee = rng.random() < 0.6
        # the cost of a batch goes with points * N^3; the FP64 factorizations and the sizes above 512 cost more each
        N = n_sp * (l_max + 1) + 1
        cost = N ** 3 * (4.0 if precision == "fp64" else 1.0) * (2.0 if N > 512 else 1.0)
        most = 0.5 * 4096 * 385 ** 3 / cost
        points = _log_int(rng, 1, max(2, min(4096, most)))
        return dict(kind=kind, n_sp=n_sp, l_max=l_max, points=points, ee=ee, precision=precision)
    if kind == "transient":
        return dict(kind=kind, n_sp=_log_int(rng, 48, 96), l_max=1, points=_log_int(rng, 1, 48),
                    steps=rng.choice([16, 25, 40]))
    if kind == "spectral":
        return dict(kind=kind, solver=rng.choice(["strang", "fully_implicit"]), Np=_log_int(rng, 25, 200),
                    Nr=_log_int(rng, 15, 63), Nvt=rng.choice([4, 8, 16]), lmax=rng.choice([1, 2]))
    return dict(kind=kind, solver=rng.choice(["XVTVRC", "fully_implicit", "sl_implicit"]), Np=_log_int(rng, 25, 200),
                Nr=_log_int(rng, 9, 63), Nvt=rng.choice([4, 8, 16]))


def _xs():
    """The package's synthetic cross sections, written once per process."""
    if not hasattr(_xs, "path") or not os.path.exists(_xs.path):
        _xs.path = write_synthetic_lxcat()
    return _xs.path


def _field(xp, t, p):
    """bench.py's field of the 1D3V workload: (V0 / gap) sin(2 pi t), ramped over x."""
    return (p["V0"] / p["L"]) * np.sin(2 * np.pi * t) * 0.5 * (1.0 + np.asarray(xp))


def _solver_0d(c, ee):
    args = types.SimpleNamespace(threads=1, sp_order=3, spline_qpts=5, ee_collisions=int(ee), verbose=0, use_gpu=1,
                                 Efreq=0.0, dt=1e-3, cycles=1, solver_type="steady-state", l_max=c["l_max"],
                                 Nr=c["n_sp"] - 1, n_pts=c["points"], precision=c.get("precision", "fp64"))
    s = bte_0d3v_batched(args, np.array([EV_MAX]), np.array([TE_NORM]), np.array([c["n_sp"] - 1]),
                         [[[l, 0] for l in range(c["l_max"] + 1)]], 1, [_xs()])
    s.assemble_operators(0, vspace_ext=vspace_grid_extension.NONE)
    return s, args


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "steady":
        # parameters of the benchmark's sweep: E/N and the ionization degree log-uniform
        s, args = _solver_0d(case, case["ee"])
        prm = batch_parameters(case["points"], seed, ion_deg_range=ION_RANGE, ebyn_range=EBYN_RANGE, ee=case["ee"])
    elif kind == "transient":
        s, args = _solver_0d(case, False)
        prm = batch_parameters(case["points"], seed, ebyn_range=(1.0, EBYN_RANGE[1]), ee=False)
        phase = rng.uniform(0.0, 2.0 * np.pi, case["points"])
        prm["eRe"], prm["eIm"] = prm["E"] * np.cos(phase), prm["E"] * np.sin(phase)
        args.Efreq, args.dt, args.cycles = 13.56e6, 1.0 / case["steps"], 1.0
    elif kind == "spectral":
        p = dict(SPECTRAL, collisions=_xs(), Np=case["Np"], Nr=case["Nr"], Nvt=case["Nvt"], lmax=case["lmax"])
        if case["solver"] == "fully_implicit":
            p["solver_type"] = "fully_implicit"
        return _state_1d(case, bte_1d3v(p), p, rng)
    else:
        p = dict(FVM, collisions=_xs(), Np=case["Np"], Nr=case["Nr"], Nvt=case["Nvt"], solver_type=case["solver"])
        b = bte_1d3v_fvm(p)
        b.init(p["dt"])
        return _state_1d(case, b, p, rng)
    for k in ("n0", "ne", "ns_by_n0", "Tg", "E", "eRe", "eIm"):
        if k in prm:
            s.set_boltzmann_parameter(0, k, prm[k])
    s.host_to_device_setup(0, 0)
    return dict(case=case, s=s, args=args, f0=torch.as_tensor(s.initialize(0, case["points"]), device="cuda"))


def _state_1d(case, b, p, rng):
    """The initial profile with a smooth random modulation over x, and the field at a random time of the period."""
    v = b.initial_condition()
    x = np.asarray(b.xp)
    mod = 1.0 + 0.2 * sum(rng.uniform(-1, 1) * np.cos(np.pi * k * (x + 1) / 2) for k in range(1, 5))
    v = (v * torch.as_tensor(mod, device="cuda")[None, :]).contiguous()
    t = rng.uniform(0.1, 0.4)
    return dict(case=case, b=b, v=v, t=t, dt=p["dt"], E=torch.as_tensor(_field(x, t, p), device="cuda"))


def run(state):
    case = state["case"]
    if case["kind"] == "steady":
        s, args = state["s"], state["args"]
        f = state["f0"]
        if case["ee"]:  # the driver's sequence: warm start without e-e collisions, then with them
            args.ee_collisions = 0
            f, _ = s.solve(0, f, ATOL, RTOL, MAXIT, "steady-state", *ALPHA)
            args.ee_collisions = 1
        f, q = s.solve(0, f, ATOL, RTOL, MAXIT, "steady-state", *ALPHA)
        return {"f": f, "energy": q["energy"], "mobility": q["mobility"], "diffusion": q["diffusion"],
                "rates": q["rates"]}
    if case["kind"] == "transient":
        u, q = state["s"].solve(0, state["f0"], 1e-30, 1e-10, 200, "transient")
        return {"u": u, "energy": q["energy"], "mobility": q["mobility"], "diffusion": q["diffusion"],
                "rates": q["rates"]}
    return state["b"].step(state["E"], state["v"], None, state["t"], state["dt"])


def work(case):
    """What the call cannot do without. Solves: parameters, operators and states once, and one factorization per
    Newton solve and point (per time step of the transient). Steps: the state in and out, the operator once."""
    if case["kind"] in ("steady", "transient"):
        nsp, nsh, P = case["n_sp"], case["l_max"] + 1, case["points"]
        n = nsp * nsh
        N = n + 1
        ee = bool(case.get("ee"))
        solves = case["steps"] if case["kind"] == "transient" else 2 if ee else 1
        ops = nsp * nsp + 35 * nsp + (2 * nsh * nsp * nsp if ee else 0)
        return {"bytes": 8.0 * (2 * n * P + 12 * P + ops), "flops": solves * P * ((2.0 / 3.0) * N ** 3 + 2.0 * N * N)}
    if case["kind"] == "spectral":
        Nr, Nvt, Nx, n = case["Nr"] + 1, case["Nvt"], case["Np"], (case["Nr"] + 1) * (case["lmax"] + 1)
        x = 2.0 * Nr * Nvt * Nx * Nx + 2.0 * Nr * Nr * Nvt * Nx
        return {"bytes": 16.0 * Nr * Nvt * Nx + 16.0 * n * n, "flops": 2.0 * x + 4.0 * n * n * Nx}
    Nr, Nvt, Nx = 5 * (case["Nr"] - 2), case["Nvt"], case["Np"]
    return {"bytes": 16.0 * Nr * Nvt * Nx + 8.0 * Nr * Nr, "flops": 60.0 * Nr * Nvt * Nx + 2.0 * Nr * Nr * Nx}


# ------------------------------------------------------------------ the same results from dense 64-bit algebra
def exact(case, seed):
    kind = case["kind"]
    if kind == "steady":
        N = case["n_sp"] * (case["l_max"] + 1) + 1
        if case["points"] * N ** 3 > 4e10:  # the batch: dense factorizations of every point take over 20 seconds
            return None
    state = prepare(case, seed)
    if kind == "steady":
        return _exact_steady(state)
    if kind == "transient":
        return _exact_transient(state)
    if kind == "spectral":
        return _exact_spectral(state)
    return _exact_fvm(state)


class _Dense0D:
    """F(h) = n0 sum_s ns C_s h + n0 Tg C_T h + E A h - (w . h) M h + ne gamma(h) U(h, h) and its derivative for a
    batch of states (P, n), from the dense assembled operators."""

    def __init__(self, state, ee):
        s, case = state["s"], state["case"]
        info = s._grid_info[0]
        x = lambda k: s.export_operator(0, k)
        self.n, self.nsh, self.vth, self.mw0 = info["n"], info["num_sh"], info["vth"], info["mw0"]
        n, P = self.n, case["points"]
        prm = s._par_bte_params[0]
        dev = lambda k: torch.as_tensor(prm[k], dtype=torch.float64, device="cuda")
        self.n0, self.ne, self.Tg, self.E, self.ns = (dev(k) for k in ("n0", "ne", "Tg", "E", "ns_by_n0"))
        self.M, self.mass, self.temp = x("MASS"), x("MASS_VEC"), x("TEMP_VEC")
        self.mob, self.diff, self.rate = x("MOBILITY"), x("DIFFUSION"), x("RATES")
        self.A = x("ADV_RAW") * (QE / ME / self.vth)
        self.u = self.mass * (self.mw0 * self.vth ** 3)
        self.p = self.u / torch.linalg.norm(self.u)
        self.Mp = self.M @ self.p
        col = x("COL_RAW")
        v = torch.linalg.solve(self.M.t(), self.u)
        nsx = self.n0 * self.ns  # (species, P)
        self.w = torch.einsum("sx,su->xu", nsx, torch.einsum("v,svu->su", v, col))
        self.C = torch.einsum("sx,svu->xvu", nsx, col) + (self.n0 * self.Tg)[:, None, None] * x("COL_GT_RAW")
        self.d = 1.0 / torch.diagonal(self.M)
        self.q = self.d * self.Mp
        self.q = self.q / torch.linalg.norm(self.q)
        self.cc = None
        if ee:
            self.cc = x("CC_A").reshape(n * n, n) @ x("HL")
            self.cc += x("CC_B").reshape(n * n, n) @ x("GL")
            self.cc = self.cc.reshape(n, n, n)

    def rows(self, h, E, jac=True):
        """(F, dF/dh) at h (P, n) and field E (P)."""
        mu = (self.w * h).sum(1)
        Mh = h @ self.M.t()
        L = self.C + E[:, None, None] * self.A
        F = torch.einsum("xab,xb->xa", L, h) - mu[:, None] * Mh
        J = (L - mu[:, None, None] * self.M - Mh[:, :, None] * self.w[:, None, :]) if jac else None
        if self.cc is not None:
            n, P = self.n, h.shape[0]
            m, t = h @ self.mass, h @ (self.temp * (QE / KB))
            kT = (t / m * self.vth ** 2 * KB).abs()
            cl = 12 * math.pi * (EPS0 * kT) ** 1.5 / (QE ** 3 * torch.sqrt(self.ne))
            g = QE ** 4 / (4 * math.pi * (EPS0 * ME) ** 2) / self.vth ** 3
            gam = self.ne * torch.log(cl) * g
            K2 = (self.cc.reshape(n * n, n) @ h.t()).reshape(n, n, P)
            U = torch.einsum("abx,xb->xa", K2, h)
            F = F + gam[:, None] * U
            if jac:
                K1 = torch.einsum("abc,xb->xac", self.cc, h)
                dg = 1.5 * g * self.ne[:, None] * (self.temp * (QE / KB) / t[:, None] - self.mass / m[:, None])
                J = J + gam[:, None, None] * (K2.permute(2, 0, 1) + K1) + U[:, :, None] * dg[:, None, :]
        return F, J

    def solve(self, J, F, rhs, scale):
        """The step of the bordered systems [J, -s Mp; s u, 0] [x; l] = [-F; s rhs], rows scaled to unit size."""
        P, n = F.shape
        B = torch.zeros((P, n + 1, n + 1), dtype=torch.float64, device="cuda")
        B[:, :n, :n] = J
        B[:, :n, n] = -scale[:, None] * self.Mp
        B[:, n, :n] = scale[:, None] * self.u
        r = torch.cat([-F, (scale * rhs)[:, None]], dim=1)
        top = B.abs().amax(dim=2)
        B /= top[:, :, None]
        lu, piv = torch.linalg.lu_factor(B)
        x = torch.linalg.lu_solve(lu, piv, (r / top)[:, :, None])
        return x[:, :n, 0]

    def merit(self, F):
        y = F * self.d
        return torch.linalg.norm(y - (y @ self.q)[:, None] * self.q, dim=1)

    def newton(self, h):
        """Steady states u . h = 1, F(h) parallel to M p, by Newton's method with halved steps."""
        h = h / (h @ self.u)[:, None]
        scale = self.C.abs().amax(dim=(1, 2)) / self.u.abs().max()
        F, J = self.rows(h, self.E)
        r = self.merit(F)
        r0 = r.clone()
        running = torch.ones_like(r, dtype=torch.bool)
        for _ in range(60):
            x = self.solve(J, F, 1.0 - h @ self.u, scale)
            small = torch.linalg.norm(x, dim=1) <= 1e-8 * torch.linalg.norm(h, dim=1)
            a, taken = torch.ones_like(r), ~running
            for _ in range(20):
                Ft, _ = self.rows(h + (a * running)[:, None] * x, self.E, jac=False)
                taken = taken | (self.merit(Ft) < r) | (small & (a == 1.0))
                if bool(taken.all()):
                    break
                a = torch.where(taken, a, 0.5 * a)
            h = h + (a * (running & taken))[:, None] * x
            F, J = self.rows(h, self.E)
            rn = self.merit(F)
            running = running & taken & ~((rn >= 0.5 * r) & (rn <= 1e-9 * r0)) & (rn > 1e-15 * r0)
            r = rn
            if not bool(running.any()):
                break
        return h

    def normalized(self, h):
        return h / ((h @ self.mass) / math.sqrt(4 * math.pi) * 2.0 * (self.vth / C_GAMMA) ** 3)[:, None]

    def qoi(self, f, effective):
        f0 = f[:, 0::self.nsh]
        field = self.E / self.n0 if effective else 1.0 / self.n0
        return {"energy": 1.5 * (f @ self.temp) / (f @ self.mass) * self.vth ** 2,
                "mobility": (f[:, 1::self.nsh] @ self.mob) * math.sqrt(3.0) * (-C_GAMMA / (3.0 * field)),
                "diffusion": (f0 @ self.diff) * (C_GAMMA / 3.0), "rates": (f0 @ self.rate.t()).t().contiguous()}


def _exact_steady(state):
    case, h = state["case"], state["f0"].t()
    o = _Dense0D(state, False)
    h = o.newton(h)
    if case["ee"]:
        o = _Dense0D(state, True)
        h = o.newton(h)
    f = o.normalized(h)
    return dict(o.qoi(f, True), f=f.t())


def _exact_transient(state):
    case, o = state["case"], _Dense0D(state, False)
    prm = state["s"]._par_bte_params[0]
    eRe, eIm = (torch.as_tensor(prm[k], dtype=torch.float64, device="cuda") for k in ("eRe", "eIm"))
    h = state["f0"].t()
    h = h / (h @ o.u)[:, None]
    dt = 1.0 / case["steps"]
    c = dt / 13.56e6
    scale = torch.full_like(o.n0, float(o.M.abs().max() / o.u.abs().max()))
    total, d = torch.zeros_like(h), torch.zeros_like(h)
    for k in range(case["steps"]):
        t = (k + 1) * dt
        E = eRe * math.cos(2 * math.pi * t) + eIm * math.sin(2 * math.pi * t)
        d = torch.zeros_like(h)
        for _ in range(8):  # M d - c F(h + d) parallel to M p, u . d = 0
            F, J = o.rows(h + d, E)
            x = o.solve(o.M - c * J, d @ o.M.t() - c * F, -(d @ o.u), scale)
            d = d + x
            if float((torch.linalg.norm(x, dim=1) / torch.linalg.norm(h, dim=1)).max()) < 1e-14:
                break
        total += 0.5 * dt * (h + h + d)
        h = h + d
    return dict(o.qoi(o.normalized(total), False), u=h.t())


def _gmres(A, M, b, tol=1e-14, m=60, rounds=6):
    """Restarted right-preconditioned GMRES in 64 bits on flat tensors."""
    x = M(b)
    nb = float(torch.linalg.norm(b))
    for _ in range(rounds):
        r = b - A(x)
        beta = float(torch.linalg.norm(r))
        if beta <= tol * nb:
            break
        V = torch.zeros((m + 1, b.numel()), dtype=torch.float64, device="cuda")
        H = torch.zeros((m + 1, m), dtype=torch.float64)
        V[0] = r / beta
        k = m
        for j in range(m):
            w = A(M(V[j]))
            for _ in range(2):
                hj = V[: j + 1] @ w
                w = w - hj @ V[: j + 1]
                H[: j + 1, j] += hj.cpu()
            nw = float(torch.linalg.norm(w))
            H[j + 1, j] = nw
            if nw <= 1e-300:
                k = j + 1
                break
            V[j + 1] = w / nw
        e = torch.zeros(k + 1, 1, dtype=torch.float64)
        e[0] = beta
        y = torch.linalg.lstsq(H[: k + 1, :k], e).solution[:, 0].to("cuda")
        x = x + M(y @ V[:k])
    return x


def _exact_spectral(state):
    b, p, E, dt = state["b"], state["b"].params, state["E"], state["dt"]
    Nr, Nvt, Nx, n = b.dof_vr, b.dof_vt, b.dof_x, b.dof_v
    nsh = n // Nr
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    Cv = p.tau * p.n0 * p.np0 * (b.op_col_en + p.Tg * b.op_col_gT)
    Av = p.tau * b.op_adv_v
    Q, Qi, d, ax = dev(b.op_adv_x_q), dev(b.op_adv_x_qinv), dev(b.op_adv_x_d), dev(b.op_adv_x)
    cth, Po, Ps, D = dev(np.cos(b.xp_vt)), dev(b.op_psh2o), dev(b.op_po2sh), dev(b.Dp)
    right = cth >= 0
    DL, DR = D.clone(), D.clone()
    DL[0], DR[-1] = 0.0, 0.0
    Dj = torch.where(right[:, None, None], DL, DR)  # (Nvt, Nx, Nx)
    flow = torch.ones((Nvt, Nx), dtype=torch.float64, device="cuda")
    flow[right, 0] = 0.0
    flow[~right, -1] = 0.0
    eye, eyen = torch.eye(Nx, dtype=torch.float64, device="cuda"), torch.eye(n, dtype=torch.float64, device="cuda")
    blocks = torch.linalg.inv(eyen - dt * (Cv + E[:, None, None] * Av))  # (Nx, n, n)

    def x_inverse(h):
        return torch.linalg.inv(eye + h * d[:, None, None, None] * cth[:, None, None] * Dj)  # (Nr, Nvt, Nx, Nx)

    def x_step(V, inv):
        W = torch.einsum("ik,kjx->ijx", Qi, V) * flow
        return torch.einsum("ik,kjx->ijx", Q, torch.einsum("rjxy,rjy->rjx", inv, W))

    def to_lm(V):
        return torch.einsum("lj,rjx->xrl", Ps, V).reshape(Nx, n)

    def to_ords(U):
        return torch.einsum("jl,xrl->rjx", Po, U.reshape(Nx, Nr, nsh))

    V = state["v"].reshape(Nr, Nvt, Nx)
    if state["case"]["solver"] == "strang":
        inv = x_inverse(0.5 * dt)
        V = to_ords(torch.einsum("xab,xb->xa", blocks, to_lm(x_step(V, inv))))
        return x_step(V, inv).reshape(Nr * Nvt, Nx)
    inv = x_inverse(dt)

    def A(v):
        V = v.reshape(Nr, Nvt, Nx)
        U = to_lm(V)
        yv = to_ords(U @ Cv.t() + E[:, None] * (U @ Av.t()))
        yx = torch.einsum("rk,kjx->rjx", ax, torch.einsum("jxy,kjy->kjx", Dj, V)) * cth[:, None]
        return (V - dt * (yv - yx) * flow).reshape(-1)

    def M(v):
        V = v.reshape(Nr, Nvt, Nx)
        U = to_lm(V)
        return x_step(V + to_ords(torch.einsum("xab,xb->xa", blocks, U) - U), inv).reshape(-1)

    return _gmres(A, M, (V * flow).reshape(-1)).reshape(Nr * Nvt, Nx)


def _exact_fvm(state):
    b, p, E, dt = state["b"], state["b"].params, state["E"], state["dt"]
    Nr, Nvt, Nx = b.dof_vr, b.dof_vt, b.dof_x
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    vr, vt, x = dev(b.grid_info["vr"]), dev(b.grid_info["vt"]), dev(b.xp)
    w = 2 * math.pi * dev(b.grid_info["vt_qw"])
    gain, loss = dev(b.op_col.gain), dev(b.op_col.loss)
    cth = torch.cos(vt)
    kappa, cA, ax = p.n0 * p.np0, QE / ME / b.bs_vth, b.bs_vth * (p.tau / p.L)
    V = state["v"].reshape(Nr, Nvt, Nx)

    def collisions(V):  # (I - c C)^-1 through the ordinate moments, c = dt tau kappa
        c = dt * p.tau * kappa
        dd = 1.0 + c * loss
        m = torch.linalg.solve(torch.diag(dd) - c * w.sum() * gain, torch.einsum("j,rjx->rx", w, V))
        return (V + c * (gain @ m)[:, None, :]) / dd[:, None, None]

    if state["case"]["solver"] == "sl_implicit":
        return collisions(_departures(V, vr, vt, x, b.vmax, E, dt * ax, dt * p.tau * cA)).reshape(Nr * Nvt, Nx)

    def dense(l, u, N):
        out = []
        for B, s in ((dev(l), -1), (dev(u), 1)):
            Dm = torch.zeros((N, N), dtype=torch.float64, device="cuda")
            for k in range(B.shape[0]):
                i = torch.arange(N, device="cuda")
                i = i[(i + s * k >= 0) & (i + s * k < N)]
                Dm[i, i + s * k] = B[k][i + s * k]
            out.append(Dm)
        return out

    vrL, vrR = dense(b.bands["vr_diag_l2r"], b.bands["vr_diag_r2l"], Nr)
    vtL, vtR = dense(b.bands["vt_diag_l2r"], b.bands["vt_diag_r2l"], Nvt)
    xL, xR = dense(b.bands["x_diag_l2r"], b.bands["x_diag_r2l"], Nx)
    north = vt <= 0.5 * math.pi
    flow = torch.ones((Nvt, Nx), dtype=torch.float64, device="cuda")
    flow[north, 0] = 0.0
    flow[~north, -1] = 0.0
    pick = lambda c, a, b2: torch.where(c[..., None, None], a, b2)
    one = lambda N: torch.eye(N, dtype=torch.float64, device="cuda")
    aE = p.tau * cA * E
    a1 = -aE[None, :] * cth[:, None]                      # (Nvt, Nx)
    i1 = torch.linalg.inv(one(Nr) + dt * a1[..., None, None] * pick(a1 >= 0, vrL, vrR))
    a2 = aE[None, :] / vr[:, None]                        # (Nr, Nx)
    i2 = torch.linalg.inv(one(Nvt) + dt * a2[..., None, None] * pick(-a2 >= 0, vtL, vtR))
    a3 = ax * vr[:, None] * cth[None, :]                  # (Nr, Nvt)
    i3 = torch.linalg.inv(one(Nx) + dt * a3[..., None, None] * pick(a3 >= 0, xL, xR))

    def split(V):
        V = collisions(V)
        V = torch.einsum("jxab,bjx->ajx", i1, V)
        V = torch.einsum("rxab,rbx->rax", i2, V)
        return torch.einsum("rjab,rjb->rja", i3, V * flow)

    if state["case"]["solver"] == "XVTVRC":
        return split(V).reshape(Nr * Nvt, Nx)
    dx = torch.where(north[:, None, None], xL, xR)        # (Nvt, Nx, Nx)
    up = (E[None, :] >= 0) == (cth[:, None] > 0)          # (Nvt, Nx)
    low = E < 0

    def A(v):
        V = v.reshape(Nr, Nvt, Nx)
        yx = V + dt * ax * vr[:, None, None] * cth[None, :, None] * torch.einsum("jab,rjb->rja", dx, V)
        dr = torch.where(up[None], torch.einsum("ab,bjx->ajx", vrR, V), torch.einsum("ab,bjx->ajx", vrL, V))
        dth = torch.where(low, torch.einsum("ab,rbx->rax", vtL, V), torch.einsum("ab,rbx->rax", vtR, V))
        adv = cth[None, :, None] * dr - dth / vr[:, None, None]
        col = (gain @ torch.einsum("j,rjx->rx", w, V))[:, None, :] - loss[:, None, None] * V
        return (yx - flow * dt * p.tau * (kappa * col + E * cA * adv)).reshape(-1)

    return _gmres(A, lambda v: split(v.reshape(Nr, Nvt, Nx)).reshape(-1), (V * flow).reshape(-1)).reshape(Nr * Nvt, Nx)


def _departures(V, vr, vt, x, vmax, E, cX, cE):
    """Trilinear interpolation of V at each value's departure point on the grid padded by one layer in v_r and
    theta (linear extrapolation below the first cell and past the first and last ordinate, zero at vmax)."""
    Nr, Nvt, Nx = V.shape
    lo = V[0] - vr[0] * (V[1] - V[0]) / (vr[1] - vr[0])
    G = torch.cat([lo[None], V, torch.zeros_like(V[:1])])
    first = G[:, 0] + (math.pi - vt[0]) * (G[:, 1] - G[:, 0]) / (vt[1] - vt[0])
    last = G[:, -1] - vt[-1] * (G[:, -1] - G[:, -2]) / (vt[-1] - vt[-2])
    # the corner layer extrapolates each direction from the first cell
    first[0] = lo[0] + (math.pi - vt[0]) * (V[0, 1] - V[0, 0]) / (vt[1] - vt[0])
    last[0] = lo[-1] - vt[-1] * (V[0, -1] - V[0, -2]) / (vt[-1] - vt[-2])
    G = torch.cat([first[:, None], G, last[:, None]], dim=1).flip(1)   # theta ascending
    z = torch.zeros(1, dtype=torch.float64, device="cuda")
    gr = torch.cat([z, vr, z + vmax])
    gt = torch.cat([z, vt.flip(0), z + math.pi])
    c = vr[:, None] * torch.cos(vt)[None, :]
    dE = cE * E
    xa = x[None, None, :] - cX * c[:, :, None]
    va = torch.sqrt(vr[:, None, None] ** 2 + 2 * c[:, :, None] * dE + dE * dE)
    ta = torch.acos(((c[:, :, None] + dE) / va).clamp(-1.0, 1.0))
    xa = xa.expand_as(va)
    ok = (va >= gr[0]) & (va <= gr[-1]) & (ta >= gt[0]) & (ta <= gt[-1]) & (xa >= x[0]) & (xa <= x[-1])

    def place(g, q):
        i = (torch.searchsorted(g, q.contiguous()) - 1).clamp(0, g.numel() - 2)
        return i, (q - g[i]) / (g[i + 1] - g[i])

    (i, a), (j, b), (k, d) = place(gr, va), place(gt, ta), place(x, xa)
    out = torch.zeros_like(va)
    for di in (0, 1):
        for dj in (0, 1):
            for dk in (0, 1):
                wgt = (a if di else 1 - a) * (b if dj else 1 - b) * (d if dk else 1 - d)
                out += wgt * G[i + di, j + dj, k + dk]
    return torch.where(ok, out, torch.zeros_like(out))
