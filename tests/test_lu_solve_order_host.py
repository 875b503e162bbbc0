"""The order of the substitution's diagonal blocks (boltzmann_gb300/csrc/lu_solve_form.h, used by
k_lu_solve), walked on the host: per step the block's owner arrives at a named barrier and goes on, every
other warp waits there. With any one warp held back as long as the others can go on, a barrier must open
only when every warp has come to the same step, or a warp would read a block that nobody has solved."""
import ctypes
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    so = str(tmp_path_factory.mktemp("lus") / "lu_solve_harness.so")
    r = subprocess.run([cxx, "-O1", "-std=c++17", "-shared", "-fPIC",
                        os.path.join(HERE, "host", "lu_solve_harness.cpp"), "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(so)


def _shape(lib, elem, P, N):
    out = (ctypes.c_int * 4)()
    lib.solve_shape(elem, P, N, out)
    return list(out)


def _walk(ops, warps, late):
    """ops[w]: (step, barrier, waits). Runs every warp but `late` as far as it can go, then `late` by one
    operation, and so on. Returns the first step whose barrier opened with arrivals that are not one of each
    warp for that step, "hang" if nobody can go on, or None."""
    at = [0] * warps
    blocked = [False] * warps
    inside = {}                                  # barrier -> (warp, step, waits) of the open phase

    def go(w):
        step, bar, waits = ops[w][at[w]]
        phase = inside.setdefault(bar, [])
        phase.append((w, step, waits))
        blocked[w] = waits
        if not waits:
            at[w] += 1
        if len(phase) < warps:
            return None
        inside[bar] = []
        for v, _, vw in phase:
            if vw:
                blocked[v] = False
                at[v] += 1
        return None if len({p[0] for p in phase}) == warps and len({p[1] for p in phase}) == 1 else step

    def ready(w):
        return at[w] < len(ops[w]) and not blocked[w]

    while any(at[w] < len(ops[w]) for w in range(warps)):
        w = next((v for v in range(warps) if v != late and ready(v)), late)
        if not ready(w):
            return "hang"
        bad = go(w)
        if bad is not None:
            return bad
    return None


@pytest.mark.parametrize("elem", [4, 8], ids=["f32", "f64"])
@pytest.mark.parametrize("N,P", [(1, 1), (33, 1), (129, 1000), (256, 1), (257, 1), (385, 305), (512, 1), (513, 1),
                                 (1024, 4), (1025, 1), (1400, 1), (1401, 1), (1500, 3), (2048, 1)])
def test_no_barrier_opens_early(lib, elem, N, P):
    width, warps, most, rows = _shape(lib, elem, P, N)
    assert 1 <= warps <= most and warps * rows * 32 >= N
    blocks = (N + width - 1) // width
    for backward in (False, True):
        ops = [[] for _ in range(warps)]
        for t in range(blocks - 1):              # the last step has no barrier
            block = blocks - 1 - t if backward else t
            owner = lib.solve_step_owner(block, width, warps)
            for w in range(warps):
                ops[w].append((t, lib.solve_step_barrier(t), w != owner))
        for late in range(warps):
            assert _walk(ops, warps, late) is None, (width, warps, late)


def test_barriers_fit_the_hardware(lib):
    """A CTA has sixteen named barriers; 0 is __syncthreads()."""
    assert all(1 <= lib.solve_step_barrier(t) <= 15 for t in range(64))
