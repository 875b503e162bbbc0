"""The autotuner above the sizes of its candidates, and choices on disk that were made with other kernels: no GPU."""
import json
import types

import pytest

from boltzmann_gb300 import autotune


def test_above_512_the_library_chooses(tmp_path, monkeypatch):
    """Nothing is timed, read or stored, also with a choice of the right-looking kernel on disk."""
    monkeypatch.setenv("BOLTZMANN_GB300_CACHE", str(tmp_path))
    monkeypatch.setattr(autotune, "_mem", {})
    monkeypatch.setattr(autotune, "_key", lambda N, device: "fake|N=%d" % N)
    monkeypatch.setattr(autotune, "time_lu", lambda *a, **k: pytest.fail("timed"))
    (tmp_path / "lu_autotune.json").write_text(json.dumps({"fake|N=769": {"kernel": 1, "ms": {}, "P": 1}}))
    assert autotune.lu_kernel_for(769) == 0 and autotune.lu_kernel_for(513) == 0


def test_choices_of_earlier_kernels_are_not_read(tmp_path, monkeypatch):
    """A file from before the kernels changed names the GPU and the size alone."""
    import torch
    monkeypatch.setenv("BOLTZMANN_GB300_CACHE", str(tmp_path))
    monkeypatch.setattr(autotune, "_mem", {})
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device=0: "fake")
    monkeypatch.setattr(autotune, "time_lu", lambda N, kernel, **k: 1.0 if kernel == 2 else 2.0)
    (tmp_path / "lu_autotune.json").write_text(json.dumps({"fake|N=385": {"kernel": 3, "ms": {}, "P": 1}}))
    assert autotune.lu_kernel_for(385) == 2
    data = json.loads((tmp_path / "lu_autotune.json").read_text())
    assert data["fake|N=385"]["kernel"] == 3 and len(data) == 2


def test_solver_asks_the_tuner(monkeypatch):
    """The drop-in solver passes on what the tuner says for its size, at every size."""
    from boltzmann_gb300 import _lib
    from boltzmann_gb300.bte_0d3v_batched import bte_0d3v_batched
    monkeypatch.setattr(autotune, "tune_lu", lambda N, device=0: {"kernel": 4})
    s = types.SimpleNamespace(_args=types.SimpleNamespace(), _precision=lambda: _lib.PREC_MIXED, _dev_id=0,
                              _grid_info=[{"n": 384}, {"n": 768}])
    assert bte_0d3v_batched._lu_kernel(s, 0) == 4 and bte_0d3v_batched._lu_kernel(s, 1) == 0
