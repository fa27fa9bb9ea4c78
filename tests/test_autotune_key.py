"""Keys of the autotuner's cache: an entry of other kernels or candidates is not
taken, and batches that run another form of the kernel, or other fields, have keys
of their own."""
import json

import pytest

from chromo_gb300 import autotune as at
from chromo_gb300.batched import ReplicaBatch
from golden_cases import load
from test_gpu_api import _setup


class _Timed(Exception):
    pass


def _build(w, g):
    raise _Timed


def test_entry_of_other_kernels_is_timed_again(tmp_path, monkeypatch):
    monkeypatch.setenv("CHROMO_GB300_TUNE_CACHE", str(tmp_path / "tune.json"))
    lengths, grids = [3000] * 4, [[16, 16, 16]] * 4
    monkeypatch.setattr(at, "kernel_version", lambda: "other kernels")
    key = at.problem_key(lengths, grids, 2, False, 152, "fake")
    old = {k: v for k, v in json.loads(key).items() if k != "kernels"}  # a key without kernels
    (tmp_path / "tune.json").write_text(json.dumps({
        k: {"shape": [5, 16], "table": {"5x16": 1.0}} for k in (key, json.dumps(old, sort_keys=True))}))
    assert at.tune(_build, lengths, grids, 2, device=("fake", 152))[0] == (5, 16)
    monkeypatch.undo()
    monkeypatch.setenv("CHROMO_GB300_TUNE_CACHE", str(tmp_path / "tune.json"))
    assert at.kernel_version() == at.kernel_version() != "other kernels"
    with pytest.raises(_Timed):
        at.tune(_build, lengths, grids, 2, device=("fake", 152), shapes=[(1, 32)])


def test_batches_of_other_forms_have_other_keys(monkeypatch):
    keys = []

    def tune(make, n_beads, grids, nb, fp64, extra_key=""):
        keys.append(extra_key)
        raise _Timed

    monkeypatch.setattr(at, "tune", tune)
    for case in ("one_binder", "twist", "fast_field", "sphere_access", "null_spherical"):
        p, _, f, c = _setup(load(case))
        with pytest.raises(_Timed):
            ReplicaBatch([p], [f], [c], autotune=True)
    assert len(set(keys)) == 5, keys
