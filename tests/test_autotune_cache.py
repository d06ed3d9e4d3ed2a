"""A choice that the tuner of the batched solver stored is taken up only by the kernel and the candidates that it was
timed with (CPU: the timing is a stand-in)."""
import json
import types

import numpy as np
import pytest


@pytest.fixture
def tuner(monkeypatch, tmp_path):
    torch = pytest.importorskip("torch")
    from ttg_gb300 import autotune
    monkeypatch.setattr(autotune, "_CACHE", str(tmp_path / "cache.json"))
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a: "GPU")
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda *a: types.SimpleNamespace(multi_processor_count=10))
    monkeypatch.setattr(autotune, "_time", lambda batch, mode, refine, ctas, reps: batch.timed.append(ctas) or float(ctas))
    monkeypatch.setattr(autotune, "_berr", lambda *a: 0.0)
    return autotune


class _Batch:
    def __init__(self):
        import torch
        self.sizes, self.nrhs, self.batch = np.array([3, 2], dtype=np.int32), 1, 2
        self.A0, self.info, self.timed = torch.zeros(13, dtype=torch.float64), torch.zeros(2, dtype=torch.int32), []

    def set_order(self, order):
        self.order = order


def test_entry_of_an_earlier_kernel_is_not_used(tuner):
    import torch  # noqa: F401
    import hashlib
    b = _Batch()
    h = hashlib.sha1(np.bincount(b.sizes, minlength=1).tobytes()).hexdigest()[:16]
    stale = {"mode": "fp64", "refine": 0, "schedule": "lpt", "ctas": 12345, "ms": 0.0}
    json.dump({"GPU|%s|1|1e-14" % h: stale}, open(tuner._CACHE, "w"))
    best = tuner.tune_batched(b, [])
    assert best["ctas"] != 12345 and b.timed
    b.timed.clear()
    assert tuner.tune_batched(b, [])["ctas"] == best["ctas"] and not b.timed  # its own entry is


def test_entry_goes_with_kernel_and_candidates(tuner, monkeypatch):
    key = tuner._key(_Batch(), 1e-14)
    monkeypatch.setattr(tuner, "_KERNEL", tuner._KERNEL + 1)
    other = tuner._key(_Batch(), 1e-14)
    monkeypatch.setattr(tuner, "_CTAS_PER_SM", (2, 4))
    assert len({key, other, tuner._key(_Batch(), 1e-14)}) == 3
