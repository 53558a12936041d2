"""Stored tuning choices are those of the kernels in use: an entry stored before the kernels changed is not
applied, nor one of a plan whose sizes take other paths (no GPU: a stand-in plan and library)."""
import json
from types import SimpleNamespace

import torch

from aero2d_b200 import _lib, autotune


class FakePlan:
    device = None
    shapes = [(256, 64)] * 16
    params = SimpleNamespace(precision=1)

    def __init__(self, *paths):
        self.config, self.taken = autotune.DEFAULT, set(paths)

    def paths(self):
        return self.taken

    def set_tuning(self, t, v):
        self.config = (t, v)

    def tuning(self):
        return self.config

    def init_freestream(self):
        pass


def stand_ins(monkeypatch):
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device: "GPU")
    monkeypatch.setattr(_lib, "load", lambda: SimpleNamespace(a2d_version=lambda: 100))


def test_a_choice_of_older_kernels_is_not_applied(tmp_path, monkeypatch):
    stand_ins(monkeypatch)
    path = tmp_path / "tuning.json"
    old = {"jvp_tile": "64x4", "sweep": "rows"}
    path.write_text(json.dumps({"GPU|lib100|mixed|256x64:16": old, "GPU|lib100.1|mixed|256x64:16": old}))
    cache = autotune.TuningCache(path)
    for plan in (FakePlan(), FakePlan("lines")):
        assert autotune.apply(plan, cache=cache) == autotune.DEFAULT
    fresh = FakePlan("lines")
    choice = autotune.apply(fresh, measure=True, cache=cache, measure_fn=lambda p: 1.0 + (p.config != ("32x8", "pairs")))
    assert choice == ("32x8", "pairs")
    assert autotune.apply(FakePlan("lines"), cache=cache) == choice       # and is found again


def test_a_choice_stays_on_its_side_of_a_limit(tmp_path, monkeypatch):
    """10 and 16 cases share a signature; which kernels they run need not be the same."""
    stand_ins(monkeypatch)
    cache = autotune.TuningCache(tmp_path / "tuning.json")
    a, b = FakePlan("lines", "fine_tiles", "arnoldi"), FakePlan("sweeps", "smooth")
    cache.put(autotune.plan_key(a), ("16x16", "rows"))
    assert autotune.apply(b, cache=cache) == autotune.DEFAULT
    assert autotune.apply(FakePlan("fine_tiles", "lines"), cache=cache) == ("16x16", "rows")   # the knobs' paths only
