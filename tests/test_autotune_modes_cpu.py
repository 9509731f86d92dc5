"""Which launches a tuned shape is taken for (host logic; plans and events are stand-ins)."""
import types

import pytest
import torch

from discoeb_gb300 import _native, autotune
from discoeb_gb300 import perturbations as pt

SMS = 152
# ms per (modes, modes per SM): few modes end on their longest, many share the SMs' FP64 units
MS = {256: {0: 156.0, 2: 155.0, 1: 146.0}, 4096: {0: 578.0, 2: 685.0, 1: 1051.0}}


def _dims():
    return _native.DebDims(12, 12, 17, 17, 15, 1, 0, 0, 0)


class _Plan:
    def __init__(self, dims, max_modes, launch=None, **kw):
        self.max_modes, self.launch = max_modes, launch

    def launch_info(self):
        return dict(stage_vectors=self.launch[0], modes_per_sm=self.launch[1], modes_in_flight=1)


class _Event:
    now = 0.0

    def __init__(self, enable_timing=True):
        self.t = None

    def record(self, s=None):
        self.t = _Event.now

    def elapsed_time(self, other):
        return other.t - self.t


@pytest.fixture
def stand_ins(monkeypatch):
    monkeypatch.delenv("DISCOEB_GB300_TUNE_CACHE", raising=False)
    monkeypatch.setattr(autotune, "_chosen", {})
    monkeypatch.setattr(autotune, "_loaded", False)
    monkeypatch.setattr(pt, "_plans", {})
    monkeypatch.setattr(_native, "Plan", _Plan)
    monkeypatch.setattr(pt, "_torch", lambda: torch)
    for name, v in dict(current_device=lambda: 0, get_device_name=lambda d: "GB300", Event=_Event,
                        synchronize=lambda: None, current_stream=lambda: None,
                        get_device_properties=lambda d: types.SimpleNamespace(multi_processor_count=SMS)).items():
        monkeypatch.setattr(torch.cuda, name, v)


def _tune(nmode):
    def launch(plan, s):
        _Event.now += MS[nmode][plan.launch[1]] + (0.0 if plan.launch[0] == "shared" else 1.0)

    return autotune.tune(_dims(), nmode, launch)[0]


def test_a_shape_tuned_on_few_modes_is_not_taken_for_many(stand_ins):
    assert _tune(256) == ("shared", 1)
    assert pt.get_plan(_dims(), 256).launch == ("shared", 1)
    assert pt.get_plan(_dims(), 4096).launch is None          # the library's default until tuned there
    assert _tune(4096) == ("shared", 0)
    assert pt.get_plan(_dims(), 4096).launch == ("shared", 0)
    assert pt.get_plan(_dims(), 256).launch == ("shared", 1)
    assert autotune.chosen(_dims()) == ("shared", 0)          # the latest choice


def test_choices_written_for_another_kernel_are_not_taken(stand_ins, tmp_path, monkeypatch):
    path = tmp_path / "tune.json"
    path.write_text('{"GB300|12|12|17|17|15|1|0|0": ["global", 6]}')
    monkeypatch.setenv("DISCOEB_GB300_TUNE_CACHE", str(path))
    assert pt.get_plan(_dims(), 256).launch is None


def test_a_shape_remembered_for_any_number_of_modes(stand_ins):
    autotune.remember(_dims(), ("global", 0))
    assert pt.get_plan(_dims(), 256).launch == ("global", 0) == pt.get_plan(_dims(), 4096).launch
    _tune(256)
    assert pt.get_plan(_dims(), 256).launch == ("shared", 1)
    assert pt.get_plan(_dims(), 4096).launch == ("global", 0)
