"""The tuner can choose the default that it replaces, and times every candidate over
the same steps."""
import types

import pytest
import torch

from biomedisa_gb300 import _native as nat
from biomedisa_gb300 import autotune as A


@pytest.mark.parametrize("sorw", [20, 300, 999, 1000, 4000])
def test_probes(sorw, monkeypatch):
    walked, clock = [], [0.0]

    def call(name, *args):
        if name == "si_walk_sorted_batch":
            walked.append((args[6], args[5], args[3]))  # edge, sweep, probe steps
            clock[0] += 1.0 if args[5] == 128 else 2.0

    class Event:
        def __init__(self, **_):
            pass

        def record(self, _):
            self.at = clock[0]

        def elapsed_time(self, other):
            return other.at - self.at

    monkeypatch.setattr(nat, "call", call)
    monkeypatch.setattr(A, "_store", lambda *_: None)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda: "test")
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=0))
    monkeypatch.setattr(torch, "empty", lambda *a, **_: types.SimpleNamespace(data_ptr=lambda: 0))
    vol = types.SimpleNamespace(work_is_float=0, Zc=5, Yc=6, Xc=7)
    edge, steps, rep = A.tune([vol], 1, [], 2, sorw, 0, 100, use_cache=False)
    assert (6, 128 if sorw >= 1000 else 32) in [w[:2] for w in walked]
    assert {w[2] for w in walked} == {min(sorw, A.PROBE_STEPS)}
    assert (edge, steps) == (6, 128) and len(rep["candidates"]) == len(walked)


@pytest.mark.gpu
@pytest.mark.parametrize("sorw", [200, 999, 1000])
def test_default_is_a_candidate(sorw, cuda):
    """The sweeps that the library takes by itself are the first candidate's."""
    import numpy as np

    from biomedisa_gb300 import smart_interpolation_batch
    lab = np.zeros((9, 12, 14), np.int32)
    lab[::3, :, 7:] = 1
    rep = {}
    smart_interpolation_batch([lab.astype(np.uint8) * 90], [lab], nbrw=1, sorw=sorw, autotune_params=False, report=rep)
    assert rep["sweeps"] == -(-sorw // A.candidates(sorw)[0][1])
