"""bench.py's count of the library's kernel launches (CPU, a fake profiler)."""
import types

import pytest
import torch

import bench


@pytest.mark.parametrize("recorded,count", [([], None), (["gbv::render_kernel", "gbv::finish_kernel", "other"], 2)])
def test_launches_are_counted_or_unknown(monkeypatch, recorded, count):
    events = [types.SimpleNamespace(device_type=torch.autograd.DeviceType.CUDA, name=n) for n in recorded]

    class Profile:
        def __init__(self, **kw):
            pass

        def __enter__(self):
            return self

        def __exit__(self, *a):
            return False

        def events(self):
            return events

    calls = []
    monkeypatch.setattr("torch.profiler.profile", Profile)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    assert bench.own_launches(lambda: calls.append(1)) == count
    assert calls
