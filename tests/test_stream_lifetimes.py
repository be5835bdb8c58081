"""Tensors of a call on another stream than the current one (engine.py), with
stand-ins for the stream, the tensors and the library: the call starts after
what was made for it on the current stream, and everything its kernels use is
recorded as in use on its stream."""
import numpy as np
import pytest
import torch

from merlict_development_kit_b200 import engine
from merlict_development_kit_b200.photons import PLANES


class Stream:
    def __init__(self, handle, log):
        self.cuda_stream = handle
        self.log = log

    def wait_stream(self, other):
        self.log.append(("wait", self.cuda_stream, other.cuda_stream))


class Tensor:
    is_cuda = True
    device = "cpu"
    at = 64

    def __init__(self, shape, dtype, log, name):
        self.shape, self.dtype, self.log, self.name = shape, dtype, log, name
        Tensor.at += 64
        self.address = Tensor.at

    def is_contiguous(self):
        return True

    def data_ptr(self):
        return self.address

    def record_stream(self, s):
        self.log.append(("in use", self.name, s.cuda_stream))


@pytest.fixture
def world(monkeypatch):
    log = []
    current = Stream(1, log)
    monkeypatch.setattr(torch.cuda, "Stream", Stream)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: current)
    monkeypatch.setattr(torch, "empty", lambda shape, dtype, device: Tensor(shape, dtype, log, "made"))

    class Lib:
        def mlgpu_propagate(self, *a):
            log.append(("call", a[-1].value))
            return 0

        def mlgpu_scene_sync_errors(self, *a):
            return 0
    monkeypatch.setattr(engine, "lib", Lib)
    monkeypatch.setattr(engine, "check", lambda rc: None)
    scene = engine.Scene.__new__(engine.Scene)
    scene._h = None
    photons = {k: Tensor((4,), torch.float64, log, k) for k in PLANES}

    class Rng:
        uniforms = np.zeros((4, 8))          # copied to the device for the call

        def _struct(self, n):
            return engine.abi.mlgpu_rng(), Tensor((4, 8), torch.float64, log, "table")

        def advance(self, n):
            pass
    return log, current, scene, photons, Rng()


def test_on_another_stream(world):
    log, current, scene, photons, rng = world
    scene.propagate(photons, rng=rng, outputs=("sensor", "time"), stream=Stream(7, log), sync=False)
    assert log[:2] == [("wait", 7, 1), ("call", 7)]
    assert sorted(x[1] for x in log[2:]) == sorted([*PLANES, "table", "made", "made"])
    assert {x[2] for x in log[2:]} == {7}


def test_only_what_is_made_here_is_waited_for(world):
    log, current, scene, photons, _ = world
    results = {"sensor": Tensor((4,), torch.int32, log, "given")}
    scene.propagate(photons, outputs=("sensor",), results=results, stream=Stream(7, log), sync=False)
    assert log[0] == ("call", 7)
    assert ("in use", "given", 7) in log


def test_on_the_current_stream(world):
    log, current, scene, photons, rng = world
    scene.propagate(photons, rng=rng, stream=current)
    scene.propagate(photons, rng=rng)
    assert log == [("call", 1), ("call", 1)]
