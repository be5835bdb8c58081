"""The order of calls on one scene from several streams, checked on the host:
csrc/in_flight.h is compiled with the host compiler against a model of
streams and events (tests/in_flight.cpp)."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

from conftest import REPO

CSRC = os.path.join(REPO, "merlict_development_kit_b200", "csrc")
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    out = str(tmp_path_factory.mktemp("in_flight") / "in_flight.so")
    # its own definitions of the runtime's calls, whatever else the process holds
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC,
                    "-I", CUDA_INCLUDE, os.path.join(REPO, "tests", "in_flight.cpp"), "-o", out],
                   check=True, capture_output=True)
    lib = C.CDLL(out)
    for f in (lib.in_flight_violations, lib.in_flight_order_among_small, lib.in_flight_capture):
        f.restype = C.c_int64
    return lib


@pytest.mark.parametrize("streams", [1, 2, 8, 9, 20])
def test_scratch_is_written_after_every_earlier_call(model, streams):
    for seed in range(20):
        assert model.in_flight_violations(streams, 400, seed) == 0


def test_small_calls_on_several_streams_run_side_by_side(model):
    assert model.in_flight_order_among_small() == 0


def test_captured_work_is_left_alone(model):
    assert model.in_flight_capture() == 0
