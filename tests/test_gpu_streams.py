"""One scene used from several streams: a call returns while its last kernels
still use the scene's scratch (csrc/in_flight.h), and the next call, on
whatever stream, comes after them.  Every result is compared bit for bit
with the same calls one by one."""
import numpy as np
import pytest

from conftest import load_golden
from merlict_development_kit_b200 import abi, photons as P

pytestmark = pytest.mark.gpu

OUT = ("sensor", "x", "y", "time", "final_leaf", "info")


@pytest.fixture(scope="module")
def telescope():
    from merlict_development_kit_b200 import engine
    flat, _, _, meta = load_golden("light_field_small")
    scene = engine.Scene(flat)
    yield scene, meta["max_interactions"]
    scene.close()


def equal(a, b):
    import torch
    return all(torch.equal(a[k].view(torch.uint8), b[k].view(torch.uint8)) for k in OUT)


@pytest.mark.parametrize("tracer,n", [("fp64", 300_001), ("fp64_queue", 100_003), ("fp32", 300_001),
                                      ("fp64", 20_011)])
def test_two_batches_on_two_streams(telescope, tracer, n):
    """More photons than one launch takes, so the pools are used: the second
    call clears and refills them while the first one's last rays are traced."""
    import torch
    from merlict_development_kit_b200 import engine
    scene, depth = telescope
    config = engine.PropagationConfig(depth)
    batches = [engine.photons_to_device(P.downward_disc_source(n + k, 5 + k, 5.55, 21.4, 0.5))
               for k in range(4)]
    kw = dict(outputs=OUT, tracer=tracer)
    one_by_one = [scene.propagate(b, config, engine.Philox(k), **kw) for k, b in enumerate(batches)]
    streams = [torch.cuda.default_stream(), torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(3):
        got = [scene.propagate(b, config, engine.Philox(k), stream=streams[k % 3], sync=False, **kw)
               for k, b in enumerate(batches)]
        torch.cuda.synchronize()
        assert [equal(a, b) for a, b in zip(one_by_one, got)] == [True]*4


def test_a_host_call_behind_a_stream(telescope):
    """The host-buffer call runs on streams of its own."""
    import ctypes as C
    import torch
    from merlict_development_kit_b200 import engine
    from merlict_development_kit_b200._native import check, lib
    scene, depth = telescope
    n = 2_200_000
    config = engine.PropagationConfig(depth)
    first = engine.photons_to_device(P.downward_disc_source(300_001, 1, 5.55, 21.4, 0.5))
    batch = P.downward_disc_source(n, 2, 5.55, 21.4, 0.5)
    kw = dict(outputs=OUT)
    want_first = scene.propagate(first, config, engine.Philox(1), **kw)
    dev = engine.photons_to_device(batch)
    want = scene.propagate(dev, config, engine.Philox(2), outputs=("sensor", "time"))
    host = {k: torch.from_numpy(np.ascontiguousarray(batch[k], np.float64)).pin_memory()
            for k in P.PLANES}
    sensor = torch.empty(n, dtype=torch.int32).pin_memory()
    time = torch.empty(n, dtype=torch.float64).pin_memory()
    ph = abi.mlgpu_photons()
    ph.dtype = abi.F64
    for k in P.PLANES:
        setattr(ph, k, host[k].data_ptr())
    res = abi.mlgpu_results()
    res.dtype = abi.F64
    res.sensor, res.time = sensor.data_ptr(), time.data_ptr()
    st = engine._settings(config, 0, "fp64", "bvh", None)
    r, _ = engine.Philox(2)._struct(n)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    got_first = scene.propagate(first, config, engine.Philox(1), stream=stream, sync=False, **kw)
    check(lib().mlgpu_propagate_host(scene.handle, C.byref(ph), n, C.byref(st), C.byref(r),
                                     C.byref(res)))
    torch.cuda.synchronize()
    assert equal(want_first, got_first)
    assert torch.equal(sensor, want["sensor"].cpu())
    assert torch.equal(time.view(torch.int64), want["time"].cpu().view(torch.int64))


def test_a_calls_tensors_outlive_it(telescope):
    """What a call on another stream reads or writes stays its own until that
    stream has passed it, although the caller lets go of it at once."""
    import torch
    from merlict_development_kit_b200 import engine
    scene, depth = telescope
    n = 20_011
    config = engine.PropagationConfig(depth)
    table = np.random.default_rng(3).random((n, 64))
    batch = P.downward_disc_source(n, 9, 5.55, 21.4, 0.5)
    want = scene.propagate(engine.photons_to_device(batch), config, engine.Replay(table), outputs=OUT)
    stream = torch.cuda.Stream()
    for _ in range(3):
        photons = engine.photons_to_device(batch)
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)      # some 10 ms in front of the call
        got = scene.propagate(photons, config, engine.Replay(table), outputs=OUT, stream=stream,
                              sync=False)
        dropped = scene.propagate(photons, config, engine.Philox(1), outputs=OUT, stream=stream,
                                  sync=False)
        sizes = [t.shape for t in photons.values()] + [t.shape for t in dropped.values()]
        del photons, dropped
        filled = [torch.full(s, 7.0, dtype=torch.float64, device="cuda") for s in sizes]
        filled += [torch.full(table.shape, 7.0, dtype=torch.float64, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        assert equal(want, got)
        assert all(bool((t == 7.0).all()) for t in filled)
        del filled


@pytest.mark.parametrize("n", [300, 300_001])
def test_errors_of_a_call_on_another_stream(n):
    """sync_errors reports what earlier propagations raised, whichever stream
    they were on, also when they are still waiting for their turn there."""
    import torch
    from merlict_development_kit_b200 import engine
    flat, _, _, meta = load_golden("mirror_absorber")
    scene = engine.Scene(flat)
    config = engine.PropagationConfig(5)
    good = engine.photons_to_device(P.isotropic_shell_source(n, 1, 4.0, 2.5))
    bad = {k: v.clone() for k, v in good.items()}
    bad["wavelength"][:] = 1500e-9
    stream = torch.cuda.Stream()
    for _ in range(2):
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)
        scene.propagate(bad, config, engine.Philox(1), stream=stream, sync=False)
        with pytest.raises(IndexError):
            scene.sync_errors()
        scene.sync_errors(stream=stream)        # reported once
        scene.propagate(good, config, engine.Philox(1))
    scene.close()


def test_bunches_on_two_streams(telescope):
    """The expansion reads counts of the scene's scratch, which the next call
    writes."""
    import torch
    from merlict_development_kit_b200 import engine
    from test_corsika import random_bunches
    scene, _ = telescope
    events = [torch.as_tensor(random_bunches(n, k)[0], device="cuda")
              for k, n in enumerate((400_003, 300_001, 400_009))]
    want = [scene.corsika_photons(b, engine.Philox(k)) for k, b in enumerate(events)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(3):
        got = [scene.corsika_photons(b, engine.Philox(k), stream=streams[k % 2])
               for k, b in enumerate(events)]
        torch.cuda.synchronize()
        for a, b in zip(want, got):
            assert all(torch.equal(a[k], b[k]) for k in (*P.PLANES, "id"))


def test_statistics_on_two_streams(telescope):
    import ctypes as C
    import torch
    from merlict_development_kit_b200._native import check, lib
    scene, _ = telescope
    ns = scene.num_sensors
    sets = []
    for k, n in enumerate((2_000_003, 1_000_001)):
        g = torch.Generator(device="cuda").manual_seed(k)
        sensor = torch.randint(-1, ns, (n,), dtype=torch.int32, device="cuda", generator=g)
        values = [torch.randn(n, dtype=torch.float32, device="cuda", generator=g) for _ in range(5)]
        sets.append((n, sensor, values))

    def call(k, stream):
        n, sensor, values = sets[k]
        out = torch.empty((ns, 12), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        return out, lambda: check(lib().mlgpu_lixel_statistics(
            scene.handle, C.c_void_p(sensor.data_ptr()),
            *[C.c_void_p(v.data_ptr()) for v in values], n, n/ns, C.c_void_p(out.data_ptr()),
            C.c_void_p(stream.cuda_stream)))
    streams = [torch.cuda.Stream() for _ in range(2)]
    want = []
    for k in range(2):
        out, run = call(k, streams[0])
        run()
        torch.cuda.synchronize()
        want.append(out)
    for _ in range(3):
        calls = [call(k, streams[k]) for k in range(2)]
        for _, run in calls:
            run()
        torch.cuda.synchronize()
        assert all(torch.equal(a.view(torch.int32), c[0].view(torch.int32))
                   for a, c in zip(want, calls))


def test_a_small_batch_in_a_graph(telescope):
    """A batch of one launch can be captured; calls before, in and behind the
    capture give what they give without it."""
    import torch
    from merlict_development_kit_b200 import engine
    scene, depth = telescope
    config = engine.PropagationConfig(depth)
    small = engine.photons_to_device(P.downward_disc_source(2003, 3, 5.55, 21.4, 0.5))
    large = engine.photons_to_device(P.downward_disc_source(100_003, 4, 5.55, 21.4, 0.5))
    want_small = scene.propagate(small, config, engine.Philox(1), outputs=OUT)
    want_large = scene.propagate(large, config, engine.Philox(2), outputs=OUT)
    results = {k: torch.empty_like(v) for k, v in want_small.items()}
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    scene.propagate(large, config, engine.Philox(2), outputs=OUT, stream=other, sync=False)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        scene.propagate(small, config, engine.Philox(1), outputs=OUT, results=results, sync=False)
    for _ in range(2):
        for v in results.values():
            v.zero_()
        graph.replay()
        got = scene.propagate(large, config, engine.Philox(2), outputs=OUT, stream=other, sync=False)
        torch.cuda.synchronize()
        assert equal(want_small, results)
        assert equal(want_large, got)
