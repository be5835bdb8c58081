"""The closest-hit walk (csrc/closest_hit.cuh) at the sizes where its warps
can go wrong -- fewer rays than a warp, a lane more than a chunk, pools that
are refilled many times -- against the oracle, bit for bit, with photons
that are not finite among the others."""
import numpy as np
import pytest

from conftest import load_golden
from merlict_development_kit_b200 import photons as P
from parity import mismatches

pytestmark = pytest.mark.gpu


def batch(name, n):
    if name == "sparse":      # most miss the telescope: ended by the first look
        return P.downward_disc_source(n, 11, 60.0, 21.4, 0.5)
    if name == "light_field_small":
        return P.downward_disc_source(n, 11, 5.55, 21.4, 0.5)
    return P.isotropic_shell_source(n, 11, 4.0, 2.5)


@pytest.mark.parametrize("name", ["primitive_zoo", "light_field_small"])
@pytest.mark.parametrize("n,pool", [(1, 0), (31, 0), (33, 0), (129, 0), (2049, 1024), (40_001, 1024),
                                    (70_003, 0), (70_003, 4096)])
def test_any_number_of_rays(oracle, name, n, pool):
    check(oracle, name, batch(name, n), pool)


@pytest.mark.parametrize("n,pool,order", [(100_003, 0, 0), (100_003, 1024, 0), (100_003, 0, 2)])
def test_a_sparse_batch(oracle, n, pool, order):
    check(oracle, "light_field_small", batch("sparse", n), pool, order)


def check(oracle, name, ph, pool, order=0):
    from merlict_development_kit_b200 import engine
    flat, _, _, meta = load_golden(name)
    n = len(ph["wavelength"])
    if n > 100:
        ph["direction_x"][7] = np.nan
        ph["support_z"][n - 1] = np.inf
        ph["support_x"][n // 2] = 1e30
    status, ref, _ = oracle.propagate(flat, ph, meta["max_interactions"], seed=5)
    assert status == 0
    scene = engine.Scene(flat)
    out = scene.propagate(engine.photons_to_device(ph),
                          engine.PropagationConfig(meta["max_interactions"]), engine.Philox(5),
                          outputs=("sensor", "x", "y", "time", "theta_x", "theta_y", "final_leaf",
                                   "info", "final_position", "final_direction"),
                          tuning={"pool_size": pool, "walk": 2, "photon_order": order})
    got = {k: v.cpu().numpy() for k, v in out.items()}
    assert mismatches(ref, got) == {}
    scene.close()


@pytest.mark.parametrize("radius", [1e2, 3e6, 1e9, 1e17])
@pytest.mark.parametrize("n", [2000, 70_003])
def test_wide_sceneries_and_rays_along_the_axes(oracle, radius, n):
    """Steps of a node's bounds over a direction component of zero stay finite;
    beyond the largest extent the level kernels take over."""
    from merlict_development_kit_b200 import engine
    from test_surface_bvh import along_the_axes, wide_scene
    flat = wide_scene(radius)
    ph = along_the_axes(n, 4)
    status, ref, _ = oracle.propagate(flat, ph, 3, seed=5)
    assert status == 0
    scene = engine.Scene(flat)
    out = scene.propagate(engine.photons_to_device(ph), engine.PropagationConfig(3),
                          engine.Philox(5), outputs=("sensor", "final_leaf", "info", "time",
                                                     "final_position", "final_direction"))
    got = {k: v.cpu().numpy() for k, v in out.items()}
    assert (ref["final_leaf"] >= 0).sum() > 0.5*n
    assert mismatches(ref, got) == {}
    scene.close()


@pytest.mark.parametrize("n,sparse,plain", [(20_011, False, 1),    # one launch for the batch
                                            (100_003, True, 2),    # first look, the listed ones
                                            (300_001, False, 3)])  # and the pool's last rays
def test_every_kernel_of_a_call_is_in_a_class(n, sparse, plain):
    """Launches counted are launches timed, but for the copies of the counters
    to the host, one before each of the host's looks."""
    from merlict_development_kit_b200 import engine
    flat, _, _, meta = load_golden("light_field_small")
    scene = engine.Scene(flat)
    ph = engine.photons_to_device(batch("sparse" if sparse else "light_field_small", n))
    config = engine.PropagationConfig(meta["max_interactions"])
    scene.propagate(ph, config)
    scene.set_profiling(True)
    before = scene.kernel_launches(), scene.wavefront_stats()["iterations"]
    scene.propagate(ph, config)
    launches = scene.kernel_launches() - before[0]
    iterations = scene.wavefront_stats()["iterations"] - before[1]
    times = scene.kernel_times()
    scene.set_profiling(False)
    timed = {k: count for k, (ms, count) in times.items() if count}
    assert timed["plain"] == plain and times["plain"][0] > 0.0
    if plain < 3:
        assert set(timed) == {"plain"} and launches == plain + (plain > 1)
    else:
        assert timed["walk"] == timed["resolve"] == iterations
        # looks: behind the first look, the first iteration, every second one
        assert launches == sum(timed.values()) + 2 + iterations//2
    scene.close()


@pytest.mark.parametrize("walk", [0, 1])
@pytest.mark.parametrize("tracer", ["fp64", "fp32"])
def test_rays_along_the_axes_far_from_the_origin(oracle, walk, tracer):
    """Boxes and rays more than 3.4e8 m from the scenery's origin, where a
    distance over the smallest direction component must stay finite as well."""
    from merlict_development_kit_b200 import engine, scenery as S
    sc = S.Scenery()
    at = 2.0**31
    for i in range(12):
        pos = (at*(i % 3 - 1), -at*(i % 2), at*(i // 6))
        sc.root.add(S.Sphere(f"s{i}", pos, S.ROT3_UNITY)).set_radius(1024.0)
    sc.init()
    flat = sc.flatten()
    centre = np.asarray(flat.node_sphere).reshape(-1, 4)[np.asarray(flat.leaf_node), :3]
    n = 1200
    rng = np.random.default_rng(2)
    d = np.eye(3)[np.arange(n) % 3]*rng.choice([-1.0, 1.0], size=(n, 1))
    off = np.round(rng.uniform(-512.0, 512.0, size=(n, 3)))*(1.0 - np.abs(d))
    ph = P.make_batch(centre[np.arange(n) % 12] + off - 65536.0*d, d, np.full(n, 433e-9))
    status, ref, _ = oracle.propagate(flat, ph, 1, seed=5)
    assert status == 0 and (ref["final_leaf"] >= 0).all()
    scene = engine.Scene(flat)
    out = scene.propagate(engine.photons_to_device(ph), engine.PropagationConfig(1), engine.Philox(5),
                          outputs=("sensor", "final_leaf"), tracer=tracer, tuning={"walk": walk})
    assert np.array_equal(out["final_leaf"].cpu().numpy(), ref["final_leaf"])
    scene.close()
