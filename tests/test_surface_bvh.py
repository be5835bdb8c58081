"""The surface BVH of the closest-hit walk, checked on the host: the builder
(csrc/bvh_build.cu) is compiled with the host compiler together with
tests/surface_bvh.cpp.  Its boxes bound the leaves' surfaces instead of their
bounding spheres, so beside the tree's own consistency the walk must reach
the leaf that the oracle -- which searches the frame tree as merlict does --
finds for a ray, on every primitive, from near and far, and along surfaces."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import REPO, golden_names, load_golden
from merlict_development_kit_b200 import photons as P

CSRC = os.path.join(REPO, "merlict_development_kit_b200", "csrc")
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    out = str(tmp_path_factory.mktemp("surface_bvh") / "surface_bvh.so")
    cmd = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC,
           "-I", os.path.join(REPO, "include"), "-I", CUDA_INCLUDE,
           "-x", "c++", os.path.join(REPO, "tests", "surface_bvh.cpp"),
           "-x", "c++", os.path.join(CSRC, "bvh_build.cu"), "-o", out]
    subprocess.run(cmd, check=True, capture_output=True)
    lib = C.CDLL(out)
    lib.surface_bvh_invariants.restype = C.c_int64
    lib.surface_bvh_misses.restype = C.c_int64
    return lib


def consistent(lib, flat):
    s = flat.as_struct()
    info = (C.c_int64 * 3)()
    assert lib.surface_bvh_invariants(C.byref(s), info) == 0
    with_geometry = int(np.count_nonzero(np.asarray(flat.leaf_primitive) != 0))
    assert info[1] == with_geometry
    return list(info)


def reaches_every_hit(lib, oracle, flat, ph):
    """The first hit of every photon, by the oracle, is reached by the walk."""
    status, ref, _ = oracle.propagate(flat, ph, 1, seed=3)
    assert status == 0
    sup = np.stack([ph[f"support_{k}"] for k in "xyz"], axis=1).astype(np.float64)
    d = np.stack([ph[f"direction_{k}"] for k in "xyz"], axis=1).astype(np.float64)
    d /= np.sqrt((d * d).sum(axis=1))[:, None]
    sup, d = np.ascontiguousarray(sup), np.ascontiguousarray(d)
    leaf = np.ascontiguousarray(ref["final_leaf"], dtype=np.int32)
    s = flat.as_struct()
    visits = C.c_int64(0)
    missed = lib.surface_bvh_misses(C.byref(s), C.c_int64(len(leaf)), C.c_void_p(sup.ctypes.data),
                                    C.c_void_p(d.ctypes.data), C.c_void_p(leaf.ctypes.data),
                                    C.byref(visits))
    assert missed == 0
    return int((leaf >= 0).sum())


def chords(n, seed, centre, radius, distance):
    """Rays from `distance` away towards points of a ball about `centre`, a
    third of them nearly in the horizontal plane (grazing flat surfaces)."""
    rng = np.random.default_rng(seed)
    v = rng.normal(size=(n, 3))
    v[::3, 2] *= 1e-3
    v /= np.linalg.norm(v, axis=1)[:, None]
    aim = centre + radius * rng.uniform(-1, 1, size=(n, 3))
    return P.make_batch(aim - v * distance * rng.uniform(0.0, 1.0, size=(n, 1)), v,
                        np.full(n, 433e-9))


@pytest.mark.parametrize("name", golden_names())
def test_every_golden_scene(checker, oracle, name):
    flat, photons, _, _ = load_golden(name)
    consistent(checker, flat)
    if len(photons["wavelength"]):
        reaches_every_hit(checker, oracle, flat, photons)
    root = np.asarray(flat.node_sphere).reshape(-1, 4)[0]
    leaves = np.asarray(flat.node_sphere).reshape(-1, 4)[np.asarray(flat.leaf_node)]
    rng = np.random.default_rng(5)
    hits = 0
    for k, distance in enumerate((2.0 * root[3], 1e3, 1e4)):
        hits += reaches_every_hit(checker, oracle, flat,
                                  chords(3000, k, root[:3], root[3], distance))
        for leaf in rng.choice(len(leaves), size=min(8, len(leaves)), replace=False):
            hits += reaches_every_hit(
                checker, oracle, flat,
                chords(500, 7 + k, leaves[leaf, :3], leaves[leaf, 3], distance))
    assert hits > 100


def test_the_light_field_telescope(checker, oracle):
    from merlict_development_kit_b200 import factories as F
    flat = F.light_field_telescope().flatten()
    nodes, leaves, levels = consistent(checker, flat)
    assert leaves == 78378 and levels <= 12
    assert reaches_every_hit(checker, oracle, flat,
                             P.downward_disc_source(5000, 3, 5.55, 21.4, 1.5)) > 3000
    # towards the sensor from the dish and from just above it
    assert reaches_every_hit(checker, oracle, flat,
                             chords(5000, 4, np.array([0.0, 0.0, 10.7]), 0.5, 10.0)) > 1000
    assert reaches_every_hit(checker, oracle, flat,
                             chords(5000, 5, np.array([0.0, 0.0, 10.71]), 0.3, 0.05)) > 1000


def test_the_large_reflector(checker, oracle):
    from merlict_development_kit_b200 import factories as F
    flat = F.large_reflector_camera().flatten()
    consistent(checker, flat)
    assert reaches_every_hit(checker, oracle, flat,
                             P.downward_disc_source(5000, 6, 40.0, 110.0, 3.5)) > 2000


def test_degenerate_surfaces_keep_their_spheres(checker):
    """A sliver triangle and bounds that are not finite: the box is the
    bounding sphere's, so every ray through the sphere reaches the leaf."""
    flat, _, _, _ = load_golden("primitive_zoo")
    prim = np.asarray(flat.leaf_primitive)
    params = np.asarray(flat.leaf_params).reshape(len(prim), -1)
    for l in np.flatnonzero(prim == 10):
        params[l, :6] = [0.0, 0.0, 1.0, 0.0, 2.0, 1e-9]
    for l in np.flatnonzero(prim == 5):
        params[l, 0] = np.nan
    flat.leaf_params = params.reshape(np.asarray(flat.leaf_params).shape)
    consistent(checker, flat)
    leaf_node = np.asarray(flat.leaf_node)
    sphere = np.asarray(flat.node_sphere).reshape(-1, 4)
    s = flat.as_struct()
    rng = np.random.default_rng(9)
    checked = 0
    for l in np.flatnonzero((prim == 10) | (prim == 5)):
        c = sphere[leaf_node[l]]
        v = rng.normal(size=(200, 3))
        v /= np.linalg.norm(v, axis=1)[:, None]
        off = rng.normal(size=(200, 3))
        off -= (off * v).sum(axis=1)[:, None] * v
        off *= (0.999 * c[3] * rng.random(200) / np.linalg.norm(off, axis=1))[:, None]
        sup = np.ascontiguousarray(c[:3] + off - 5.0 * c[3] * v)
        d = np.ascontiguousarray(v)
        leaf = np.full(200, l, np.int32)
        visits = C.c_int64(0)
        assert checker.surface_bvh_misses(
            C.byref(s), C.c_int64(200), C.c_void_p(sup.ctypes.data), C.c_void_p(d.ctypes.data),
            C.c_void_p(leaf.ctypes.data), C.byref(visits)) == 0
        checked += 1
    assert checked >= 1


def wide_scene(radius):
    """A ground disc of `radius` under a few small surfaces."""
    from merlict_development_kit_b200 import scenery as S
    sc = S.Scenery()
    sc.root.add(S.Disc("ground", (0.0, 0.0, -2.0), S.ROT3_UNITY)).set_radius(radius)
    for i in range(20):
        d = sc.root.add(S.Disc(f"d{i}", (3.0*i, -2.0*i, 0.1*i), S.Rot3(0.02*i, -0.01*i, 0.0)))
        d.set_radius(0.5)
        s = sc.root.add(S.Sphere(f"s{i}", (-3.0*i - 1.5, 2.0*i, 5.0), S.ROT3_UNITY))
        s.set_radius(0.7)
    sc.init()
    return sc.flatten()


def along_the_axes(n, seed):
    """Rays with one or two components that are exactly zero."""
    rng = np.random.default_rng(seed)
    d = np.zeros((n, 3))
    d[:, 2] = -1.0
    d[1::4] = [0.0, 0.6, -0.8]
    d[2::4] = [-1.0, -0.0, 0.0]
    d[3::4, 0] = 1e-25
    sup = rng.uniform(-60.0, 60.0, size=(n, 3))
    sup[:, 2] = rng.uniform(0.0, 30.0, n)
    return P.make_batch(sup, d, np.full(n, 433e-9))


@pytest.mark.parametrize("radius", [1e2, 1e6, 2e6, 3e6, 1e7, 1e9, 1e13])
def test_wide_sceneries_and_rays_along_the_axes(checker, oracle, radius):
    flat = wide_scene(radius)
    assert consistent(checker, flat)[2] >= 1
    assert reaches_every_hit(checker, oracle, flat, along_the_axes(2000, 3)) > 1000


def test_no_surface_tree_beyond_the_largest_extent(checker):
    flat = wide_scene(1e17)
    s = flat.as_struct()
    info = (C.c_int64 * 3)()
    assert checker.surface_bvh_invariants(C.byref(s), info) == 0
    assert list(info) == [0, 0, 0]
