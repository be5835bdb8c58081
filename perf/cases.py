"""The work a user of this framework has it do, as cases that can be timed and
compared: one photon event, batches of photons, the host-buffer call, and the
rows either side of the tracer (CORSIKA bunches, the signal chain, the
calibration, the learned surrogate).

Every case goes through the package's public entry points the way its own
benchmark and tests call them: one Scene per telescope (a user builds it once
and keeps it), the photons of a call already on the device (or in page-locked
host memory for the host-buffer call), default knobs.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from merlict_development_kit_b200 import (_native, abi, calibration, engine, factories,
                                          photons as P, signal_chain, surrogate)
from merlict_development_kit_b200.scenery import Func1

# the light-field telescope of the benchmark: 252 facets, 1,039 lenses,
# 63,379 lixels (78,378 surfaces)
TELESCOPE = dict(focal_length=10.7, aperture_radius=5.35, fov_deg=6.5, pixel_fov_deg=0.186,
                 paxels_on_diagonal=9, housing_overhead=1.1, reflectivity=0.9)
DISC = dict(disc_radius=5.55, height=21.4, max_zenith_deg=1.5)
FOUR = ("sensor", "x", "y", "time")
HISTORY_BYTES = 64
DRAWS = 1000        # key of the draws that decide how many photons or pulses come out
NET_FLOPS = 2.0 * (128 * 256 + 3 * 256 * 256 + 256 * 73)
NET_PARAMS = 128 * 256 + 256 + 3 * (256 * 256 + 256) + 256 * 73 + 73


def listed():
    return [
        # one small air-shower event, the reference's per-event loop: most
        # photons miss the telescope, latency is everything
        dict(name="event_300", kind="event", photons=300),
        # an ordinary event of the same loop
        dict(name="event_20k", kind="event", photons=20_011),
        # the largest single event, with its arrivals binned per lixel in time
        dict(name="event_1m_binned", kind="event", photons=999_983, time_bins=50),
        # the headline batch: parallel-ish light onto the dish, then counts per lixel
        dict(name="telescope_10m", kind="telescope", photons=10_000_000),
        # many uneven events concatenated into one call
        dict(name="showers_200", kind="showers", events=200),
        # the single-precision form on the large segmented reflector
        dict(name="reflector_fp32_8m", kind="reflector", photons=8_000_003, tracer="fp32"),
        # the call a host program makes: page-locked arrays in and out
        dict(name="host_4m", kind="host", photons=4_000_037),
        # everything after binning for one event: background, conversion, pulses
        dict(name="signal_1m", kind="signal", photons=1_000_000),
        # a plenoscope calibration at the size the reference's configuration sets
        dict(name="calibrate_8m", kind="calibrate", photons=8_000_000),
        # CORSIKA bunches of a large event expanded into photons
        dict(name="corsika_2m", kind="corsika", bunches=2_000_003),
        # the surrogate network applied to a batch, and one step of its training
        dict(name="surrogate_forward_1m", kind="forward", photons=1_000_003),
        dict(name="surrogate_train_64k", kind="train", photons=65_536),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["event", "event", "event", "telescope", "telescope", "showers", "reflector",
                       "camera", "host", "signal", "calibrate", "corsika", "forward", "train"])
    if kind == "event":
        n = _size(rng, 100, 1_000_000)
        return dict(kind=kind, photons=n, time_bins=rng.choice([0, 0, 20, 100]))
    if kind == "telescope":
        return dict(kind=kind, photons=_size(rng, 50_000, 10_000_000),
                    tracer=rng.choice(["fp64", "fp64", "fp32"]))
    if kind == "showers":
        return dict(kind=kind, events=rng.randint(20, 200))
    if kind == "reflector":
        return dict(kind=kind, photons=_size(rng, 100_000, 8_000_000),
                    tracer=rng.choice(["fp64", "fp32"]))
    if kind == "camera":
        return dict(kind=kind, photons=_size(rng, 1000, 400_000), history=rng.random() < 0.5)
    if kind == "host":
        return dict(kind=kind, photons=_size(rng, 100_000, 5_000_000))
    if kind == "signal":
        return dict(kind=kind, photons=_size(rng, 10_000, 2_000_000))
    if kind == "calibrate":
        return dict(kind=kind, photons=_size(rng, 500_000, 8_000_000))
    if kind == "corsika":
        return dict(kind=kind, bunches=_size(rng, 5_000, 4_000_000))
    if kind == "forward":
        return dict(kind=kind, photons=_size(rng, 10_000, 2_000_000))
    return dict(kind="train", photons=128 * rng.randint(64, 1024))


# ---- what a program keeps: its telescopes and the sensor's description ------

@functools.lru_cache(maxsize=None)
def _flat(which):
    if which == "reflector":
        return factories.large_reflector_camera().flatten()
    if which == "camera":
        return factories.reflector_camera().flatten()
    return factories.light_field_telescope(**TELESCOPE).flatten()


@functools.lru_cache(maxsize=None)
def _scene(which):
    return engine.Scene(_flat(which))


@functools.lru_cache(maxsize=None)
def _signal_config():
    g = factories.LightFieldSensorGeometry(factories.LightFieldSensorConfig(
        expected_imaging_system_focal_length=TELESCOPE["focal_length"],
        expected_imaging_system_max_aperture_radius=TELESCOPE["aperture_radius"],
        max_FoV_diameter=math.radians(TELESCOPE["fov_deg"]),
        pixel_FoV_hex_flat2flat=math.radians(TELESCOPE["pixel_fov_deg"]),
        num_paxel_on_pixel_diagonal=TELESCOPE["paxels_on_diagonal"],
        housing_overhead=TELESCOPE["housing_overhead"],
        lens_refraction=Func1([[200e-9, 1.5], [1200e-9, 1.5]]),
        bin_reflection=Func1([[200e-9, 0.9], [1200e-9, 0.9]])))
    light = signal_chain.NightSkyBackgroundLight(
        g, Func1([[250e-9, 1e17], [400e-9, 3e17], [700e-9, 2e17]]))
    converter = signal_chain.PhotoElectricConverterConfig(
        Func1([[200e-9, 0.0], [450e-9, 0.6], [1200e-9, 0.0]]), 5e6, 0.1)
    return signal_chain.SignalChainConfig(converter, light, 50e-9, 0.5e-9, 0.4e-9)


def _event_sizes(case):
    """Log-uniform in [1e2, 1e6] photons per event, as the benchmark's
    batched events: the first of one fixed list, so that the size of a case
    does not depend on the seed."""
    return P.cherenkov_event_sizes(200, 2024)[:case["events"]]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


# ---- the state of one program before the call -------------------------------

def prepare(case, seed):
    kind = case["kind"]
    n = case.get("photons", 0)
    st = {"case": case, "seed": seed}
    if kind in ("event", "showers"):
        st["scene"] = _scene("telescope")
        sizes = [n] if kind == "event" else _event_sizes(case)
        st["photons"], _ = P.cherenkov_events(sizes, seed, device="cuda")
    elif kind == "telescope":
        st["scene"] = _scene("telescope")
        st["photons"] = P.downward_disc_source_device(n, seed, **DISC, dtype=_dtype(case))
    elif kind == "reflector":
        st["scene"] = _scene("reflector")
        st["photons"] = P.downward_disc_source_device(n, seed, 40.0, 110.0, 3.5,
                                                      dtype=_dtype(case))
    elif kind == "camera":
        st["scene"] = _scene("camera")
        st["photons"] = P.downward_disc_source_device(n, seed, 2.2, 10.0, 2.0)
    elif kind == "host":
        st["scene"] = _scene("telescope")
        st["in"] = {k: v.cpu().pin_memory() for k, v in
                    P.downward_disc_source_device(n, seed, **DISC).items()}
        st["out"] = {"sensor": torch.empty(n, dtype=torch.int32).pin_memory()}
        for k in FOUR[1:]:
            st["out"][k] = torch.empty(n, dtype=torch.float64).pin_memory()
        st["counts"] = torch.empty(st["scene"].num_sensors, dtype=torch.int32).pin_memory()
    elif kind == "signal":
        st["scene"] = _scene("telescope")
        # the same light in every seed, its photons in another order under
        # other ids: so every seed gives the same number of pulses
        ph = P.downward_disc_source_device(n, 17, **DISC)
        hit = st["scene"].propagate(ph, engine.PropagationConfig(10), engine.Philox(5),
                                    outputs=("sensor", "time"))
        at = torch.randperm(n, generator=_generator(seed), device="cuda")
        st["config"] = _signal_config()
        st["arrivals"] = (hit["sensor"][at], hit["time"][at], ph["wavelength"][at],
                          torch.arange(n, dtype=torch.int32, device="cuda"))
        st["efficiency"] = 0.3 + 0.4 * torch.rand(st["scene"].num_sensors, device="cuda",
                                                  generator=_generator(3))
    elif kind == "calibrate":
        st["scene"] = _scene("telescope")
    elif kind == "corsika":
        st["scene"] = _scene("telescope")
        st["bunches"] = _bunches(case["bunches"], seed)
    elif kind in ("forward", "train"):
        # plane mode: the network models the photon 5 cm below the lenses
        st["model"] = surrogate.Surrogate(_flat("telescope"), seed=seed,
                                          plane_z=TELESCOPE["focal_length"] - 0.05)
        g = _generator(seed)
        x = torch.zeros((n, surrogate.IN_LD), device="cuda")
        x[:, :5] = torch.rand((n, 5), generator=g, device="cuda") * 2.0 - 1.0
        st["x"] = x
        if kind == "train":
            # outputs as a part-trained network has them: of order one
            w, _, b = surrogate.param_slices()[4]
            st["model"].params[w] *= 30.0
            st["model"].params[b] = torch.linspace(-1.0, 1.0, 73, device="cuda")
            st["model"].pack()
            st["t"] = torch.randn((n, 4), generator=g, device="cuda")
            st["r"] = (torch.rand(n, generator=g, device="cuda") < 0.6).to(torch.uint8)
            st["loss"] = torch.zeros(1, device="cuda")
            st["grads"] = torch.zeros_like(st["model"].params)
    return st


def _dtype(case):
    return torch.float32 if case.get("tracer", "fp64") == "fp32" else torch.float64


def _bunches(n, seed):
    """Bunches as the benchmark makes them: within 150 m, within 4 degrees of
    the zenith, weights uniform in [0, 16], a seventh of them whole (the same
    weights in every seed: so every seed gives the same number of photons)."""
    u = torch.rand((7, n), generator=_generator(seed), device="cuda", dtype=torch.float64)
    theta, phi = torch.deg2rad(4.0 * u[2]), 2.0 * math.pi * u[3]
    weight = 16.0 * torch.rand(n, generator=_generator(3), device="cuda", dtype=torch.float64)
    weight[::7] = torch.floor(weight[::7])
    b = [30000.0 * u[0] - 15000.0, 30000.0 * u[1] - 15000.0, torch.sin(theta) * torch.cos(phi),
         torch.sin(theta) * torch.sin(phi), 10.0 * u[4] - 5.0, 5e5 + 1.5e6 * u[5], weight,
         -700.0 + 450.0 * u[6]]
    return torch.stack(b, dim=1).float().contiguous()


# ---- one pass ----------------------------------------------------------------

def run(st):
    case, seed = st["case"], st["seed"]
    kind = case["kind"]
    if kind in ("event", "showers", "telescope"):
        dtype = _dtype(case)
        out = st["scene"].propagate(st["photons"], engine.PropagationConfig(10),
                                    engine.Philox(seed), tracer=case.get("tracer", "fp64"),
                                    outputs=FOUR, out_dtype=dtype)
        if kind == "telescope":
            return out, st["scene"].bin_arrivals(out["sensor"])[0]
        if case.get("time_bins"):
            # 1 km from the production point to the ground, within 100 ns
            t0 = 1e3 / 299792458.0
            return out, st["scene"].bin_arrivals(out["sensor"], out["time"], case["time_bins"],
                                                 t0 - 50e-9, t0 + 150e-9)
        return out
    if kind == "reflector":
        return st["scene"].propagate(st["photons"], engine.PropagationConfig(5),
                                     engine.Philox(seed), tracer=case["tracer"], outputs=FOUR,
                                     out_dtype=_dtype(case))
    if kind == "camera":
        return st["scene"].propagate(st["photons"], engine.PropagationConfig(5),
                                     engine.Philox(seed), history=case["history"],
                                     outputs=FOUR + ("theta_x", "theta_y"))
    if kind == "host":
        return _run_host(st)
    if kind == "signal":
        s = signal_chain.run(st["scene"], st["config"], *st["arrivals"], st["efficiency"],
                             engine.Philox(DRAWS))
        return (s.channel_offset, s.arrival_time_slice, s.simulation_truth_id, s.nsb_count,
                s.nsb_exposure_start_time)
    if kind == "calibrate":
        return calibration.calibrate(st["scene"], TELESCOPE["aperture_radius"],
                                     math.radians(TELESCOPE["fov_deg"]) / 2.0,
                                     num_photons=case["photons"], seed=seed)
    if kind == "corsika":
        return st["scene"].corsika_photons(st["bunches"], engine.Philox(DRAWS))
    model = st["model"]
    if kind == "forward":
        return model.forward(st["x"])[:, :73]   # the other seven columns are padding
    model.train_step(st["x"], st["t"], st["r"], 2e-3, loss=st["loss"], grads=st["grads"])
    return {"loss": st["loss"], "grads": st["grads"], "params": model.params, "m": model.m,
            "v": model.v}


def _run_host(st):
    n = st["case"]["photons"]
    ph, res, rng = abi.mlgpu_photons(), abi.mlgpu_results(), abi.mlgpu_rng()
    ph.dtype, res.dtype = abi.F64, abi.F64
    for k, t in st["in"].items():
        setattr(ph, k, t.data_ptr())
    for k, t in st["out"].items():
        setattr(res, k, t.data_ptr())
    rng.mode, rng.seed = abi.RNG_PHILOX, st["seed"]
    settings = abi.mlgpu_settings(10, 0, abi.TRACER_FP64, 0, abi.TRAVERSAL_BVH)
    _native.check(_native.lib().mlgpu_propagate_and_bin_host(
        st["scene"].handle, C.byref(ph), n, C.byref(settings), C.byref(rng), C.byref(res),
        C.c_void_p(st["counts"].data_ptr()), None, 0, 0.0, 0.0))
    return st["out"], st["counts"]


# ---- what a pass cannot do without --------------------------------------------

def work(case):
    """Photon planes in (seven values), results out, and for the arithmetic of
    a traced photon the surfaces it really meets, not the search for them:
    about 400 operations (a transform, a quadric, a reflection or Fresnel
    step) for each of its interactions."""
    kind = case["kind"]
    n = case.get("photons", 0)
    out = 20 if case.get("tracer") == "fp32" else 28     # sensor, x, y, time
    inp = 28 if case.get("tracer") == "fp32" else 56
    sensors = {"reflector": 8443, "camera": 1440}.get(kind, 63379)
    if kind == "event":
        return {"bytes": (inp + out) * n + 4 * sensors * ((case.get("time_bins") or -1) + 1),
                "flops": 60.0 * n}
    if kind == "showers":
        total = int(_event_sizes(case).sum())
        return {"bytes": (inp + out) * total, "flops": 60.0 * total}
    if kind == "telescope":
        return {"bytes": (inp + out) * n + 4 * sensors, "flops": 1400.0 * n}
    if kind == "reflector":
        return {"bytes": (inp + out) * n, "flops": 800.0 * n}
    if kind == "camera":
        return {"bytes": (inp + out + 16 + (6 * HISTORY_BYTES if case["history"] else 0)) * n,
                "flops": 800.0 * n}
    if kind == "host":
        return {"bytes": (inp + out) * n + 4 * sensors, "flops": 1400.0 * n}
    if kind == "signal":
        # sensor, time, wavelength and id in; about three pulses for five photons out
        return {"bytes": 24 * n + 3 * n + 16 * sensors, "flops": 100.0 * n}
    if kind == "calibrate":
        return {"bytes": 48 * sensors, "flops": 1400.0 * n}
    if kind == "corsika":
        return {"bytes": 32 * case["bunches"] + 8 * 60 * case["bunches"],
                "flops": 60.0 * case["bunches"]}
    if kind == "forward":
        return {"bytes": (32 + 292) * n + 4 * NET_PARAMS, "flops": NET_FLOPS * n}
    return {"bytes": (32 + 16 + 1) * n + 32 * NET_PARAMS, "flops": 3.0 * NET_FLOPS * n}


def tolerance(case):
    """The tracers, the calibration, the signal chain and the bunches promise
    merlict's own results bit for bit, on each photon by itself.  The network
    multiplies in BF16 (8 bits) through five layers."""
    if case["kind"] == "forward":
        return {"rel": 1e-2, "max": 0.2}
    if case["kind"] == "train":
        return {"rel": 1.2e-2, "max": 0.5}
    return "exact"


# ---- the same in 64 bits --------------------------------------------------------

def exact(case, seed):
    """The bunches and the network in plain torch, in 64 bits.  A traced
    photon has none: a search of up to 78,378 surfaces for each interaction
    of each photon takes plain torch minutes (and the tracer's results are
    compared bit for bit); nor has the signal chain, whose draws follow one
    another photon by photon."""
    if case["kind"] == "corsika":
        return _exact_corsika(_bunches(case["bunches"], seed), DRAWS)
    if case["kind"] in ("forward", "train"):
        return _exact_network(case, prepare(case, seed))
    return None


def _uniforms(seed, n):
    """First uniform of Philox4x32-10 streams 0..n-1 (Salmon et al., SC'11),
    counter (0, stream low, stream high, tag), as the package documents it."""
    low = 0xFFFFFFFF
    c = [torch.zeros(n, dtype=torch.int64, device="cuda"), torch.arange(n, device="cuda"),
         torch.zeros(n, dtype=torch.int64, device="cuda"),
         torch.full((n,), 0x6D6C6374, dtype=torch.int64, device="cuda")]
    k0, k1 = seed & low, (seed >> 32) & low
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57      # the low 64 bits of each product
        c = [((p1 >> 32) & low) ^ c[1] ^ k0, p1 & low, ((p0 >> 32) & low) ^ c[3] ^ k1, p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & low, (k1 + 0xBB67AE85) & low
    return ((c[0] << 21) | (c[1] >> 11)).double() * 2.0 ** -53


def _exact_corsika(bunches, seed):
    b = bunches.double()
    whole = torch.floor(b[:, 6])
    count = whole.long() + (_uniforms(seed, len(b)) <= b[:, 6] - whole).long()
    u, v = b[:, 2], b[:, 3]
    z = torch.sqrt(1.0 - u * u - v * v)
    norm = torch.sqrt(u * u + v * v + z * z)
    along = b[:, 4] * 1e-9 * 299792458.0 + 1e3
    planes = (b[:, 0] * 1e-2 - u / norm * along, b[:, 1] * 1e-2 - v / norm * along,
              z / norm * along, u, v, -z, (b[:, 7] * 1e-9).abs())
    of = torch.repeat_interleave(torch.arange(len(b), device="cuda"), count)
    out = {k: p[of] for k, p in zip(P.PLANES, planes)}
    out["id"] = of.int()
    return out


def _exact_network(case, st):
    train = case["kind"] == "train"
    params = st["model"].params.double().requires_grad_(train)
    losses, outputs = [], []
    rows = 1 << 17
    for a in range(0, case["photons"], rows):
        y = _network(params, st["x"][a:a + rows].double())
        if not train:
            outputs.append(y.detach())
            continue
        loss = _loss(y, st["t"][a:a + rows].double(),
                     st["r"][a:a + rows].bool()) / case["photons"]
        loss.backward()
        losses.append(loss.detach())
    if not train:
        return torch.cat(outputs)
    return {"loss": torch.stack(losses).sum().reshape(1), "grads": params.grad, "params": None,
            "m": None, "v": None}


def _network(params, x):
    """Five inputs, sin and cos of pi 2^l x for 12 octaves, four layers of 256
    with SiLU, 73 outputs."""
    angle = math.pi * x[:, :5, None] * (2.0 ** torch.arange(12, device="cuda").double())
    waves = torch.stack([torch.sin(angle), torch.cos(angle)], dim=-1).reshape(len(x), 120)
    h = torch.cat([x[:, :5], waves, torch.zeros((len(x), 3), device="cuda").double()], dim=1)
    at = 0
    for layer, (fin, fout) in enumerate(((128, 256), (256, 256), (256, 256), (256, 256),
                                         (256, 73))):
        w = params[at:at + fin * fout].reshape(fout, fin)
        at += fin * fout
        h = h @ w.T + params[at:at + fout]
        at += fout
        if layer < 4:
            h = torch.nn.functional.silu(h)
    return h


def _loss(y, t, reached):
    """Cross-entropy of the reach logit, and for the photons that reached the
    negative log-likelihood under the mixture of eight Gaussians."""
    total = torch.nn.functional.binary_cross_entropy_with_logits(y[:, 0], reached.double(),
                                                                 reduction="sum")
    part = y[:, 1:].reshape(-1, 8, 9)
    sigma = part[:, :, 5:9].clamp(-9.0, 3.0)
    z = (t[:, None, :] - part[:, :, 1:5]) * torch.exp(-sigma)
    each = (-0.5 * z * z - sigma - 0.5 * math.log(2.0 * math.pi)).sum(dim=2)
    joint = torch.logsumexp(torch.log_softmax(part[:, :, 0], dim=1) + each, dim=1)
    return total - joint[reached].sum()
