"""The work a user of this package has it do, as timed cases.

Whole simulations through the drop-in ``run_linear`` and ``run_hypercube`` (the reference's own
entry points), the repeated backward pass of a kept photon map, the float64-geometry tracer,
waveform gradients, and the two neighbour searches of the C ABI on their own.
"""

import contextlib
import ctypes as C
import dataclasses
import math
import os

import numpy as np
import torch

from pyalbsim_gb300 import workloads
from pyalbsim_gb300._native import load_library
from pyalbsim_gb300.adjoint import simulate_with_jacobian, with_parameters
from pyalbsim_gb300.batch import run_hypercube, surface_gate
from pyalbsim_gb300.config import (
    LaserConfig, RunConfig, SceneConfig, SeaFloorConfig, SeaSurfaceConfig, SensorConfig, SimulationConfig,
    HeatmapConfig, TurbidityLayerConfig, WaterConfig,
)
from pyalbsim_gb300.config.gpu import GpuRunOptions
from pyalbsim_gb300.engine import GpuEngine
from pyalbsim_gb300.execution.linear import run_linear
from pyalbsim_gb300.utils.parameter_profile import ExponentialParameter, LinearParameter

# The sweep's ranges: the drop-in sweep's fields over the ranges of the hypercube workload.
SWEEP = {
    "height": (1.0, 40.0), "absorption": (0.02, 0.5), "scattering": (0.05, 1.5), "asymmetry": (0.80, 0.95),
    "floor_albedo": (0.05, 0.40), "surface_roughness": (0.1, 0.55), "field_of_view": (10e-3, 60e-3),
}


def listed():
    return [
        # the smallest call: one neighbour query batch on device buffers inside a caller's own loop
        {"name": "knn_noalloc_3k", "kind": "knn_noalloc", "points": 3000, "queries": 400, "k": 100},
        # KDTree.query on host arrays: a photon map checked or analysed outside a simulation
        {"name": "knn_200k", "kind": "knn", "points": 200_003, "queries": 20_011, "k": 100, "planar": False},
        # one batch of backward photons on a kept map, the default batch size (RunConfig)
        {"name": "backward_5k", "kind": "backward", "scene": "small", "forward": 100_000, "backward": 5_000, "k": 100},
        # run_linear with every default of the reference: shallow turbid water, heatmaps on, batches
        {"name": "linear_default", "kind": "linear", "scene": "default", "forward": 100_000, "backward": 25_000,
         "batches_forward": 10, "batches_backward": 5, "k": 100},
        # the CPU-runnable workload: 5 m of clear water from 400 m
        {"name": "linear_small_100k", "kind": "linear", "scene": "small", "forward": 100_000, "backward": 25_000,
         "batches_forward": 1, "batches_backward": 1, "k": 100},
        # the headline scene at a quick-look size, and at the largest that a case may take
        {"name": "linear_large_1m", "kind": "linear", "scene": "large", "forward": 1_000_000, "backward": 250_000,
         "batches_forward": 1, "batches_backward": 1, "k": 100},
        {"name": "linear_large_10m", "kind": "linear", "scene": "large", "forward": 10_000_000, "backward": 2_500_000,
         "batches_forward": 1, "batches_backward": 1, "k": 100},
        # depth-profiled water (the reference's TurbidityLayerModel), odd photon counts
        {"name": "linear_profiled", "kind": "linear", "scene": "profiled", "forward": 200_003, "backward": 50_001,
         "batches_forward": 1, "batches_backward": 1, "k": 32},
        # the fixed-radius estimate in place of the k nearest
        {"name": "linear_radius", "kind": "linear", "scene": "small_hg", "forward": 100_000, "backward": 25_000,
         "batches_forward": 1, "batches_backward": 1, "k": 100, "radius": 0.5},
        # the reference's own sweep: many small configurations, one call
        {"name": "sweep_8", "kind": "sweep", "samples": 8, "forward": 100_000, "backward": 25_000},
        # one gradient of an inversion step: adjoint run plus depth run, gated window
        {"name": "gradient_1m", "kind": "gradient", "forward": 1_000_000, "backward": 250_000},
        # the float64-geometry tracer, which runs that must match the reference photon by photon use
        {"name": "precise_200k", "kind": "precise", "scene": "large", "forward": 200_000, "backward": 50_000, "k": 100},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["knn_noalloc", "knn", "backward", "linear", "linear", "linear", "linear", "sweep", "gradient", "precise"])
    if kind == "knn_noalloc":
        k = rng.randint(1, 256)
        return {"kind": kind, "points": _log(rng, max(k, 64), 4096), "queries": _log(rng, 16, 20_000), "k": k}
    if kind == "knn":
        k = rng.randint(1, 256)
        return {"kind": kind, "points": _log(rng, 1_000, 1_000_000), "queries": _log(rng, 500, 40_000), "k": k,
                "planar": rng.random() < 0.3}
    if kind == "sweep":
        n = _log(rng, 20_000, 200_000)
        return {"kind": kind, "samples": rng.randint(2, 12), "forward": n, "backward": n // 4}
    if kind == "gradient":
        n = _log(rng, 50_000, 2_000_000)
        return {"kind": kind, "forward": n, "backward": n // 4}
    k = rng.choice([16, 32, 50, 100, 100, 100, 137, 256])
    if kind == "precise":
        n = _log(rng, 20_000, 400_000)
        return {"kind": kind, "scene": rng.choice(["small", "large"]), "forward": n, "backward": n // 4, "k": k}
    if kind == "backward":
        return {"kind": kind, "scene": rng.choice(["small", "large"]), "forward": _log(rng, 50_000, 1_000_000),
                "backward": _log(rng, 1_000, 100_000), "k": k}
    scene = rng.choice(["default", "small", "large", "large", "profiled", "small_hg"])
    n = _log(rng, 20_000, {"default": 500_000, "profiled": 300_000}.get(scene, 3_000_000))
    case = {"kind": kind, "scene": scene, "forward": n, "backward": max(n // rng.choice([2, 4, 4, 10]), 500),
            "batches_forward": rng.choice([1, 1, 3, 10]), "batches_backward": rng.choice([1, 1, 2, 5]), "k": k}
    if scene == "small_hg":
        case["forward"], case["backward"] = min(n, 200_000), min(case["backward"], 50_000)
        case["radius"] = round(rng.uniform(0.1, 0.5), 3)
    return case


# ---------------------------------------------------------------------------------------------
# configurations
# ---------------------------------------------------------------------------------------------

def _profiled():
    """Two depth-profiled layers, linear and exponential, in a low and slow survey geometry."""
    return SimulationConfig(
        scene=SceneConfig(flying_height=10.0),
        water=WaterConfig(layers=(
            TurbidityLayerConfig(height=1.0, absorption_coefficient=LinearParameter(0.05, 0.3),
                                 scattering_coefficient=LinearParameter(0.5, 1.5),
                                 refractive_index=LinearParameter(1.33, 1.35)),
            TurbidityLayerConfig(height=1.5, absorption_coefficient=ExponentialParameter(0.1, 0.4),
                                 scattering_coefficient=0.8, refractive_index=ExponentialParameter(1.34, 1.36),
                                 salinity=LinearParameter(30.0, 38.0)),
        )),
        laser=LaserConfig(divergence_angle=5e-3, nadir_angle=10.0, azimuth_angle=30.0, pulse_fwhm=3e-9),
        sensor=SensorConfig(aperture_radius=0.1, field_of_view=50e-3, sample_rate=int(1e9)),
        sea_floor=SeaFloorConfig(albedo=0.2),
        sea_surface=SeaSurfaceConfig(albedo=0.1, roughness=float(np.sqrt(0.05))),
        heatmap=HeatmapConfig(enabled=False),
    )


def _scene(case):
    name = case["scene"]
    if name == "default":
        cfg = SimulationConfig()
    elif name == "profiled":
        cfg = _profiled()
    elif name == "small_hg":
        cfg = workloads.small(0.9, radius=case.get("radius"))
    else:
        cfg = workloads.workload_config(name)
    return dataclasses.replace(cfg, photon_mapping_k=case["k"])


def _gradient_config():
    """The adjoint workload: 12 m of HG water, 10% above its truth, 200 ns around the returns."""
    truth = np.array([12.0, 0.08, 0.30, 0.90, 0.18, math.sqrt(0.08)])
    cfg = with_parameters(workloads.large(hg=0.9), 1.1 * truth)
    return dataclasses.replace(cfg, waveform_gate=surface_gate(cfg))


# ---------------------------------------------------------------------------------------------
# state
# ---------------------------------------------------------------------------------------------

def _clouds(case, seed):
    """Points as photon maps hold them (a dense spot and a wide halo around it, a plane or a
    volume 400 m below the sensor) and queries in and beyond them."""
    rng = np.random.default_rng(seed)
    m, q = case["points"], case["queries"]
    core = rng.normal(scale=[0.3, 1.0, 0.3], size=(m // 2, 3)) + [0.0, -402.0, 0.0]
    halo = rng.uniform([-4.0, -406.0, -4.0], [4.0, -400.0, 4.0], size=(m - m // 2, 3))
    pts = np.concatenate([core, halo])
    qs = rng.uniform([-6.0, -408.0, -6.0], [6.0, -398.0, 6.0], size=(q, 3))
    if case.get("planar"):
        pts[:, 1] = -400.0
        qs[: q // 2, 1] = -400.0
    return np.ascontiguousarray(pts.astype(np.float32)), np.ascontiguousarray(qs)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "seed": int(seed)}
    if kind == "knn_noalloc":
        pts, qs = _clouds(case, seed)
        n = len(qs) * case["k"]
        state["lib"] = load_library()
        state["points"], state["queries"] = torch.from_numpy(pts).cuda(), torch.from_numpy(qs).cuda()
        state["idx"] = torch.empty(n, dtype=torch.int32, device="cuda")
        state["dist"] = torch.empty(n, dtype=torch.float64, device="cuda")
    elif kind == "knn":
        state["points"], state["queries"] = _clouds(case, seed)
        state["engine"] = GpuEngine(workloads.small())
    elif kind == "backward":
        eng = GpuEngine(_scene(case))
        eng.forward(case["forward"], int(seed))
        eng.build_maps()
        state["engine"] = eng
    elif kind == "linear":
        state["config"] = _scene(case)
        state["run"] = RunConfig(
            photons_per_batch_forward=case["forward"] // case["batches_forward"], batches_forward=case["batches_forward"],
            photons_per_batch_backward=case["backward"] // case["batches_backward"],
            batches_backward=case["batches_backward"])
    elif kind == "sweep":
        # one window for every depth: the samples' waveforms then have the same bins
        base = workloads.small(hg=0.9)
        state["config"] = dataclasses.replace(base, waveform_gate=surface_gate(base, length=400e-9))
        state["run"] = RunConfig(photons_per_batch_forward=case["forward"], batches_forward=1,
                                 photons_per_batch_backward=case["backward"], batches_backward=1)
    elif kind == "gradient":
        state["config"] = _gradient_config()
    elif kind == "precise":
        state["config"] = _scene(case)
    else:
        raise ValueError(kind)
    return state


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------

def _named(waveforms):
    return {t.name: w for t, w in waveforms.items()}


def run(state):
    case, seed = state["case"], state["seed"]
    kind = case["kind"]
    if kind == "knn_noalloc":
        p, q = state["points"], state["queries"]
        rc = state["lib"].alb_knn_noalloc(
            C.c_void_p(p.data_ptr()), case["points"], C.c_void_p(q.data_ptr()), case["queries"], case["k"],
            C.c_void_p(state["idx"].data_ptr()), C.c_void_p(state["dist"].data_ptr()),
            C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError(state["lib"].alb_last_error(None).decode())
        return {"idx": state["idx"], "dist": state["dist"]}
    if kind == "knn":
        dist, idx = state["engine"].ctx.knn(state["points"], state["queries"], case["k"])
        return {"idx": idx, "dist": dist}
    if kind == "backward":
        eng = state["engine"]
        eng.ctx.reset_waveform()
        eng.backward(case["backward"], seed, first=0)
        return _named(eng.waveform())
    if kind == "linear":
        with open(os.devnull, "w") as sink, contextlib.redirect_stdout(sink):
            return _named(run_linear(state["config"], state["run"], rng=np.random.default_rng(seed)))
    if kind == "sweep":
        out = run_hypercube(SWEEP, case["samples"], state["run"], seed=seed, base=state["config"])
        return {"s%02d" % i: _named(s["waveform"]) for i, s in enumerate(out)}
    if kind == "gradient":
        w, jac = simulate_with_jacobian(state["config"], case["forward"], case["backward"], seed)
        return {"waveform": w, "jacobian": jac}
    with GpuEngine(state["config"], GpuRunOptions(precise=True)) as eng:
        eng.forward(case["forward"], seed)
        eng.build_maps()
        eng.backward(case["backward"], seed)
        return _named(eng.waveform())


# ---------------------------------------------------------------------------------------------
# work and exact values
# ---------------------------------------------------------------------------------------------

# Records per forward photon, and gathers per backward photon, of each scene (counted on seed 1).
PER_PHOTON = {
    "default": (28.2, 28.2), "small": (7.2, 7.2), "small_hg": (7.3, 7.3), "large": (38.0, 38.1),
    "profiled": (8.7, 9.2), "gradient": (19.7, 19.7), "sweep": (40.0, 40.0),
}


def work(case):
    """A record is written once by the tracer, then read and written once by the index (32 B
    each); a query is written and read once (48 B); a neighbour takes 64 operations (distance,
    weight, sum) and an event 64. A standalone search reads its points and queries and writes
    its answers, and takes 8 operations a neighbour candidate."""
    kind, k = case["kind"], case.get("k", 100)
    if kind in ("knn", "knn_noalloc"):
        m, q = case["points"], case["queries"]
        return {"bytes": 12 * m + 24 * q + 12 * q * k, "flops": 8 * q * k}
    per_f, per_b = PER_PHOTON[case.get("scene", kind)]
    runs = case.get("samples", 2 if kind == "gradient" else 1)
    rec = 0 if kind == "backward" else per_f * case["forward"] * runs
    qry = per_b * case["backward"] * runs
    return {"bytes": 96 * rec + 96 * qry, "flops": 64 * (rec + qry) + 64 * qry * k}


def exact(case, seed):
    """The neighbour searches by brute force in 64 bits. The simulations are Monte Carlo runs
    on this package's own random streams: nothing else gives their values."""
    if case["kind"] not in ("knn", "knn_noalloc"):
        return None
    pts, qs = _clouds(case, seed)
    p, q = torch.from_numpy(pts).cuda().double(), torch.from_numpy(qs).cuda()
    out = []
    for c in torch.split(q, max(1, (1 << 28) // len(p))):
        d2 = (p[None, :, 0] - c[:, None, 0]) ** 2
        d2 += (p[None, :, 1] - c[:, None, 1]) ** 2
        d2 += (p[None, :, 2] - c[:, None, 2]) ** 2
        out.append(torch.topk(d2, case["k"], dim=1, largest=False, sorted=True)[0].sqrt())
    dist = torch.cat(out)
    if case["kind"] == "knn_noalloc":
        dist = dist.reshape(-1)
    return {"idx": None, "dist": dist.cpu().numpy()}
