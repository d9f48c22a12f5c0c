"""Forward calls whose record stores turn out too small, and calls that measure their rates first: records, counters,
the radius heatmap and the waveform are those of calls that had room from the start, bit for bit."""

import dataclasses

import numpy as np
import pytest

from pyalbsim_gb300 import workloads
from pyalbsim_gb300._native import ALB_OPT_MAP_CAPACITY, batch_run
from pyalbsim_gb300.config import SimulationConfig
from pyalbsim_gb300.engine import GpuEngine
from pyalbsim_gb300.scene import build_scene

pytestmark = pytest.mark.gpu


def _run(cfg, forward, backward, room=0):
    with GpuEngine(cfg) as eng:
        if room:
            eng.ctx.set_option(ALB_OPT_MAP_CAPACITY, room)
        events = 0
        for a, b in zip(forward, forward[1:]):
            eng.forward(b - a, 5)
            st = eng.ctx.stats()
            assert st["photons"] == st["forward_photons"] == b - a
            assert st["events"] == st["forward_events"]
            events += st["events"]
        sizes = [eng.ctx.map_size(c) for c in range(4)]
        eng.build_maps()
        queries = 0
        for a, b in zip(backward, backward[1:]):
            eng.backward(b - a, 5)
            queries += sum(v["queries"] for k, v in eng.ctx.stats().items() if k.startswith("gather"))
        heat = eng.ctx.heatmaps() if eng.scene.heatmap_enabled else ()
        return [eng.waveform_array(f64=True), *heat], (events, sizes, queries)


def _assert_equal(a, b):
    assert a[1] == b[1]
    for x, y in zip(a[0], b[0]):
        assert np.abs(x).sum() > 0
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("scene", ["small", "default"])
def test_a_call_with_a_pilot_equals_calls_without(gpu_available, scene):
    """More than 2^18 photons in a first call: 2^14 are traced first to measure the rates, and the rest
    appends to their records."""
    cfg = workloads.small() if scene == "small" else SimulationConfig()
    n = (1 << 18) + 777
    one = _run(cfg, [0, n], [0, 5_000])
    _assert_equal(one, _run(cfg, [0, 100, n // 2, n], [0, 5_000]))


def test_a_backward_call_with_a_pilot_equals_calls_without(gpu_available):
    """Forward calls of fewer than 1024 photons measure no rates: a large backward call measures its own."""
    cfg = workloads.small()
    forward = list(range(0, 20_001, 1_000))
    one = _run(cfg, forward, [0, 70_001])
    stepwise = _run(cfg, forward, [0, 500, 70_001])
    _assert_equal(one, stepwise)


def _turbid():
    """Some hundreds of scatter records per photon: more than a first small call has room for."""
    cfg = SimulationConfig()
    layer = dataclasses.replace(cfg.water.layers[0], height=30.0, absorption_coefficient=0.01, scattering_coefficient=4.0)
    return dataclasses.replace(cfg, water=dataclasses.replace(cfg.water, layers=(layer,)))


@pytest.mark.parametrize("n", [3_000, (1 << 18) + 5])
def test_a_call_traced_again_equals_one_with_room(gpu_available, n):
    """The first trace overflows its stores: counters, records and the radius heatmap are undone and the photons
    traced again."""
    cfg = _turbid()
    once = _run(cfg, [0, n], [0, 1_000])
    assert once[1][1][1] > 130 * n
    _assert_equal(once, _run(cfg, [0, n], [0, 1_000], room=800 * n))
    _assert_equal(once, _run(cfg, [0, n // 3, n], [0, 1_000]))


def test_a_batch_worker_s_rates_do_not_matter(gpu_available):
    """One worker runs a clear scene, then a turbid one with the clear one's rates, then a clear one."""
    gate = (2.6e-6, 300e-9)
    clear = dataclasses.replace(workloads.small(0.9), waveform_gate=gate)
    layer = dataclasses.replace(clear.water.layers[0], scattering_coefficient=3.0, height=20.0)
    turbid = dataclasses.replace(clear, water=dataclasses.replace(clear.water, layers=(layer,)))
    scenes = [build_scene(c) for c in (clear, turbid, clear)]
    nf, nb = [30_000, 20_000, 10_000], [3_000, 2_000, 1_000]
    together, _, status, _ = batch_run(scenes, nf, nb, [1, 2, 3], streams=1)
    assert not status.any()
    for i in range(3):
        alone, _, status, _ = batch_run(scenes[i:i + 1], nf[i:i + 1], nb[i:i + 1], [i + 1], streams=1)
        assert not status.any() and np.abs(alone[0]).sum() > 0
        np.testing.assert_array_equal(together[i], alone[0])
