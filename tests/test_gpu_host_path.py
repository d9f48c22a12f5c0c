"""The host side of a run: buffer sizes measured by a first few photons, gathers of a small run beside one
another, and device memory kept between contexts change no value. A waveform is a sum of integers, so
the same photons give the same bits however the calls divide them."""

import dataclasses

import numpy as np
import pytest

from pyalbsim_gb300 import workloads
from pyalbsim_gb300.batch import surface_gate
from pyalbsim_gb300.config import SimulationConfig
from pyalbsim_gb300.config.gpu import GpuRunOptions
from pyalbsim_gb300.engine import GpuEngine
from pyalbsim_gb300.scene import build_scene

pytestmark = pytest.mark.gpu

N = 70_000  # more photons than a call traces without measuring its rates first


def _run(cfg, cuts, trim=False):
    with GpuEngine(cfg, GpuRunOptions()) as eng:
        if trim:
            assert eng.ctx.lib.alb_trim_memory(0) == 0
        for a, b in zip(cuts, cuts[1:]):
            eng.forward(b - a, 5)
        eng.build_maps()
        for a, b in zip(cuts, cuts[1:]):
            eng.backward(b - a, 5)
        wf = [eng.ctx.waveform(c, f64=True) for c in range(4)]
        heat = eng.ctx.heatmaps() if eng.scene.heatmap_enabled else ()
        return wf + list(heat), [eng.ctx.map_size(c) for c in range(4)]


@pytest.mark.parametrize("scene", ["small", "default"])
def test_one_call_equals_many(gpu_available, scene):
    cfg = workloads.small() if scene == "small" else SimulationConfig()
    one, sizes = _run(cfg, [0, N])
    many, sizes_many = _run(cfg, [0, 100, N // 2, N], trim=True)
    assert sizes == sizes_many and sum(sizes) > N
    assert np.abs(one[1]).sum() > 0
    for a, b in zip(one, many):
        np.testing.assert_array_equal(a, b)


def test_trim_refuses_an_unknown_device(gpu_available):
    with GpuEngine(workloads.small(), GpuRunOptions()) as eng:
        assert eng.ctx.lib.alb_trim_memory(4096) != 0
        eng.forward(100, 1)  # the device in use is unchanged


def test_shared_class_words_of_a_long_timeline(gpu_available):
    """More than 2^20 bins: the channels share one set of class words and gather in series. A window of the
    timeline has few bins, one set per channel and gathers side by side: the same bits in it."""
    cfg = workloads.small()
    cfg = dataclasses.replace(cfg, sensor=dataclasses.replace(cfg.sensor, sample_rate=32 * cfg.sensor.sample_rate))

    def run(c):
        with GpuEngine(c, GpuRunOptions()) as eng:
            eng.forward(5_000, 5)
            eng.build_maps()
            eng.backward(1_500, 5)
            return eng.waveform_array(f64=True)

    full = run(cfg)
    assert full.shape[-1] > 1 << 20
    gated = dataclasses.replace(cfg, waveform_gate=surface_gate(cfg, length=100e-9))
    part, first = run(gated), build_scene(gated).gate_start
    assert part.shape[-1] < 1 << 20 and np.abs(part).sum() > 0
    np.testing.assert_array_equal(part, full[:, first:first + part.shape[-1]])
