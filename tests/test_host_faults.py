"""What the host code does with several devices and when a call fails, on a CUDA runtime of host memory
(fake_runtime.cpp): no GPU is needed and none is used."""

import ctypes as C

import numpy as np
import pytest

import fake_cuda
from pyalbsim_gb300 import workloads
from pyalbsim_gb300.config import SimulationConfig
from pyalbsim_gb300._native import ALB_OPT_ADJOINT, NativeContext, scene_struct
from pyalbsim_gb300.scene import build_scene


@pytest.fixture(scope="module")
def library():
    return fake_cuda.load()


@pytest.fixture
def lib(library):
    library.fake_reset()
    yield library
    library.fake_reset()


class Context(NativeContext):
    def __init__(self, lib, scene, device=0):
        self.lib, self.scene = lib, scene
        self._params, self._keep = scene_struct(scene)
        self.h = C.c_void_p()
        self._check(lib.alb_create(C.byref(self._params), device, C.byref(self.h)))


def test_calls_use_the_context_s_device_whatever_is_current(lib):
    scene = build_scene(workloads.small(0.9))
    ctx = [Context(lib, scene, d) for d in (0, 1)]
    calls = [
        lambda c: c.set_option(ALB_OPT_ADJOINT, 1),
        lambda c: c.trace(True, 3000),
        lambda c: c.build_maps(),
        lambda c: c.trace(False, 800),
        lambda c: c.waveform(1),
        lambda c: c.waveform(1, f64=True),
        lambda c: c.jacobian(),
        lambda c: c.adjoint(np.ones((4, scene.n_bins))),
        lambda c: c.stats(),
        lambda c: c.export_map(1),
        lambda c: c.reset_waveform(),
        lambda c: c.reset(),
        lambda c: c.close(),
    ]
    for call in calls:
        for d in (0, 1):
            lib.cudaSetDevice(1 - d)
            call(ctx[d])
            assert not fake_cuda.violations(lib)
    assert lib.fake_used(0) == 0 and lib.fake_used(1) == 0


def _rates(lib, records, queries=(1.0, 8.0, 1.0)):
    lib.fake_rates(np.array(records, np.float64).ctypes.data, np.array(queries, np.float64).ctypes.data)


@pytest.mark.parametrize("first", [False, True])
def test_a_forward_call_out_of_memory_leaves_the_simulation_as_it_was(lib, first):
    """A large first call measures its record rates on its first photons, then has no room for the rest: the
    records and the radius heatmap are those from before the call, so that it can be made again."""
    _rates(lib, [1.0, 90.0, 1.0, 1.0])
    ctx = Context(lib, build_scene(SimulationConfig()))
    if first:  # records of an earlier call (too few photons to measure rates)
        ctx.trace(True, 500)
    sizes = [ctx.map_size(c) for c in range(4)]
    radius = ctx.heatmaps()[2]
    n = 400_000
    lib.fake_limit(0, lib.fake_used(0) + (1 << 30))  # the pilot's records take 0.1 GB, the rest 2.4
    with pytest.raises(RuntimeError, match="out of device memory"):
        ctx.trace(True, n)
    traced = lib.fake_traced()
    assert 0 < traced < n  # the pilot ran
    assert [ctx.map_size(c) for c in range(4)] == sizes
    np.testing.assert_array_equal(ctx.heatmaps()[2], radius)
    lib.fake_limit(0, 1 << 40)
    ctx.trace(True, n)
    assert [ctx.map_size(c) - s for c, s in enumerate(sizes)] == [n, 90 * n, n, n]
    assert ctx.heatmaps()[2][0] - radius[0] == n
    ctx.close()
    assert not fake_cuda.violations(lib)


def test_a_forward_call_with_a_device_error_leaves_the_simulation_as_it_was(lib):
    """A trace that hits its iteration cap, or a replay that runs out of variates, has appended records by then."""
    ctx = Context(lib, build_scene(SimulationConfig()))
    ctx.trace(True, 2_000)
    sizes, radius = [ctx.map_size(c) for c in range(4)], ctx.heatmaps()[2]
    lib.fake_fail_trace(-6)
    with pytest.raises(RuntimeError, match="iteration cap|replay|device error"):
        ctx.trace(True, 3_000)
    assert [ctx.map_size(c) for c in range(4)] == sizes
    np.testing.assert_array_equal(ctx.heatmaps()[2], radius)
    ctx.trace(True, 3_000)
    assert [ctx.map_size(c) - n for c, n in enumerate(sizes)] == [3_000, 24_000, 3_000, 3_000]
    assert ctx.heatmaps()[2][0] - radius[0] == 3_000
    ctx.close()


def test_a_failed_replay_keeps_no_device_memory(lib):
    """A replayed backward call on maps of too few records (an ordinary error: more photons are traced and the call
    repeated) gives the uploaded variates back."""
    _rates(lib, [0.01, 0.01, 0.01, 0.01])
    ctx = Context(lib, build_scene(workloads.small()))
    ctx.trace(True, 1_000)
    ctx.build_maps()
    replay = (np.zeros(11, np.int64), np.zeros(100_000), np.zeros(100_000, np.float32))
    used = []
    for _ in range(3):
        with pytest.raises(IndexError, match="fewer than k"):
            ctx.trace(False, 10, replay=replay)
        used.append(lib.fake_used(0))
    assert used[2] == used[0] < 1 << 30
    with pytest.raises(ValueError, match="replay offsets"):
        ctx.trace(False, 11, replay=replay)
    ctx.close()
    assert lib.fake_used(0) == 0


@pytest.mark.parametrize("radius", [None, 0.5])
def test_gathers_that_cannot_be_joined_are_waited_for(lib, radius):
    """The gathers of a small call run on streams of their own. Whichever event of the call cannot be
    recorded, no stream works on after it, nothing was freed under one, and no scratch stays taken."""
    ctx = Context(lib, build_scene(workloads.small(0.9, radius=radius)))
    ctx.trace(True, 3000)
    ctx.build_maps()
    ctx.trace(False, 800)
    used, failed = lib.fake_used(0), 0
    for n in range(1, 30):
        lib.fake_fail_record(n)
        try:
            ctx.trace(False, 800)
        except RuntimeError:
            failed += 1
        assert lib.fake_busy() == 0, n
        assert lib.fake_used(0) == used, n
        assert not fake_cuda.violations(lib), n
    assert failed == 4  # the fork and the three joins; the others are times of phases
    lib.fake_fail_record(0)
    ctx.close()
    assert lib.fake_used(0) == 0


def test_a_failed_map_build_keeps_no_timing_events(lib):
    ctx = Context(lib, build_scene(workloads.small()))
    ctx.trace(True, 100_000)
    lib.fake_limit(0, lib.fake_used(0))
    events = []
    for _ in range(3):
        with pytest.raises(RuntimeError, match="index build failed"):
            ctx.build_maps()
        events.append(lib.fake_events())
    assert events[2] == events[0]
    ctx.close()
    assert lib.fake_events() == 0


def test_a_call_does_not_report_an_earlier_call_s_allocation_failure(lib):
    """After a map build or a search that had no memory, the same call with memory succeeds."""
    ctx = Context(lib, build_scene(workloads.small()))
    ctx.trace(True, 100_000)
    pts, qs = np.zeros((5_000, 3), np.float32), np.zeros((100, 3))
    lib.fake_limit(0, lib.fake_used(0))
    with pytest.raises(RuntimeError, match="index build failed"):
        ctx.build_maps()
    with pytest.raises(RuntimeError, match="knn allocation failed"):
        ctx.knn(pts, qs, 3)
    with pytest.raises(RuntimeError, match="read-back buffer"):
        ctx.waveform(1)
    lib.fake_limit(0, 1 << 40)
    ctx.build_maps()
    ctx.knn(pts, qs, 3)
    ctx.trace(False, 100)
    ctx.close()


def _batch(lib, monkeypatch, scenes, n_forward, n_backward, **options):
    from pyalbsim_gb300 import _native

    monkeypatch.setattr(_native, "_lib", lib)
    lib.fake_trace_ms(2)  # the workers run side by side
    n = len(scenes)
    return _native.batch_run(scenes, [n_forward] * n, [n_backward] * n, range(n), **options)[2]


def test_batch_admits_the_room_that_a_first_call_takes(lib, monkeypatch):
    """A context's first small call takes room for far more records than most scenes make, and a batch worker
    keeps it: what the workers hold together stays within 80% of the device, and no instance runs twice."""
    _rates(lib, [1.0, 6.0, 1.0, 1.0], [1.0, 6.0, 1.0])
    lib.fake_limit(0, 40 << 30)
    scene = build_scene(workloads.small())
    status = _batch(lib, monkeypatch, [scene] * 600, 200_000, 50_000, streams=64)
    assert not status.any()
    assert lib.fake_traced() == 600 * 250_000
    assert lib.fake_peak(0) < 0.8 * (40 << 30)


def test_batch_admits_the_sums_of_a_long_timeline(lib, monkeypatch):
    """Few photons, but 84 000 bins with their Jacobian: 0.13 GB of sums for each worker's context."""
    _rates(lib, [1.0, 6.0, 1.0, 1.0], [1.0, 6.0, 1.0])
    lib.fake_limit(0, 2 << 30)
    scene = build_scene(workloads.large(hg=0.9))
    assert scene.n_bins > 80_000
    status = _batch(lib, monkeypatch, [scene] * 60, 2_000, 500, streams=40, adjoint=True)
    assert not status.any()
    assert lib.fake_traced() == 60 * 2_500
    assert lib.fake_peak(0) < 0.8 * (2 << 30)


def test_trim_memory_gives_a_device_s_idle_memory_back(lib, monkeypatch):
    from pyalbsim_gb300 import _native
    from pyalbsim_gb300.engine import trim_memory

    monkeypatch.setattr(_native, "_lib", lib)
    lib.cudaSetDevice(0)
    trim_memory(1)
    assert (lib.fake_trims(0), lib.fake_trims(1)) == (0, 1)
    with pytest.raises(ValueError, match="no such device"):
        trim_memory(2)


@pytest.mark.parametrize("records", [6.0, 40.0])
def test_a_first_call_without_its_full_room_takes_less(lib, records):
    """No memory for 96 scatter records a photon: the call starts with room for 8, and is traced again where the
    scene makes more."""
    _rates(lib, [1.0, records, 1.0, 1.0])
    ctx = Context(lib, build_scene(workloads.small()))
    n = 200_000
    lib.fake_limit(0, lib.fake_used(0) + (400 << 20))  # 0.67 GB for 96 records a photon, 0.06 for 8, 0.28 for 40
    ctx.trace(True, n)
    assert [ctx.map_size(c) for c in range(4)] == [n, records * n, n, n]
    assert lib.fake_traced() == (n if records < 8 else 2 * n)
    ctx.close()
    assert lib.fake_used(0) == 0 and not fake_cuda.violations(lib)
