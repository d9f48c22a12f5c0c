"""What the host code does with several devices and when a call fails, on a CUDA runtime of host memory
(fake_runtime.cpp): no GPU is needed and none is used."""

import ctypes as C

import numpy as np
import pytest

import fake_cuda
from pyalbsim_gb300 import workloads
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
