"""Device functions of the library on arrays of their own (device_checks.cu, compiled here)."""

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from pyalbsim_gb300.build import ARCH, CSRC, FLAGS, INCLUDE, nvcc_path

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def dev(gpu_available, tmp_path_factory):
    out = str(tmp_path_factory.mktemp("device") / "checks.so")
    cmd = [nvcc_path(), *ARCH, *FLAGS, "-shared", "-I", INCLUDE, "-I", CSRC, "-o", out, os.path.join(HERE, "device_checks.cu")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(out)


def _gpu(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("on", [0, 1])
def test_word_cache_adds_to_the_words_it_is_given(dev, on):
    """Cached and direct adds end in the words. Off, a key may wrap to any value (arrays of more than 2^32
    words): nothing is cached, whatever the key, so nothing is flushed into another array's word."""
    i = np.array([0, 5, 7, 5, 0, 3], np.uint64)
    v = np.array([1, -2, 1 << 40, 30, -(1 << 33), 7], np.int64)
    # off: keys 0 (of word 5 too), and the mark of an empty slot
    base = np.zeros(6, np.uint32) if on else np.array([0, 2**32 - 5, 0, 2**32 - 5, 0, 2**32 - 4], np.uint32)
    words, other = _gpu(np.zeros(8, np.int64)), _gpu(np.zeros(8, np.int64))
    args = [_gpu(i.view(np.int64)), _gpu(base.view(np.int32)), _gpu(v)]
    first, second = (words, other) if on else (other, other)
    rc = dev.check_word_cache(_p(words), *[_p(a) for a in args], 6, on, _p(first), C.c_uint32(8 if on else 0), _p(second))
    assert rc == 0
    want = np.zeros(8, np.int64)
    np.add.at(want, i.astype(np.int64), v)
    np.testing.assert_array_equal(words.cpu().numpy(), want)
    assert not other.cpu().numpy().any()


@pytest.mark.parametrize("nmax", [1, 7, 4_000, 420_000, 8_000_000, 30_000_000, 300_000_000])
@pytest.mark.parametrize("down", [True, False])
def test_steps_to_a_plane_are_the_first_past_it(dev, nmax, down):
    """Crossings at the last steps of a span, the first after it and anywhere in it, with steps and heights of
    every size: the count is decided by the exact comparison, however far the estimate is off."""
    rng = np.random.default_rng(nmax)
    n = 200_000
    at = np.where(rng.random(n) < 0.7, nmax + rng.integers(-2, 4, n), np.floor(nmax * rng.random(n))).clip(0)
    sy = np.exp(rng.uniform(np.log(1e-9), np.log(2.0), n)) * (-1.0 if down else 1.0)
    y0 = rng.uniform(-40.0, 0.0, n)
    lim = y0 + (at - rng.uniform(0.2, 0.8, n)) * sy
    lim = np.where(at > 0, lim, np.nextafter(y0, y0 + sy))  # the start is on the near side of the plane
    bad = _gpu(np.zeros(1, np.int64))
    args = [_gpu(a) for a in (y0, sy, lim)]
    assert dev.check_steps(*[_p(a) for a in args], C.c_int64(n), C.c_int64(nmax), _p(bad)) == 0
    assert bad.item() == 0


@pytest.mark.parametrize("kind", ["random", "mantissas", "times", "angles", "heights"])
def test_quotients_by_a_constant_are_the_division_operator_s(dev, kind):
    """Random operands, mantissas next to powers of two (where a quotient's estimate is off the most), and the
    operands in use: times over the sample step, angles over the bin width, depths over a layer's height."""
    rng = np.random.default_rng(3)
    n = 1 << 24
    if kind == "random":
        x, b = np.exp(rng.uniform(-30, 30, n)) * rng.choice([-1.0, 1.0], n), np.exp(rng.uniform(-30, 30, n))
    elif kind == "mantissas":
        near = lambda: (rng.choice([1.0, 2.0], n) + rng.choice([-1.0, 1.0], n)  # noqa: E731
                        * rng.integers(0, 40, n) * rng.choice([2.0**-23, 2.0**-52], n)) * 2.0 ** rng.integers(-20, 20, n)
        x, b = near(), near()
    elif kind == "times":
        x, b = rng.uniform(0.0, 1e6, n), rng.integers(1, 200, n).astype(np.float64)
    elif kind == "angles":
        x, b = rng.uniform(0.0, np.pi, n), np.full(n, np.pi / rng.integers(100, 20_000))
    else:
        x, b = rng.uniform(0.0, 60.0, n), rng.uniform(0.1, 60.0, n)
    bad = _gpu(np.zeros(2, np.int64))
    args = [_gpu(x), _gpu(b)]
    assert dev.check_quotients(*[_p(a) for a in args], C.c_int64(n), _p(bad)) == 0
    assert bad.tolist() == [0, 0]
