"""Neighbour searches where many points lie at one distance: more than a search's candidate buffers and its
band of near ties hold. The k nearest are then any of the tied points, but exactly k of them, none
twice, and every nearer one."""

import ctypes as C
import dataclasses

import numpy as np
import pytest

from pyalbsim_gb300 import workloads
from pyalbsim_gb300._native import load_library
from pyalbsim_gb300.config.gpu import GpuRunOptions
from pyalbsim_gb300.engine import GpuEngine

pytestmark = pytest.mark.gpu


def _noalloc(pts, qs, k):
    torch = pytest.importorskip("torch")
    lib = load_library()
    p, q = torch.from_numpy(pts).cuda(), torch.from_numpy(qs).cuda()
    idx = torch.empty((len(qs), k), dtype=torch.int32, device="cuda")
    dist = torch.empty((len(qs), k), dtype=torch.float64, device="cuda")
    rc = lib.alb_knn_noalloc(C.c_void_p(p.data_ptr()), len(pts), C.c_void_p(q.data_ptr()), len(qs), k,
                             C.c_void_p(idx.data_ptr()), C.c_void_p(dist.data_ptr()), None)
    assert rc == 0
    torch.cuda.synchronize()
    return dist.cpu().numpy(), idx.cpu().numpy()


def _knn(pts, qs, k):
    with GpuEngine(workloads.small()) as eng:
        return eng.ctx.knn(pts, qs, k)


def _check(search, pts, qs, k):
    from scipy.spatial import cKDTree

    pts, qs = np.ascontiguousarray(pts, np.float32), np.ascontiguousarray(qs, np.float64)
    dist, idx = search(pts, qs, k)
    ref = cKDTree(pts.astype(np.float64)).query(qs, k=range(1, k + 1))[0]
    # the same three products and two sums in float64, and a square root: under 4 eps
    np.testing.assert_allclose(dist, ref, rtol=4 * np.finfo(np.float64).eps, atol=0)
    assert idx.min() >= 0 and idx.max() < len(pts)
    assert all(len(set(row)) == k for row in idx.tolist())
    own = np.sqrt(((pts[idx].astype(np.float64) - qs[:, None, :]) ** 2).sum(axis=2))
    np.testing.assert_allclose(own, dist, rtol=4 * np.finfo(np.float64).eps, atol=0)


def _lattice(shape, rng):
    pts = np.stack(np.meshgrid(*[np.arange(n, dtype=np.float64) for n in shape], indexing="ij"), axis=-1).reshape(-1, 3)
    centre = (np.array(shape) - 1.0) / 2.0
    # lattice points, cell centres (eight and more at each distance) and points anywhere
    qs = np.concatenate([np.floor(centre)[None], centre[None], rng.integers(0, shape, size=(10, 3)),
                         rng.integers(0, shape, size=(10, 3)) + 0.5, rng.uniform(-2.0, 18.0, size=(20, 3))])
    return rng.permutation(pts), qs


@pytest.mark.parametrize("search", [_noalloc, _knn])
@pytest.mark.parametrize("shape", [(16, 16, 16), (64, 1, 64)])
@pytest.mark.parametrize("k", [33, 128, 224, 225, 240, 255, 256])
def test_lattice(gpu_available, search, shape, k):
    pts, qs = _lattice(shape, np.random.default_rng(k))
    _check(search, pts, qs, k)


@pytest.mark.parametrize("search", [_noalloc, _knn])
@pytest.mark.parametrize("copies", [33, 100, 257, 300, 2_000])
@pytest.mark.parametrize("k", [1, 10, 40, 100, 256])
def test_duplicates_before_nearer_points(gpu_available, search, copies, k):
    """Copies of one point stored before nearer points, and copies among others."""
    rng = np.random.default_rng(copies)
    far = np.tile([[1.0, 0.0, 0.0]], (copies, 1))
    near = rng.uniform(-0.3, 0.3, size=(5, 3))
    rest = rng.uniform(1.5, 3.0, size=(300, 3))
    qs = np.concatenate([np.zeros((1, 3)), rng.normal(scale=0.05, size=(20, 3))])
    _check(search, np.concatenate([far, near, rest]), qs, k)
    _check(search, rng.permutation(np.concatenate([far, near, rest])), qs, k)


def _waveform(k, copies, n_backward, precise, forward=2_000):
    cfg = dataclasses.replace(workloads.small(0.9), photon_mapping_k=k)
    with GpuEngine(cfg, GpuRunOptions(precise=precise)) as eng:
        for _ in range(copies):
            eng.forward(forward, 5, first=0)  # the same photons again
        eng.build_maps()
        eng.backward(n_backward, 5)
        return eng.waveform_array(f64=True)


@pytest.mark.parametrize("precise", [False, True])
@pytest.mark.parametrize("copies,k,once", [(40, 80, 2), (64, 128, 2), (128, 256, 2), (300, 100, 1), (600, 256, 1)])
@pytest.mark.parametrize("n_backward", [700, 70_001])
def test_gather_of_repeated_photons(gpu_available, copies, k, once, n_backward, precise):
    """Every record `copies` times: k neighbours are k / once copies of each of the `once` nearest, so the
    waveform is k / once times that of the photons traced once. Contributions are equal and
    summed as integers; the reading as float64 rounds once on each side. (70 001 backward photons: planar gathers
    by runs where k <= 128.)"""
    if precise and n_backward > 1_000:
        n_backward = 1_000
    a, b = _waveform(k, copies, n_backward, precise), _waveform(once, 1, n_backward, precise)
    assert all(np.abs(w).sum() > 0 for w in b)
    np.testing.assert_allclose(a, b * (k // once), rtol=4 * np.finfo(np.float64).eps, atol=0)


@pytest.mark.parametrize("divergence", [1e-12, 3e-8, 1e-6])
def test_surface_gather_around_a_narrow_beam(gpu_available, divergence):
    """A beam of hardly any width: every surface query has its neighbours, out of 100 000, within a few
    units of double-float distance or at one point. The k-th distance is scipy's, and the same photons in one
    call and in several give the same bits."""
    from scipy.spatial import cKDTree

    cfg = workloads.small()
    cfg = dataclasses.replace(cfg, laser=dataclasses.replace(cfg.laser, divergence_angle=divergence))

    def run(cuts):
        with GpuEngine(cfg) as eng:
            eng.keep_record_ids()
            eng.forward(100_000, 5)
            eng.build_maps()
            for a, b in zip(cuts, cuts[1:]):
                eng.backward(b - a, 5)
            return (eng.waveform_array(f64=True), eng.ctx.stats()["crowded_queries"], eng.ctx.export_queries(2),
                    eng.ctx.export_map(2)[0])

    a, crowded, q, pts = run([0, 2_000])
    b = run([0, 700, 2_000])[0]
    assert (crowded > 1_000) == (divergence < 1e-7)
    d = cKDTree(pts.astype(np.float64)).query(q["pos"], k=[cfg.photon_mapping_k])[0][:, 0]
    np.testing.assert_allclose(q["rk"], d, rtol=4 * np.finfo(np.float64).eps, atol=0)
    assert np.abs(a[2]).sum() > 0
    np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("k", [1, 2, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("m", [16, 1_023, 1_024, 1_025, 4_096])
def test_many_queries_of_few_neighbours(gpu_available, m, k):
    """From 2^14 queries (k <= 4) or 2^16 (k <= 16) on, a lane answers a query; the same queries in smaller calls
    are answered by warps. Random points, a lattice with many ties, coincident points, and queries without an
    answer: the same indices and distances."""
    rng = np.random.default_rng(m)
    n = 1 << (14 if k <= 4 else 16)
    third = m // 3
    pts = rng.normal(size=(m, 3))
    pts[:third] = np.round(pts[:third] * 2.0) / 2.0
    pts[third : third + third // 2] = [1.0, 0.0, 0.0]
    pts = np.ascontiguousarray(pts.astype(np.float32))
    qs = rng.normal(size=(n, 3))
    qs[::3] = np.round(qs[::3] * 4.0) / 4.0
    qs[5, 1], qs[77, 0] = np.nan, np.inf
    dist, idx = _noalloc(pts, qs, k)
    for a in range(0, n, n // 8):
        d, i = _noalloc(pts, np.ascontiguousarray(qs[a : a + n // 8]), k)
        np.testing.assert_array_equal(dist[a : a + n // 8], d)
        np.testing.assert_array_equal(idx[a : a + n // 8], i)
    assert (idx[[5, 77]] == -1).all() and np.isnan(dist[[5, 77]]).all()
    ok = np.setdiff1d(np.arange(0, n, 37), [5, 77])
    _check(lambda p, q, kk: (dist[ok], idx[ok]), pts, qs[ok], k)
