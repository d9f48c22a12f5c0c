"""The gather's result does not depend on how its queries are ordered or cut into chunks: the
waveform is a sum in fixed point over exact neighbour sets. Query counts around the edges of the
chunk rule (one query, a few, one per resident warp) and of the key width (2^18), each against the
unsorted order, bit for bit."""

import dataclasses

import numpy as np
import pytest

from pyalbsim_gb300 import workloads
from pyalbsim_gb300.config.gpu import GpuRunOptions
from pyalbsim_gb300.engine import GpuEngine

pytestmark = pytest.mark.gpu


def _waveform(cfg, n_backward, sort):
    with GpuEngine(cfg, GpuRunOptions(sort_queries=sort)) as eng:
        eng.forward(20_000, 5)
        eng.build_maps()
        eng.backward(n_backward, 5)
        return eng.waveform_array(f64=True)


@pytest.mark.parametrize("n_backward", [1, 3, 2_433, 70_001])
@pytest.mark.parametrize("k", [1, 100])
def test_waveform_does_not_depend_on_the_query_order(gpu_available, n_backward, k):
    cfg = dataclasses.replace(workloads.small(), photon_mapping_k=k)
    a, b = _waveform(cfg, n_backward, True), _waveform(cfg, n_backward, False)
    assert np.abs(a).sum() > 0
    np.testing.assert_array_equal(a, b)


def test_radius_waveform_does_not_depend_on_the_query_order(gpu_available):
    cfg = workloads.small(0.9, radius=0.2)
    np.testing.assert_array_equal(_waveform(cfg, 2_000, True), _waveform(cfg, 2_000, False))


@pytest.mark.parametrize("precise", [False, True])
@pytest.mark.parametrize("k", [1, 31, 100, 128, 129, 256])
def test_scatter_search_finds_the_kth_distance(gpu_available, k, precise):
    """The scatter search on both sides of its candidate-buffer sizes (k = 128 / 129) and with
    queries of one and two floats per coordinate: the k-th distances against scipy's KDTree. Both
    are float64 distances between the same points; they differ by the rounding of three
    products and two sums, under 4 eps."""
    from scipy.spatial import cKDTree

    cfg = dataclasses.replace(workloads.small(), photon_mapping_k=k)
    for n_backward in (2, 700):
        with GpuEngine(cfg, GpuRunOptions(precise=precise)) as eng:
            eng.keep_record_ids()
            eng.forward(20_000, 7)
            eng.build_maps()
            eng.backward(n_backward, 7)
            q = eng.ctx.export_queries(1)
            pts = eng.ctx.export_map(1)[0]
        d = cKDTree(pts.astype(np.float64)).query(q["pos"], k=[k])[0][:, 0]
        assert len(d) > 0
        np.testing.assert_allclose(q["rk"], d, rtol=4 * np.finfo(np.float64).eps, atol=0)


def test_heatmap_sums_on_both_sides_of_the_class_word_limit(gpu_available):
    """Heatmaps of up to 512 bins add through class words and float32 cell numbers, larger ones
    directly and in float64. With every contribution inside, the totals of a 512 and a 513 bin map
    are the same fixed-point sum; reading it as float64 rounds once per cell, 2^-53 of it."""
    from pyalbsim_gb300.config import HeatmapConfig, SimulationConfig

    def totals(bins):
        cfg = dataclasses.replace(
            SimulationConfig(), heatmap=HeatmapConfig(bins=bins, water_extent=1000.0, seafloor_extent=1000.0))
        with GpuEngine(cfg) as eng:
            eng.forward(5_000, 3)
            eng.build_maps()
            eng.backward(1_250, 3)
            w, f, r = eng.ctx.heatmaps()
        return w.sum(), f.sum(), r.sum()

    a, b = totals(512), totals(513)
    assert a[0] > 0 and a[1] > 0 and a[2] > 0
    np.testing.assert_allclose(a, b, rtol=1e-12)


@pytest.mark.parametrize("bins", [200, 600])
def test_heatmap_cells_match_the_precise_formula(gpu_available, bins):
    """Scatter-radius free check of the cell numbers: the seafloor map's marginal over x equals a
    histogram of the same contributions at half the resolution, summed in pairs."""
    from pyalbsim_gb300.config import HeatmapConfig, SimulationConfig

    def maps(n):
        cfg = dataclasses.replace(SimulationConfig(), heatmap=HeatmapConfig(bins=n, water_extent=4.0, seafloor_extent=16.0))
        with GpuEngine(cfg) as eng:
            eng.forward(5_000, 3)
            eng.build_maps()
            eng.backward(1_250, 3)
            w, f, _ = eng.ctx.heatmaps()
        return w.reshape(n, n), f.reshape(n, n)

    # extents are powers of two and bins even, so the coarse cells' edges are fine cells' edges; a
    # cell's float64 quotient rounds onto an edge only for values within 1e-15 of it
    for fine, coarse in zip(maps(bins), maps(bins // 2)):
        pairs = fine.reshape(bins // 2, 2, bins // 2, 2).sum(axis=(1, 3))
        # truncation toward zero puts (-1, 0) into cell 0 on both grids: the outermost row and
        # column of the coarse map reach one coarse cell out, those of the fine map one fine cell
        np.testing.assert_allclose(pairs[1:, 1:], coarse[1:, 1:], rtol=1e-12, atol=1e-300)


def _check_knn(pts, qs, k):
    from scipy.spatial import cKDTree

    with GpuEngine(workloads.small()) as eng:
        dist, idx = eng.ctx.knn(pts, qs, k)
    ref, _ = cKDTree(pts.astype(np.float64)).query(qs, k=range(1, k + 1))
    # the same three products and two sums in float64, and a square root: under 4 eps
    np.testing.assert_allclose(dist, ref, rtol=4 * np.finfo(np.float64).eps, atol=0)
    d = np.sqrt(((pts[idx].astype(np.float64) - qs[:, None, :]) ** 2).sum(axis=2))
    np.testing.assert_allclose(d, dist, rtol=4 * np.finfo(np.float64).eps, atol=0)


@pytest.mark.parametrize("planar", [False, True])
@pytest.mark.parametrize("m", [1, 31, 33, 255, 256, 257, 4_097, 65_536, 65_537])
def test_index_of_every_size_answers_like_kdtree(gpu_available, m, planar):
    """Records at the edges of a leaf, of a warp's 256, of a sort tile and of the 24-bit keys."""
    rng = np.random.default_rng(m)
    pts = rng.normal(scale=[0.3, 1.0, 0.3], size=(m, 3)).astype(np.float32)
    qs = rng.uniform(-2.0, 2.0, size=(200, 3))
    if planar:
        pts[:, 1] = -400.0
        qs[:, 1] = -400.0
    _check_knn(pts, qs, min(m, 20))


@pytest.mark.parametrize("m", [3_000, 70_001])
def test_index_of_crowded_keys_answers_like_kdtree(gpu_available, m):
    """One point a thousand kilometres away: the keys cannot tell the others apart, and the records
    take the exact k-d order. Duplicates and a lattice beside it."""
    rng = np.random.default_rng(m)
    pts = rng.normal(scale=0.2, size=(m, 3))
    pts[: m // 3] = np.round(pts[: m // 3] * 20.0) / 20.0
    pts[0] = [1.0e6, 0.0, 0.0]
    _check_knn(pts.astype(np.float32), rng.uniform(-0.5, 0.5, size=(100, 3)), 33)


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("k", [1, 100, 128, 129])
def test_planar_searches_by_runs_equal_single_ones(gpu_available, k, adjoint):
    """Planar gathers of 2^16 queries and more search by runs where k <= 128, smaller ones one query at a
    time, and queries far from the spot leave the runs: the same photons in one backward call and
    in calls below the limit, bit for bit (the Jacobian too)."""
    cfg = dataclasses.replace(workloads.small(0.9), photon_mapping_k=k)

    def run(cuts):
        with GpuEngine(cfg, GpuRunOptions(adjoint=adjoint)) as eng:
            eng.forward(20_000, 5)
            eng.build_maps()
            for a, b in zip(cuts, cuts[1:]):
                eng.backward(b - a, 5)
            return eng.waveform_array(f64=True), eng.jacobian() if adjoint else None

    (wa, ja), (wb, jb) = run([0, 66_000]), run([0, 20_000, 40_000, 66_000])
    assert np.abs(wa).sum() > 0
    np.testing.assert_array_equal(wa, wb)
    if adjoint:
        assert np.abs(ja).sum() > 0
        np.testing.assert_array_equal(ja, jb)


def test_radius_work_items_on_both_sides_of_their_room(gpu_available):
    """A radius that holds the whole map: 700 photons want more work items (a query's boxes of 32 leaves)
    than the 2^20 there is room for, and the rest is searched in place; half of the photons at a
    time want fewer. The same photons, bit for bit."""
    cfg = workloads.small(0.9, radius=2_000.0)

    def run(cuts):
        with GpuEngine(cfg, GpuRunOptions()) as eng:
            eng.forward(100_000, 5)
            eng.build_maps()
            assert eng.ctx.map_size(1) > 380 * 1024
            for a, b in zip(cuts, cuts[1:]):
                eng.backward(b - a, 5)
            return eng.waveform_array(f64=True)

    a, b = run([0, 700]), run([0, 350, 700])
    assert np.abs(a).sum() > 0
    np.testing.assert_array_equal(a, b)
