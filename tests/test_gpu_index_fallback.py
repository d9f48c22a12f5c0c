"""The exact k-d order of the index, which records take whose keys do not tell them apart (one point far outside
the others): every kind of per-CTA cell and the streaming partition levels, against scipy's KDTree."""

import numpy as np
import pytest

from pyalbsim_gb300 import workloads
from pyalbsim_gb300.engine import GpuEngine

pytestmark = pytest.mark.gpu


def _check(pts, qs, ks):
    sp = pytest.importorskip("scipy.spatial")
    pts = pts.astype(np.float32)
    tree = sp.cKDTree(pts.astype(np.float64))
    with GpuEngine(workloads.small()) as eng:
        def search(p, k):
            before = eng.ctx.stats()["launches"]
            out = eng.ctx.knn(p, qs, k)
            return *out, eng.ctx.stats()["launches"] - before

        inside = pts.copy()
        inside[0] = pts[1]
        plain = search(inside, ks[0])[2]
        for k in ks:
            dist, idx, launches = search(pts, k)
            assert launches >= plain + 8, (launches, plain)  # the k-d order was built
            ref_d, ref_i = tree.query(qs, k)
            # the same three products and two sums in float64, and a square root: under 4 eps
            np.testing.assert_allclose(dist, ref_d, rtol=4 * np.finfo(np.float64).eps, atol=0)
            for i in range(len(qs)):
                assert set(ref_i[i][ref_d[i] < ref_d[i][-1]]) <= set(idx[i]), (k, i)


@pytest.mark.parametrize("leaves", [2048 + 512 + 5, 2048 + 256 + 5, 2048 + 100, 256 + 128 + 3])
def test_cells_of_every_kind(gpu_available, leaves):
    """Perfect cells of 128, 64 and 32 leaves, general cells, single leaves and a partial last one; points on a
    coarse lattice and duplicates among them."""
    rng = np.random.default_rng(leaves)
    m = 32 * leaves - 11
    pts = rng.normal(scale=[0.5, 3.0, 0.5], size=(m, 3)) + [0.0, -405.0, 0.0]
    lat = rng.random(m) < 0.33
    pts[lat] = np.round(pts[lat] * 10.0) / 10.0
    dup = rng.random(m) < 0.1
    pts[dup] = pts[rng.integers(0, m, int(dup.sum()))]
    near = pts[rng.integers(0, m, 800)].astype(np.float32).astype(np.float64) + rng.normal(scale=0.03, size=(800, 3))
    far = np.stack([rng.uniform(-20, 20, 200), rng.uniform(-420, -390, 200), rng.uniform(-20, 20, 200)], 1)
    pts[0] = [1.0e6, 0.0, 0.0]
    _check(pts, np.concatenate([near, far]), (100, 7))


@pytest.mark.parametrize("planar", [False, True])
def test_streaming_partition_levels(gpu_available, planar):
    """3e6 points: more than nine levels above the per-CTA cells."""
    rng = np.random.default_rng(3)
    m = 3_000_001
    pts = rng.normal(scale=[0.5, 3.0, 0.5], size=(m, 3)) + [0.0, -405.0, 0.0]
    if planar:
        pts[:, 1] = -400.0
    qs = pts[rng.integers(0, m, 500)].astype(np.float32).astype(np.float64) + rng.normal(scale=0.01, size=(500, 3))
    pts[0] = [1.0e6, 0.0, 0.0]
    _check(pts, qs, (32,))
