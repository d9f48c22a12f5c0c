"""A photon's records depend on its number alone, not on the lane, warp or launch that traces it:
photons traced in one call against the same photons traced in several, record by record, at photon
counts around a warp, a block and a refill."""

import numpy as np
import pytest

from fixtures import config_from_fixture, load
from pyalbsim_gb300 import workloads
from pyalbsim_gb300.config.gpu import GpuRunOptions
from pyalbsim_gb300.engine import GpuEngine

pytestmark = pytest.mark.gpu


def _records(cfg, options, cuts):
    with GpuEngine(cfg, options) as eng:
        eng.keep_record_ids()
        for a, b in zip(cuts, cuts[1:]):
            eng.forward(b - a, 9)
        out = []
        for c in range(4):
            pos, d, e, t, _, _, pid = eng.ctx.export_map(c)
            rows = np.concatenate([pid[:, None].astype(np.float64), t[:, None], pos, d, e[:, None]], axis=1)
            out.append(rows[np.lexsort(rows.T[::-1])])
    return out


@pytest.mark.parametrize("precise", [False, True])
@pytest.mark.parametrize("scene", ["small", "profiled"])
@pytest.mark.parametrize("n", [1, 33, 129, 2_000])
def test_records_do_not_depend_on_the_launch(gpu_available, scene, precise, n):
    cfg = workloads.small() if scene == "small" else config_from_fixture(load("replay_profiled.npz"))
    options = GpuRunOptions(precise=precise)
    one, many = _records(cfg, options, [0, n]), _records(cfg, options, [0, n // 3, n // 2, n])
    assert sum(len(r) for r in one) >= n
    for a, b in zip(one, many):
        np.testing.assert_array_equal(a, b)
