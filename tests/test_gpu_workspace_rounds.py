"""Shifts, reversals and copies in the global-memory workspace take several
rounds of a warp at once; panels whose sizes end in the first, a middle and the
last of them (a copied vector holds 8 nodes, a round 32 lanes) give the tours,
costs and work of the shared-memory placement, whose rounds are single."""
import numpy as np
import pytest

from tests import _cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 63, 192, 193, 256, 385, 767, 768, 776, 1153])
@pytest.mark.parametrize("ls_mode", [0, 1])
def test_global_rounds_equal_shared(engine_lib, n, ls_mode):
    import gplsaco_gb300 as g
    keys, seeds = np.array([3, 3, 4], np.uint64), np.array([1, 2, 3], np.uint64)
    got = {}
    for workspace in (1, 2):
        e = g.FacoBatchEngine(n, 3, g.FixedFacoSettings(ants=11, retention=0.95, workspace=workspace, ls_mode=ls_mode))
        for key in (3, 4):
            e.register_problem(key, _cases.uniform_instance(n, seed=n + key).astype(np.float64))
        e.begin(keys, seeds, 8)
        e.step(24)
        got[workspace] = e.finish()
        e.close()
    assert np.array_equal(got[1]["costs"], got[2]["costs"])
    assert np.array_equal(got[1]["colony_work"], got[2]["colony_work"])
    assert all(np.array_equal(a, b) for a, b in zip(got[1]["tours"], got[2]["tours"]))
