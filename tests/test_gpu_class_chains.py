"""A small uneven batch runs its size classes as chains of their own without
being asked to, whole graph replays and remainders alike; results equal the
unchained run's."""
import numpy as np
import pytest

from tests import _cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,classes", [((200, 1000), 2), ((100, 300, 600), 3), ((300, 310), 1)])
def test_classes_are_chains(engine_lib, sizes, classes):
    import gplsaco_gb300 as g
    got = {}
    for chains in (0, 1):
        e = g.FacoBatchEngine(max(sizes), len(sizes) + 1, g.FixedFacoSettings(ants=9, retention=0.9, chains=chains))
        for i, n in enumerate(sizes):
            e.register_problem(i, _cases.uniform_instance(n, seed=n).astype(np.float64))
        keys = np.array([*range(len(sizes)), 0], np.uint64)
        e.begin(keys, np.arange(keys.size, dtype=np.uint64), 8)
        for steps in (5, 32, 3):
            e.step(steps)
        plan = e.launch_plan()
        assert plan["size_classes"] == classes
        if classes > 1 and chains == 0:
            assert classes <= plan["chains"] <= keys.size   # every class in at least one
        else:
            assert plan["chains"] == 0
        got[chains] = e.finish()
        e.close()
    assert np.array_equal(got[0]["costs"], got[1]["costs"])
    assert np.array_equal(got[0]["colony_work"], got[1]["colony_work"])
    assert all(np.array_equal(a, b) for a, b in zip(got[0]["tours"], got[1]["tours"]))
