"""A run restored from a snapshot equals the uninterrupted one with the ants in
shared memory and in the global-memory workspace, whose ants copy the parent's
inverse (rebuilt on restore, not part of a snapshot), plain and under a
controller that restarts."""
import numpy as np
import pytest

from tests import _cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("workspace", [1, 2])
@pytest.mark.parametrize("n,restarts", [(61, False), (300, False), (129, True)])
def test_restored_run_equals_straight_run(engine_lib, workspace, n, restarts):
    import gplsaco_gb300 as g
    keys, seeds = np.array([5, 5, 6], np.uint64), np.array([1, 2, 3], np.uint64)
    # score 1 for restarting actions (descriptor 9), 0 for the others
    program = dict(ir_version=1, numeric_spec_id=1, feature_spec_id=3, opcode=[0], operand=[9], constant_bits=[])

    def engine():
        e = g.FacoBatchEngine(n, 3, g.FixedFacoSettings(ants=9, retention=0.9, workspace=workspace))
        for key in (5, 6):
            e.register_problem(key, _cases.uniform_instance(n, seed=n + key).astype(np.float64))
        return e

    def begin(e):
        if restarts:
            e.begin_programs(keys, seeds, [program], total_iterations=40)
        else:
            e.begin(keys, seeds, 8)

    straight = engine()
    begin(straight)
    straight.step(40)
    want = straight.finish()
    broken = engine()
    begin(broken)
    broken.step(19)
    state = broken.capture_state()
    broken.finish()
    resumed = engine()
    resumed.restore_state(state)
    resumed.step(21)
    got = resumed.finish()
    assert np.array_equal(got["costs"], want["costs"]) and np.array_equal(got["colony_work"], want["colony_work"])
    assert all(np.array_equal(a, b) for a, b in zip(got["tours"], want["tours"]))
    for e in (straight, broken, resumed):
        e.close()
