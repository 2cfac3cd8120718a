"""Rules by which the engine shapes an evaluation's launches, from its own host
source, and panels whose size classes fall on both sides of them."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from tests import _cases

CSRC = Path(__file__).resolve().parents[1] / "gplsaco_gb300" / "csrc"

ENTRY = """
#include "faco_host.h"
extern "C" unsigned batch_from(int always, int full, int global_workspace) {
    return faco::host_batch_from(always, full, global_workspace);
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    at = tmp_path_factory.mktemp("rules")
    (at / "entry.cpp").write_text(ENTRY)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", f"-I{CSRC}", str(at / "entry.cpp"),
                    "-o", str(at / "rules.so")], check=True)
    return C.CDLL(str(at / "rules.so"))


def test_batch_line_is_that_of_the_launch(host):
    # (always, full, global workspace): on request none; else by where the launch's own ants keep their tours
    for full in (0, 1):
        for workspace in (0, 1):
            assert host.batch_from(1, full, workspace) == 0
    assert host.batch_from(0, 0, 0) < host.batch_from(0, 1, 0) < host.batch_from(0, 0, 1) == host.batch_from(0, 1, 1)


@pytest.mark.gpu
@pytest.mark.parametrize("chains", [0, 1])
def test_classes_with_lines_of_their_own(engine_lib, chains):
    """Instances of 300 and of 2100 nodes in one panel, the large class in the
    global-memory workspace (no tuner): batches chosen by class, with chains
    and without, change nothing."""
    import gplsaco_gb300 as g
    got = {}
    for follow in (0, 1, 2):
        e = g.FacoBatchEngine(2100, 6, g.FixedFacoSettings(ants=16, retention=0.98, autotune=0, chains=chains,
                                                           follow=follow))
        for key, n in enumerate((300, 2100)):
            e.register_problem(key, _cases.uniform_instance(n, seed=n).astype(np.float64))
        e.begin(np.array([0, 0, 0, 1, 1, 0], np.uint64), np.arange(6, dtype=np.uint64), 8)
        e.step(150)
        got[follow] = e.finish()
        e.close()
    for follow in (0, 2):
        assert np.array_equal(got[follow]["costs"], got[1]["costs"])
        assert np.array_equal(got[follow]["colony_work"], got[1]["colony_work"])
        assert all(np.array_equal(a, b) for a, b in zip(got[follow]["tours"], got[1]["tours"]))
