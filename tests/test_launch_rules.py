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
extern "C" float shared_factor(int full, unsigned block_bytes) { return faco::host_shared_factor(full, block_bytes); }
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


@pytest.mark.parametrize("n,sign", [(2049, -1), (2500, -1), (3000, -1), (3500, 1), (4485, 1), (5000, 1), (10000, 1)])
def test_shared_memory_is_favoured_while_three_blocks_fit(host, n, sign):
    """A full panel's class above N=2048 keeps shared memory, though it times
    like the workspace when alone, where three blocks of four ants (8 n bytes of
    coordinates; per ant 4 n of tour and inverse, n / 4 of bits) fit on an SM,
    and the workspace elsewhere; a panel that is not full goes by the times."""
    host.shared_factor.restype = C.c_float
    words = (n + 31) // 32
    block = (8 * n + 15) // 16 * 16 + 4 * ((4 * ((n + 7) // 8 * 8) + 8 * words + 15) // 16 * 16)
    assert host.shared_factor(0, block) == 1.0
    assert np.sign(host.shared_factor(1, block) - 1.0) == sign


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
