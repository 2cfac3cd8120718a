"""The checklist local search at the LS widths where its packing of several
pops into one warp pass changes shape: one candidate per node, rows of half a
warp and one more, and rows of a whole warp (a node with both prefixes wide
takes two rounds); random tours give wide prefixes.  Tours, checklist order and
every counter are whole numbers and equal the oracle's."""
import numpy as np
import pytest

from tests import _cases
from tests.test_gpu_parity import _compare_ant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [1, 2, 8, 16, 17, 31, 32])
@pytest.mark.parametrize("n", [33, 260])
@pytest.mark.parametrize("ls_mode", [0, 1])
def test_checklist_widths(engine_lib, oracle, n, w, ls_mode):
    import gplsaco_gb300 as g
    xy = _cases.coordinates(n, 1, seed=4000 + n + w)
    matrix = oracle.euc2d_matrix(xy)
    rows = _cases.ls_rows(matrix, w, reverse=False)
    ants = 8
    tours, visits, targets = _cases.ant_tasks(n, ants, seed=n * 13 + w)
    for cap in (1, 31, 33, 64, 65, 2**32 + 5):
        gpu = g.ant_diagnostic(xy, rows, tours, targets, cap, visits=visits, ls_mode=ls_mode)
        for t in range(ants):
            ref = oracle.ant(tours[t], rows, int(targets[t]), cap, xy=xy, visit=visits[t], ls_mode=ls_mode)
            _compare_ant(gpu, t, ref, f"n={n} w={w} cap={cap} ant={t} ls_mode={ls_mode}")
