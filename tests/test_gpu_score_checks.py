"""Scoring checks its features on the device: values outside [0, 1] and
non-finite ones are refused wherever they stand, before masks are, and the
caller's outputs stay as they are; scores at block-edge colony counts equal the
oracle's bit for bit."""
import ctypes as C

import numpy as np
import pytest

from tests import _programs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("colonies", [1, 3, 4, 5, 129])
def test_scores_and_refusals(engine_lib, oracle, colonies):
    import gplsaco_gb300 as g
    rng = np.random.default_rng(900 + colonies)
    program = _programs.random_program(rng, extended=True, feature_spec_id=2)
    features = rng.random((12, colonies, 32), dtype=np.float32)
    features[0, 0, 0], features[11, -1, 31] = 0.0, 1.0
    masks = rng.integers(1, 0xFFFFFFFF, size=colonies, dtype=np.uint32)
    got = g.score_cuda(program, features, masks)
    scores, actions = oracle.score(program, features, masks)
    assert np.array_equal(got["scores"], scores) and np.array_equal(got["actions"], actions)
    arr = (type(g.program_to_c(program)) * 1)(g.program_to_c(program))
    for at in ((0, 0, 0), (11, colonies - 1, 31), (5, colonies // 2, 17)):
        for bad in (np.nan, np.inf, -np.inf, np.float32(-1e-30), np.nextafter(np.float32(1), np.float32(2))):
            broken, none = features.copy(), masks.copy()
            broken[at] = bad
            none[-1] = 0
            with pytest.raises(ValueError, match="features must be finite"):
                g.score_cuda(program, broken, masks)
            with pytest.raises(ValueError, match="features must be finite"):
                g.score_controller_cuda(program, broken, none)
            out_s, out_a = np.full((colonies, 32), 7.0, np.float32), np.full(colonies, 7, np.int32)
            assert engine_lib.faco_score(C.cast(arr, C.c_void_p), 1, broken.ctypes.data, 12, masks.ctypes.data,
                                         colonies, out_s.ctypes.data, out_a.ctypes.data) != 0
            assert (out_s == 7.0).all() and (out_a == 7).all()
    none = masks.copy()
    none[colonies // 2] = 0
    with pytest.raises(ValueError, match="no legal action"):
        g.score_cuda(program, features, none)
