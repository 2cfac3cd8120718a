"""Training over rows taken in an order on the device equals, bit for bit,
training on the rows copied in that order, at batches of one tile, of partial
tiles, of more tiles than the step kernel sums at a time, and of more rows than
there are; orders out of range are refused."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,batch", [(1, 1), (127, 128), (5000, 4224), (9000, 4100), (3000, 10_000)])
def test_train_order_equals_copied_rows(engine_lib, rows, batch):
    from gplsaco_gb300 import prior
    rng = np.random.default_rng(rows)
    x = prior.to_bf16_bits(rng.random((rows, 8), dtype=np.float32))
    y = (rng.random(rows) < 0.2).astype(np.float32)
    order = rng.permutation(rows).astype(np.uint32)
    xs, ys = np.ascontiguousarray(x[order]), np.ascontiguousarray(y[order])
    params = [prior.init_params(3), prior.init_params(3)]
    losses = np.zeros((2, 3), np.float32)
    assert engine_lib.faco_mlp_train(params[0].ctypes.data, xs.ctypes.data, ys.ctypes.data, rows, 3, batch,
                                     C.c_float(3e-3), losses[0].ctypes.data) == 0
    assert engine_lib.faco_mlp_train_order(params[1].ctypes.data, x.ctypes.data, y.ctypes.data, order.ctypes.data,
                                           rows, 3, batch, C.c_float(3e-3), losses[1].ctypes.data) == 0
    assert np.array_equal(params[0], params[1]) and np.array_equal(losses[0], losses[1])
    assert np.isfinite(losses).all() and not np.array_equal(params[0], prior.init_params(3))
    order[rows // 2] = rows
    assert engine_lib.faco_mlp_train_order(params[1].ctypes.data, x.ctypes.data, y.ctypes.data, order.ctypes.data,
                                           rows, 3, batch, C.c_float(3e-3), losses[1].ctypes.data) != 0
