"""faco_pheromone_step_noalloc, whose error word the update kernel hands to the
caller's variable, over sizes from the smallest to many blocks, with rows of four
candidates and odd ones, aligned buffers and shifted ones: equal to the
host-buffer step bit for bit; a bad parent or candidate anywhere, the last entry
included, is reported and leaves everything untouched."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ARGS = [float(np.float32(v)) for v in (0.98, 1e-7, 2e-6, 1.3e-8)]


@pytest.mark.parametrize("n,k,shift", [(3, 1, 0), (3, 2, 0), (33, 4, 0), (100, 7, 0), (1024, 16, 1), (8192, 32, 0),
                                       (8193, 32, 0), (11264, 20, 0), (11265, 20, 0), (11264, 23, 0), (2000, 33, 0)])
def test_noalloc_sizes(engine_lib, n, k, shift):
    import torch
    rng = np.random.default_rng(n + k)
    primary = rng.integers(0, n, (n, k)).astype(np.uint32)
    parent = rng.permutation(n).astype(np.uint32)
    primary[np.arange(n), 0] = np.roll(parent, -1)[np.argsort(parent)]
    eta = rng.uniform(1e-6, 1.0, (n, k)).astype(np.float32)
    trails = rng.uniform(1e-7, 2e-6, (n, k)).astype(np.float32)
    want_t, want_p = trails.copy(), np.zeros_like(trails)
    assert engine_lib.faco_pheromone_step(n, k, primary.ctypes.data, parent.ctypes.data, *map(C.c_float, ARGS),
                                          eta.ctypes.data, want_t.ctypes.data, want_p.ctypes.data) == 0

    def device(a):   # `shift` words past an aligned start
        buf = torch.zeros(a.size + shift, dtype=torch.float32 if a.dtype == np.float32 else torch.int32, device="cuda")
        buf[shift:] = torch.from_numpy(np.ascontiguousarray(a).view(np.float32 if a.dtype == np.float32 else np.int32)
                                       .reshape(-1)).cuda()
        return buf[shift:]

    def step(primary_d, parent_d, trails_d, products_d):
        torch.cuda.synchronize()
        return engine_lib.faco_pheromone_step_noalloc(n, k, primary_d.data_ptr(), parent_d.data_ptr(),
                                                      *map(C.c_float, ARGS), device_eta.data_ptr(),
                                                      trails_d.data_ptr(), products_d.data_ptr(), None)

    device_eta = device(eta)
    for bad_parent, at, value in ((True, n - 1, n), (True, n - 1, int(parent[0])), (False, n * k - 1, n),
                                  (False, 0, 2**31 - 1), (False, (n * k) // 2, n)):
        broken = (parent if bad_parent else primary).copy().reshape(-1)
        broken[at] = value
        t, p = device(trails), device(np.full_like(trails, 7.0))
        code = step(device(primary) if bad_parent else device(broken), device(broken) if bad_parent else device(parent),
                    t, p)
        assert code != 0
        assert np.array_equal(t.cpu().numpy(), trails.reshape(-1)) and (p == 7.0).all()
    t, p = device(trails), device(np.zeros_like(trails))
    assert step(device(primary), device(parent), t, p) == 0, engine_lib.faco_last_error()
    assert np.array_equal(t.cpu().numpy(), want_t.reshape(-1)) and np.array_equal(p.cpu().numpy(), want_p.reshape(-1))
