"""The device's integer EUC_2D length (faco_common.cuh), compiled for the host
with an estimate that is off by up to eight on purpose: the length is the
exactly rounded one whatever the estimate, over coincident points, unit steps,
half-way neighbours of squares and spans up to the registration limit."""
import ctypes as C
import subprocess
import sys
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "tests" / "emulation"))

SOURCE = """
#include <mutex>
#include "faco_common.cuh"
std::mutex g_atomic;
thread_local Warp* tl_warp = nullptr;
thread_local unsigned tl_lane = 0;
extern "C" void lengths(const int* p, const int* q, long n, int* out) {
    for (long i = 0; i < n; ++i)
        out[i] = faco::euc2d(int2{p[2 * i], p[2 * i + 1]}, int2{q[2 * i], q[2 * i + 1]});
}
"""


def test_euc2d_is_exact_for_any_near_estimate(tmp_path):
    import make_emulator
    make_emulator.generate()
    header = (make_emulator.BUILD / "faco_common.cuh").read_text()
    assert "r = std::sqrt(x);" in header
    (tmp_path / "lengths.cpp").write_text(SOURCE)
    rng = np.random.default_rng(5)
    p = np.concatenate([rng.integers(-span, span + 1, (20_000, 2)) for span in
                        (1, 3, 40, 1000, 10**5, 10**6, 2**23 - 1)]).astype(np.int32)
    q = np.roll(p, 1, axis=0)
    q[::7] = p[::7]
    q[1::7] = p[1::7] + [0, 1]
    d = p.astype(np.int64) - q
    s = (d * d).sum(axis=1)
    keep = (np.abs(d) < 2**24).all(axis=1)
    p, q, s = np.ascontiguousarray(p[keep]), np.ascontiguousarray(q[keep]), s[keep]
    want = np.floor(np.sqrt(s.astype(np.float64)) + 0.5).astype(np.int64)
    assert ((want * want - want < s) | (want == 0)).all() and (s <= want * want + want).all()
    for off in (0.0, 0.51, -0.51, 1.2, -1.2, 3.0, -3.0, 8.0, -8.0):
        (tmp_path / "faco_common.cuh").write_text(
            header.replace("r = std::sqrt(x);", f"r = std::max(0.0f, std::sqrt(x) + {off!r}f);")
                  .replace("#include <cstdint>", "#include <algorithm>\n#include <cstdint>", 1))
        lib = tmp_path / f"lengths_{off}.so"
        subprocess.run(["g++", "-std=c++20", "-O2", "-fPIC", "-shared", "-ffp-contract=off", f"-I{tmp_path}",
                        f"-I{make_emulator.HERE}", str(tmp_path / "lengths.cpp"), "-o", str(lib), "-lpthread"],
                       check=True)
        out = np.zeros(len(p), np.int32)
        C.CDLL(str(lib)).lengths(p.ctypes.data_as(C.c_void_p), q.ctypes.data_as(C.c_void_p), C.c_long(len(p)),
                                 out.ctypes.data_as(C.c_void_p))
        assert np.array_equal(out, want), off
