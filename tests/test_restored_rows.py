"""What a restore takes from a snapshot besides copying it: the inverse of each
tour, built only for a permutation (on the CPU, from the engine's own host
source), the walk that its colonies start from, and the refusal of a snapshot
whose tours or parent neighbours could not be a colony's, checksum and all else
being right."""
import ctypes as C
import struct
import subprocess
from pathlib import Path

import numpy as np
import pytest

from tests import _cases

CSRC = Path(__file__).resolve().parents[1] / "gplsaco_gb300" / "csrc"

ENTRY = """
#include "faco_host.h"
extern "C" int inverse_of(const unsigned short* order, unsigned n, unsigned short* out) {
    return faco::host_inverse(order, n, out);
}
extern "C" unsigned mean_walk(unsigned long long steps, unsigned iterations, unsigned ants) {
    return faco::host_mean_walk(steps, iterations, ants);
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    at = tmp_path_factory.mktemp("host")
    (at / "entry.cpp").write_text(ENTRY)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", f"-I{CSRC}", str(at / "entry.cpp"),
                    str(CSRC / "faco_prepare.cpp"), "-o", str(at / "host.so")], check=True)
    return C.CDLL(str(at / "host.so"))


@pytest.mark.parametrize("n", [3, 8, 1000, 10000])
def test_inverse_only_of_a_permutation(host, n):
    def call(order):
        order, out = np.ascontiguousarray(order, np.uint16), np.zeros(n, np.uint16)
        return host.inverse_of(order.ctypes.data_as(C.c_void_p), n, out.ctypes.data_as(C.c_void_p)), out

    rng = np.random.default_rng(n)
    for order in (np.arange(n), np.arange(n)[::-1], rng.permutation(n)):
        ok, out = call(order)
        assert ok and np.array_equal(out, np.argsort(order))
        for at, value in ((0, order[1]), (n - 1, order[0]), (n // 2, n), (1, 0xffff)):
            broken = order.copy()
            broken[at] = value   # a node twice, or one beyond the last
            assert not call(broken)[0]


@pytest.mark.parametrize("steps,iterations,ants,walk", [(0, 0, 32, 0), (32 * 7, 1, 32, 7), (32 * 400 * 61 + 5, 400, 32, 61),
                                                        (9999 * 4096 * 2**32 - 1, 2**32 - 1, 4096, 9999)])
def test_walk_of_a_restored_colony(host, steps, iterations, ants, walk):
    host.mean_walk.argtypes = [C.c_ulonglong, C.c_uint, C.c_uint]
    host.mean_walk.restype = C.c_uint
    assert host.mean_walk(steps, iterations, ants) == walk


def _fnv1a(data: bytes) -> int:
    h = 1469598103934665603
    for byte in data:
        h = ((h ^ byte) * 1099511628211) & (2**64 - 1)
    return h


@pytest.mark.gpu
@pytest.mark.parametrize("workspace", [1, 2])
def test_broken_rows_are_refused(engine_lib, workspace):
    import gplsaco_gb300 as g
    n, colonies = 21, 2
    keys, seeds = np.array([4, 4], np.uint64), np.array([1, 2], np.uint64)
    e = g.FacoBatchEngine(n, colonies, g.FixedFacoSettings(ants=9, retention=0.9, workspace=workspace))
    e.register_problem(4, _cases.uniform_instance(n, seed=3).astype(np.float64))
    e.begin(keys, seeds, 8)
    e.step(6)
    state = e.capture_state().to_bytes()
    e.step(7)
    want = e.finish()
    # the closing rows: parent, neighbours, epoch best, global best, checksum
    pad = (n + 7) // 8 * 8
    total = colonies * pad
    ends = np.cumsum([0, 2 * total, 4 * total, 2 * total, 2 * total])
    base = len(state) - 8 - int(ends[-1])
    row = {name: base + int(at) for name, at in zip(("parent", "near", "epoch", "global"), ends)}
    for name, size in (("parent", 2), ("epoch", 2), ("global", 2), ("near", 4)):
        for colony in range(colonies):
            for value in ("other", n):
                broken = bytearray(state[:-8])
                at = row[name] + size * (colony * pad + n // 2)
                other = bytes(broken[at - size:at])
                broken[at:at + size] = other if value == "other" else struct.pack("<H" if size == 2 else "<I", value)
                broken += struct.pack("<Q", _fnv1a(broken))
                with pytest.raises(ValueError, match="snapshot"):
                    e.restore_state(g.CountedState(bytes(broken)))
    # and the engine goes on from the sound one
    e.restore_state(g.CountedState(state))
    e.step(7)
    got = e.finish()
    assert np.array_equal(got["costs"], want["costs"])
    assert all(np.array_equal(a, b) for a, b in zip(got["tours"], want["tours"]))
    e.close()


@pytest.mark.gpu
def test_broken_archive_is_refused(engine_lib):
    """The 12-feature controller's archive (the snapshot's last rows: two sides of
    four tours with their positions) and its start list."""
    import gplsaco_gb300 as g
    n, pad = 30, 32
    keys, seeds = np.array([4], np.uint64), np.array([1], np.uint64)
    program = dict(ir_version=1, numeric_spec_id=1, feature_spec_id=2, opcode=[0], operand=[0], constant_bits=[])
    e = g.FacoBatchEngine(n, 1, g.FixedFacoSettings(ants=9, retention=0.9))
    e.register_problem(4, _cases.uniform_instance(n, seed=3).astype(np.float64))
    e.begin_programs(keys, seeds, [program], total_iterations=20)
    e.step(7)
    state = e.capture_state().to_bytes()
    e.step(5)
    want = e.finish()
    rows = len(state) - 8 - 2 * 16 * pad
    body = bytearray(state[:-8])
    # the controller state before the rows ends: size, side, alternative, mask, start count, reserved,
    # positions of node 0 [4], start nodes [16]
    tail = struct.Struct("<6I4I16H")
    control = rows - tail.size
    size, side, _, _, _, _, *p0 = tail.unpack_from(body, control)
    at = rows + 2 * 4 * 2 * pad * side
    assert 1 <= size <= 4 and side <= 1
    tour = np.frombuffer(bytes(body), np.uint16, n, at)
    assert np.array_equal(np.sort(tour), np.arange(n)) and tour[p0[0]] == 0
    breaks = {"node": (at, struct.pack("<H", n)), "twice": (at, struct.pack("<H", int(tour[1]))),
              "position": (at + 2 * pad + 2 * 5, struct.pack("<H", n)), "size": (control, struct.pack("<I", 5)),
              "side": (control + 4, struct.pack("<I", 2)), "starts": (control + 16, struct.pack("<I", 17)),
              "zero": (control + 24, struct.pack("<I", n))}
    for where, value in breaks.values():
        broken = bytearray(body)
        broken[where:where + len(value)] = value
        broken += struct.pack("<Q", _fnv1a(broken))
        with pytest.raises(ValueError, match="snapshot archive"):
            e.restore_state(g.CountedState(bytes(broken)))
    e.restore_state(g.CountedState(state))
    e.step(5)
    got = e.finish()
    assert np.array_equal(got["costs"], want["costs"])
    assert all(np.array_equal(a, b) for a, b in zip(got["tours"], want["tours"]))
    e.close()
