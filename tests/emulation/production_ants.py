"""Runs ants of the emulated ant kernel in the variants the engine launches
(production_entry.cpp) against the oracle's ant, as run_ants.py does for the
plain modes; exits non-zero on the first difference.  Test infrastructure only.

    python tests/emulation/production_ants.py KIND N K ITERATIONS [MODE,...]

The optional last argument limits the run to those engine modes.
"""
import ctypes as C
import os
import subprocess
import sys
from pathlib import Path

import make_emulator
import run_ants

BUILD = make_emulator.HERE / "_build" / "production"
LIB = BUILD / "libant_production.so"
ENTRY = make_emulator.HERE / "production_entry.cpp"
TWO_OPT, OR_OPT = 16, 32
FOLLOW = (5, 6, 7)
# a colony below the line of its launch, one on it, and a launch without a line
CHOICES = {False: ((30, 29),), True: ((30, 29), (30, 30), (0, 0))}


def build():
    sources = [make_emulator.HERE / "warp_shim.h", make_emulator.HERE / "uniform_check.h", ENTRY,
               Path(__file__), Path(make_emulator.__file__),
               *(make_emulator.CSRC / f for f in ("faco_common.cuh", "faco_ant.cuh", "faco_kernels.cu"))]
    if LIB.exists() and LIB.stat().st_mtime >= max(p.stat().st_mtime for p in sources):
        return LIB
    BUILD.mkdir(parents=True, exist_ok=True)
    make_emulator.BUILD = BUILD
    cpp = make_emulator.generate()
    text = cpp.read_text().replace((make_emulator.HERE / "emulator_entry.cpp").read_text(), "")
    batch = 'uniform_check("batched",'
    assert text.count(batch) == 1 and "emu_ant" not in text
    text = text.replace(batch, "if (tl_lane == 0) ++emu_batches; " + batch)
    text = text.replace("namespace faco {", "static unsigned emu_batches = 0;\nnamespace faco {", 1)
    cpp.write_text(text + ENTRY.read_text())
    tmp = LIB.with_suffix(f".{os.getpid()}.tmp")
    subprocess.run(["g++", "-std=c++20", "-O2", "-fPIC", "-shared", "-ffp-contract=off", "-Wno-unknown-pragmas",
                    f"-I{BUILD}", f"-I{make_emulator.HERE}", str(cpp), "-o", str(tmp), "-lpthread"], check=True)
    os.replace(tmp, LIB)
    return LIB


class Variant:
    """run_ants' library for one (batch_from, walk)."""

    def __init__(self, lib, batch_from, walk):
        vp = C.c_void_p
        self.call = lib.emu_production_ant
        self.call.argtypes = [C.c_uint32] * 7 + [vp] * 8 + [C.c_ulonglong, C.c_uint32, C.c_uint32, C.c_uint32,
                                                            C.c_longlong, C.c_uint32, vp, vp, vp, vp, vp]
        self.choice, self.batches = (batch_from, walk), C.c_uint(0)

    def emu_ant(self, mode, *rest):
        return self.call(mode, *self.choice, *rest, C.byref(self.batches))


def main() -> None:
    kind, n, k, iterations = sys.argv[1], int(sys.argv[2]), int(sys.argv[3]), int(sys.argv[4])
    modes = tuple(int(m) for m in sys.argv[5].split(",")) if len(sys.argv) > 5 else (0, 4, 5, 6, 7)
    lib = C.CDLL(str(build()))
    make = run_ants.instances.uniform if kind == "uniform" else run_ants.instances.clustered
    xy = make(n, 500 + n)
    b, w = min(64, n - 1 - k), min(20, n - 1)
    prep, key, parent, products = run_ants._state(xy, k, b, w, iterations, seed=3)
    runs = 0
    for mode in modes:
        for ls_mode, search in ((0, TWO_OPT), (1, OR_OPT)):
            for batch_from, walk in CHOICES[mode in FOLLOW]:
                variant = Variant(lib, batch_from, walk)
                batch, ant = run_ants.ANTS[runs % len(run_ants.ANTS)]
                run_ants._ant(variant, mode | search, ls_mode, xy, prep, key, parent, products, k, b, w, batch, ant)
                # batches exactly where the colony's walk reaches the line of its launch
                assert (variant.batches.value > 0) == (mode in FOLLOW and walk >= batch_from), (mode, batch_from, walk)
                runs += 1
    print(f"{kind} n={n} k={k} it={iterations}: {runs} production ants equal the oracle")


if __name__ == "__main__":
    main()
