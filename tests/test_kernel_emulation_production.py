"""The ant kernel's source on the CPU (tests/emulation) in the variants the
engine launches -- each mode compiled for one local search, single or batched
steps by the colony's last walk, and in the global-memory workspace the
parent's inverse copied from the colony -- against the oracle's ant, bit for
bit, lanes delayed at random; batches are tried exactly where the colony's
walk reaches the launch's line.  Sizes: one copied vector short of whole, one
that ends in the second of a copy's three rounds, and one above 2048 nodes,
where every relocation is deferred."""
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("kind,n,k,iterations,modes", [("uniform", 61, 8, 0, None),
                                                       ("clustered", 389, 15, 60, None),
                                                       ("clustered", 2100, 16, 10, "4,6")])
def test_production_variants_match_oracle(oracle, kind, n, k, iterations, modes):
    args = [kind, str(n), str(k), str(iterations)] + ([modes] if modes else [])
    out = subprocess.run([sys.executable, str(ROOT / "tests" / "emulation" / "production_ants.py")] + args,
                         capture_output=True, text=True, timeout=900, cwd=ROOT)
    assert out.returncode == 0, (out.stdout[-2000:], out.stderr[-3000:])
    assert "production ants equal the oracle" in out.stdout
