"""The zerocheck's plain rounds at sizes where the weighted ones normally run: a high coordinate of the
point is 0 or 1, which the weighted form cannot divide by. Every message and the final values against the
oracle's (tests/native/plain_rounds.cu), and the same point as drawn (weighted) beside them."""
import os
import subprocess

import pytest

from flock_gb300 import BLAKE3, KECCAK, SHA256

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def harness():
    import __graft_entry__ as g

    out_dir = os.path.join(ROOT, "tests", "native", "_build")
    os.makedirs(out_dir, exist_ok=True)
    exe = os.path.join(out_dir, "plain_rounds")
    src = os.path.join(ROOT, "tests", "native", "plain_rounds.cu")
    objs = [os.path.join(g.OBJ_DIR, f)
            for f in ("witness.o", "commit.o", "sumcheck.o", "rounds.o", "backend.o", "host_accel.o")]
    deps = [src] + objs + g._headers() + [os.path.join(ROOT, "oracle", "cpu_backend.h")]
    if not os.path.exists(exe) or os.path.getmtime(exe) < max(os.path.getmtime(p) for p in deps):
        g._run([g._nvcc(), *g.NVCC_FLAGS, src, *objs, "-o", exe, "-lpthread"])
    return exe


@pytest.mark.parametrize("kind,log_n,from_top,value", [
    (BLAKE3, 11, 0, 0),   # weighted chunks of 2^10 as drawn; a grid of one pass over the pairs
    (KECCAK, 9, 1, 1),
    (SHA256, 13, 3, 0),   # folds of 2^19 and 2^18 pairs: four and two passes of the widest grid
    (BLAKE3, 13, 9, 1),   # the lowest coordinate of the chunks' weight
    (BLAKE3, 13, 10, 0),  # the one below it: the weighted rounds
    (BLAKE3, 13, 0, 2),   # as drawn
])
def test_rounds_match_oracle(harness, kind, log_n, from_top, value):
    r = subprocess.run([harness, str(kind), str(1 << log_n), str(from_top), str(value)], stdout=subprocess.PIPE,
                       stderr=subprocess.STDOUT, text=True, timeout=900)
    assert r.returncode == 0 and "PLAIN ROUNDS OK" in r.stdout, r.stdout[-2000:]
