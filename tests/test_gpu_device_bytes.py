"""A union backend's counted device bytes and their estimate against the device's free memory: the jagged
assist's vectors (56 bytes a dense word, 470 MB here) are part of all three."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_union_bytes_are_counted():
    import __graft_entry__ as g

    out_dir = os.path.join(ROOT, "tests", "native", "_build")
    os.makedirs(out_dir, exist_ok=True)
    exe = os.path.join(out_dir, "device_bytes")
    src = os.path.join(ROOT, "tests", "native", "device_bytes.cu")
    objs = [os.path.join(g.OBJ_DIR, f)
            for f in ("witness.o", "commit.o", "sumcheck.o", "rounds.o", "backend.o", "host_accel.o")]
    if not os.path.exists(exe) or os.path.getmtime(exe) < max(os.path.getmtime(p) for p in [src] + objs + g._headers()):
        g._run([g._nvcc(), *g.NVCC_FLAGS, src, *objs, "-o", exe, "-lpthread"])
    r = subprocess.run([exe, "14", "10000", "6000", "15000"], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
    words = r.stdout.split()
    held, counted, estimate, dense = (int(words[words.index(k) + 1]) for k in ("held", "counted", "estimate", "dense_words"))
    assert dense == 1 << 23
    # about 75 allocations, each rounded up to at most 2 MiB
    assert -(16 << 20) <= held - counted <= 75 * (2 << 20), r.stdout
    assert abs(estimate - counted) <= 16 << 20, r.stdout
