"""Witness kernels that split an instance's chunks over several threads: batches below and above a
block of instances, and union slots with counts that fill no warp, one word past a block and one
instance. Byte identity with the oracle."""
import pytest

import flock_gb300
import oracle
from flock_gb300 import BLAKE3, KECCAK, SHA256, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,log_n", [(BLAKE3, 8), (SHA256, 7), (KECCAK, 6), (BLAKE3, 11), (SHA256, 11), (KECCAK, 9)])
def test_batch_matches_oracle(kind, log_n):
    recs = inputs.batch(kind, 1 << log_n, 40 + log_n)
    with flock_gb300.SETUPS[kind](1 << log_n) as s:
        assert s.prove_fast_bytes(recs, b"witness") == oracle.prove_fast_bytes(kind, recs, b"witness")


@pytest.mark.parametrize("counts", [[65, 1, 33], [1, 63, 128]])
def test_union_matches_oracle(counts):
    with flock_gb300.UnionSetup([BLAKE3, SHA256, KECCAK], 7) as u:
        recs = [inputs.batch(k, c, 5) for k, c in zip(u.slot_kinds, counts)]
        assert u.prove_bytes(counts, recs, b"w") == oracle.prove_union_bytes(u.slot_kinds, 7, counts, recs, b"w")
