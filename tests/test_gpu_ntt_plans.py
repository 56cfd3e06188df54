"""Codeword transforms over the pass plans: fused passes of every depth the committed sizes use,
byte-table and window-table passes and the sizes between them; byte identity with the oracle
(the bundle opens rows of the transform and of every level's)."""
import pytest

import flock_gb300
import oracle
from flock_gb300 import BLAKE3, KECCAK, SHA256, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,log_n", [
    (SHA256, 7),   # 9 layers: fused 5 + 4
    (KECCAK, 7),   # 10: 5 + 5
    (SHA256, 9),   # 11: 6 + 5
    (BLAKE3, 11),  # 12: 6 + 6
    (BLAKE3, 12),  # 13: 5 + 4 + 4
    (BLAKE3, 14),  # 2^17 positions, 12 lanes: window, then byte tables, then fused
    (BLAKE3, 15),  # 23 lanes
])
def test_bundle_matches_oracle(kind, log_n):
    recs = inputs.batch(kind, 1 << log_n, 30 + log_n)
    with flock_gb300.SETUPS[kind](1 << log_n) as s:
        got = s.prove_fast_bytes(recs, b"ntt")
    assert got == oracle.prove_fast_bytes(kind, recs, b"ntt")
