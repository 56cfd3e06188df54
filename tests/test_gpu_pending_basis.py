"""The pending eq basis of an out-of-domain point (stored without its first coordinate): levels whose
pairs fit a block's part, one block and many blocks, and the one that takes its factors from
tables; the merged-open weight from column tables at its shortest columns. Byte identity with the oracle."""
import pytest

import flock_gb300
import oracle
from flock_gb300 import BLAKE3, KECCAK, SHA256, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,log_n", [(BLAKE3, 8), (KECCAK, 10), (SHA256, 11), (BLAKE3, 14), (SHA256, 15)])
def test_bundle_matches_oracle(kind, log_n):
    recs = inputs.batch(kind, 1 << log_n, 60 + log_n)
    with flock_gb300.SETUPS[kind](1 << log_n) as s:
        assert s.prove_fast_bytes(recs, b"pending") == oracle.prove_fast_bytes(kind, recs, b"pending")
