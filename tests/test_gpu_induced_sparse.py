"""The induced basis's directly formed layers at level sizes above the fused ones (2^17 and 2^18
positions), where several queries share a block; byte identity with the oracle."""
import pytest

import flock_gb300
import oracle
from flock_gb300 import BLAKE3, KECCAK, SHA256, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,log_n", [(BLAKE3, 14), (KECCAK, 12), (SHA256, 15)])
def test_bundle_matches_oracle(kind, log_n):
    recs = inputs.batch(kind, 1 << log_n, 80 + log_n)
    with flock_gb300.SETUPS[kind](1 << log_n) as s:
        assert s.prove_fast_bytes(recs, b"induced") == oracle.prove_fast_bytes(kind, recs, b"induced")
