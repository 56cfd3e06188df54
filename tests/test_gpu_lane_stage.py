"""Ligerito's lane stage at the shapes where it changes form: four, five and six lane variables
(m = 28, 29 and the rest), lane dots with and without window tables (rows below and from 2^16),
a row count of one short block; byte identity with the oracle."""
import pytest

import flock_gb300
import oracle
from flock_gb300 import BLAKE3, KECCAK, SHA256, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,log_n", [
    (KECCAK, 6),    # 2^9 rows: the smallest, a sixth of a fold block
    (BLAKE3, 13),   # 2^14 rows, six lane variables, lane dots without tables
    (SHA256, 13),   # 2^17 rows, four lane variables, 13 lanes, window tables
    (SHA256, 14),   # 2^17 rows, five lane variables, 25 lanes
])
def test_bundle_matches_oracle(kind, log_n):
    recs = inputs.batch(kind, 1 << log_n, 70 + log_n)
    with flock_gb300.SETUPS[kind](1 << log_n) as s:
        got = [s.prove_fast_bytes(recs, b"lanes") for _ in range(2)]
    want = oracle.prove_fast_bytes(kind, recs, b"lanes")
    assert got[0] == want and got[1] == want
