"""The zerocheck's weighted rounds at the sizes where their chunk changes (none, 2^10, 2^11 and 2^12
words, with live words that end inside and at the end of a chunk), and a union's full-length
vectors; byte identity with the oracle."""
import pytest

import flock_gb300
import oracle
from flock_gb300 import BLAKE3, KECCAK, SHA256, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,log_n", [
    (BLAKE3, 10),   # 94208 live words: the plain form
    (BLAKE3, 11),   # 188416: chunks of 2^10, live words a whole number of them
    (KECCAK, 9),    # 170496: the last chunk half live
    (SHA256, 13),   # 1.6 M: chunks of 2^11
    (KECCAK, 13),   # 2.7 M: chunks of 2^12
])
def test_bundle_matches_oracle(kind, log_n):
    recs = inputs.batch(kind, 1 << log_n, 90 + log_n)
    with flock_gb300.SETUPS[kind](1 << log_n) as s:
        got = s.prove_fast_bytes(recs, b"weighted")
    assert got == oracle.prove_fast_bytes(kind, recs, b"weighted")


def test_union_bundle_matches_oracle():
    types, nu, counts = [SHA256, BLAKE3], 12, [3000, 4096]
    with flock_gb300.UnionSetup(types, nu) as u:
        recs = [inputs.batch(k, c, 7) for k, c in zip(u.slot_kinds, counts)]
        got = u.prove_bytes(counts, recs, b"weighted")
        assert got == oracle.prove_union_bytes(u.slot_kinds, nu, counts, recs, b"weighted")
