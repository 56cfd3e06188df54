"""Zerocheck round 1 on bit planes: fewer xo than SMs, a last xo that is partly live, several xo a
warp, a union's full-length vectors; byte identity with the oracle."""
import pytest

import flock_gb300
import oracle
from flock_gb300 import BLAKE3, KECCAK, SHA256, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,log_n", [(KECCAK, 6), (SHA256, 7), (SHA256, 8), (KECCAK, 9), (BLAKE3, 13)])
def test_bundle_matches_oracle(kind, log_n):
    recs = inputs.batch(kind, 1 << log_n, 60 + log_n)
    with flock_gb300.SETUPS[kind](1 << log_n) as s:
        assert s.prove_fast_bytes(recs, b"round1") == oracle.prove_fast_bytes(kind, recs, b"round1")


def test_union_bundle_matches_oracle():
    types, nu, counts = [KECCAK, SHA256, BLAKE3], 5, [31, 32, 9]
    with flock_gb300.UnionSetup(types, nu) as u:
        recs = [inputs.batch(k, c, 8) for k, c in zip(u.slot_kinds, counts)]
        assert u.prove_bytes(counts, recs, b"r1") == oracle.prove_union_bytes(u.slot_kinds, nu, counts, recs, b"r1")
