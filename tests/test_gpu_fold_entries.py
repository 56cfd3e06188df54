"""The table fold with a thread on two entries and a trade between neighbouring lanes: live lengths that
end inside a warp's 64 entries and at an odd one (ragged unions), and whole ones. Byte identity
with the oracle."""
import pytest

import flock_gb300
import oracle
from flock_gb300 import BLAKE3, KECCAK, SHA256, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types,nu,counts", [([KECCAK, BLAKE3], 11, [2047, 1001]), ([SHA256, BLAKE3], 11, [2047, 2046])])
def test_union_matches_oracle(types, nu, counts):
    with flock_gb300.UnionSetup(types, nu) as u:
        recs = [inputs.batch(k, c, 9) for k, c in zip(u.slot_kinds, counts)]
        assert u.prove_bytes(counts, recs, b"f") == oracle.prove_union_bytes(u.slot_kinds, nu, counts, recs, b"f")


@pytest.mark.parametrize("kind,log_n", [(KECCAK, 11), (SHA256, 12)])
def test_bundle_matches_oracle(kind, log_n):
    recs = inputs.batch(kind, 1 << log_n, 70 + log_n)
    with flock_gb300.SETUPS[kind](1 << log_n) as s:
        assert s.prove_fast_bytes(recs, b"entries") == oracle.prove_fast_bytes(kind, recs, b"entries")
