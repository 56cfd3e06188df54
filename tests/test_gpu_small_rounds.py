"""Small sumcheck rounds (one product per thread): rounds of one block with idle pairs, of several
blocks, and with a zero tail that ends inside a block; the trees above these codewords take one to
three fused levels. Byte identity with the oracle."""
import pytest

import flock_gb300
import oracle
from flock_gb300 import BLAKE3, KECCAK, SHA256, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,log_n", [(KECCAK, 6), (SHA256, 7), (BLAKE3, 9), (SHA256, 10), (BLAKE3, 10)])
def test_bundle_matches_oracle(kind, log_n):
    recs = inputs.batch(kind, 1 << log_n, 20 + log_n)
    with flock_gb300.SETUPS[kind](1 << log_n) as s:
        for dom in (b"small", b"rounds"):
            assert s.prove_fast_bytes(recs, dom) == oracle.prove_fast_bytes(kind, recs, dom)


def test_union_bundle_matches_oracle():
    types, nu, counts = [KECCAK, BLAKE3], 7, [77, 1]
    with flock_gb300.UnionSetup(types, nu) as u:
        recs = [inputs.batch(k, c, 3) for k, c in zip(u.slot_kinds, counts)]
        assert u.prove_bytes(counts, recs, b"s") == oracle.prove_union_bytes(u.slot_kinds, nu, counts, recs, b"s")
