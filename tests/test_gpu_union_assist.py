"""Union proofs whose jagged multipoint assist runs on the device: areas of every residue mod 4
(a fold reads four entries together, some past the area), one slot with a single row, an empty slot between two
others, and a size whose fold rounds start in the byte-table form; byte identity with the
oracle."""
import pytest

import flock_gb300
import oracle
from flock_gb300 import BLAKE3, KECCAK, SHA256, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types,nu,counts", [
    ([KECCAK], 6, [1]),                              # 333 words: 1 mod 4
    ([SHA256], 8, [3]),                              # 597: 1 mod 4, odd height
    ([SHA256, BLAKE3], 7, [2, 127]),                 # 2 mod 4
    ([KECCAK, SHA256], 7, [1, 2]),                   # 731: 3 mod 4
    ([KECCAK, SHA256, BLAKE3], 6, [64, 0, 64]),      # full slots around an empty one
    ([KECCAK, SHA256, BLAKE3], 11, [1500, 777, 2048]),  # 2^20 dense words
])
def test_union_bundle_matches_oracle(types, nu, counts):
    with flock_gb300.UnionSetup(types, nu) as u:
        recs = [inputs.batch(k, max(c, 1), 40 + i)[:c] for i, (k, c) in enumerate(zip(u.slot_kinds, counts))]
        want = oracle.prove_union_bytes(u.slot_kinds, nu, counts, recs, b"assist")
        assert u.prove_bytes(counts, recs, b"assist") == want
        assert u.prove_bytes(counts, recs, b"assist") == want
