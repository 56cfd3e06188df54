"""The bit-sum kernel's plans: the fewest row tiles, columns that leave warps and column slots
empty, one and several column groups; byte identity with the oracle (s_hat_v_c, the lincheck's row
fold and Ligerito's lane dots all come from it)."""
import pytest

import flock_gb300
import oracle
from flock_gb300 import BLAKE3, KECCAK, SHA256, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types,nu,counts", [
    ([KECCAK, SHA256], 6, [3, 64]),           # two tiles of instances
    ([KECCAK, SHA256, BLAKE3], 5, [32, 7, 1]),  # one tile (the smallest union), 1024 union columns
])
def test_union_bundle_matches_oracle(types, nu, counts):
    with flock_gb300.UnionSetup(types, nu) as u:
        recs = [inputs.batch(k, c, 11 + c) for k, c in zip(u.slot_kinds, counts)]
        got = u.prove_bytes(counts, recs, b"bits")
        assert got == oracle.prove_union_bytes(u.slot_kinds, nu, counts, recs, b"bits")


@pytest.mark.parametrize("kind,log_n", [(BLAKE3, 8), (SHA256, 11), (KECCAK, 12)])
def test_bundle_matches_oracle(kind, log_n):
    recs = inputs.batch(kind, 1 << log_n, 50 + log_n)
    with flock_gb300.SETUPS[kind](1 << log_n) as s:
        got = s.prove_fast_bytes(recs, b"bits")
    assert got == oracle.prove_fast_bytes(kind, recs, b"bits")
