"""Round messages, caps and openings published by the kernels into mapped host memory: provers of
different sizes and hashes on threads of their own, several bundles each (the flags and the opening
buffer are used again), byte for byte as the oracle's."""
from concurrent.futures import ThreadPoolExecutor

import pytest

import flock_gb300
import oracle
from flock_gb300 import BLAKE3, KECCAK, SHA256, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jobs", [[(BLAKE3, 8)], [(KECCAK, 6), (SHA256, 9), (BLAKE3, 11), (BLAKE3, 8)]])
def test_bundles_of_concurrent_provers_match_oracle(jobs):
    def run(job):
        kind, log_n = job
        with flock_gb300.SETUPS[kind](1 << log_n) as s:
            return [s.prove_fast_bytes(inputs.batch(kind, 1 << log_n, r), b"publish") for r in range(3)]

    with ThreadPoolExecutor(len(jobs)) as pool:
        got = list(pool.map(run, jobs))
    for (kind, log_n), bundles in zip(jobs, got):
        for r, b in enumerate(bundles):
            assert b == oracle.prove_fast_bytes(kind, inputs.batch(kind, 1 << log_n, r), b"publish")
