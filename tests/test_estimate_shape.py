"""The device-byte estimate has at least the buffers whose sizes follow from the shape alone: the witness
vectors, the codeword at rate 1/2, the zerocheck's and the merged open's fold vectors."""
import pytest

from flock_gb300 import BLAKE3, KECCAK, SHA256
from flock_gb300.serving import estimate_device_bytes

K_LOG = {BLAKE3: 14, SHA256: 15, KECCAK: 16}      # log2 of a block's bits
USED_COLS = {BLAKE3: 92, SHA256: 199, KECCAK: 333}  # of its 128-bit columns


@pytest.mark.parametrize("kind", [BLAKE3, SHA256, KECCAK])
@pytest.mark.parametrize("log_n", [8, 13, 18])
def test_estimate_covers_the_shape(kind, log_n):
    words = 1 << (K_LOG[kind] + log_n - 7)
    dense = USED_COLS[kind] << log_n
    vectors = 3 * words + 3 * words + 5 * words // 2  # z, a, b; zerocheck folds; weight and merged folds
    least = 16 * (vectors + 2 * dense)
    estimate = estimate_device_bytes(kind, 1 << log_n)
    assert least + (120 << 20) <= estimate <= 2 * least + (400 << 20)
