"""The device-byte estimate of a shape is arithmetic: it needs no device, and grows with the batch."""
import pytest

from flock_gb300 import BLAKE3, KECCAK, SHA256
from flock_gb300.serving import estimate_device_bytes


@pytest.mark.parametrize("kind", [BLAKE3, SHA256, KECCAK])
def test_estimate_grows_with_the_batch(kind):
    est = [estimate_device_bytes(kind, 1 << ln) for ln in (8, 12, 16, 18)]
    assert est == sorted(est) and est[0] > 100 << 20 and est[-1] > 2 * est[-2] - (1 << 30)
