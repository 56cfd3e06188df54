"""The product rates that the bench's roofline divides by. Products by a constant are fastest in the form
that the kernels' window tables have: by its lookups, 2.75 cycles of an SM's shared-memory pipe a table
product, three in four products at 152 SMs and 2070 MHz are 1.5e11 / s, against 4.87e10 by multiply alone.
Byte tables reach 1.66 times the multiply rate, so a peak measured with them stays below 1.9 times."""
import ctypes

import pytest

import flock_gb300

pytestmark = pytest.mark.gpu


def test_constant_products_beat_the_byte_tables():
    lib = flock_gb300.load()
    mul, mix = ctypes.c_double(), ctypes.c_double()
    flock_gb300._native.check(lib.flock_gb300_f128_mul_rate(256, ctypes.byref(mul)))
    flock_gb300._native.check(lib.flock_gb300_f128_table_mix_rate(256, ctypes.byref(mix)))
    assert mix.value > 1.9 * mul.value > 0
