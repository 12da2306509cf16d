"""The roofline's denominators (csrc/intpeak.cu): each rate is measured, and wider
products of the tensor cores do not compare fewer windows and patterns a second."""
import ctypes
import os

import pytest

pytestmark = pytest.mark.gpu
PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cas-offinder-rust-old_b200")


def test_rates(cof_mod):
    lib = ctypes.CDLL(os.path.join(PKG, "libcof_peak.so"))
    out = (ctypes.c_double * 6)()
    assert lib.cof_peak_products(0, out) == 0
    k64, k96 = list(out)[:3], list(out)[3:]
    for rates in (k64, k96):
        assert rates[0] > 1e12 and all(b > 0.95 * a for a, b in zip(rates, rates[1:]))
    assert all(b <= 1.05 * a for a, b in zip(k64, k96))
