"""The correctly rounded product and quotient of the integer units equal the
IEEE ones on random pairs and on special operands (asam_probe_div)."""
from __future__ import annotations

import ctypes as C

import pytest

from asam_gb300 import _lib

pytestmark = pytest.mark.gpu


# 0: significands only; 479-500: products and quotients around the ends of the
# exponent range the integer path takes
@pytest.mark.parametrize("span", [0, 1, 240, 479, 481, 500])
def test_products_and_quotients_bitwise(built_lib, span):
    bad = C.c_longlong(-1)
    _lib.check(_lib.load().asam_probe_div(40_000_000, 77 + span, span, C.byref(bad)), "asam_probe_div")
    assert bad.value == 0
