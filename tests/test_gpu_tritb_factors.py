"""A block-cycle hierarchy pays for the zebra order's factors only when it takes
that order, and once."""
from __future__ import annotations

import numpy as np
import pytest

from asam_gb300 import TriTBHierarchy

pytestmark = pytest.mark.gpu

COEFS = dict(beta0_dtp=0.5, fac1_l=1.0, fac1_r=1.0, grav_comp=1.0, fac_anela=0.25, fac2_l=1.0, fac2_r=1.0, fac3_l=1.0,
             fac3_r=1.0)


def _hierarchy(n3, n2, n1, ref_level):
    rng = np.random.default_rng(1)

    def field(*shape):
        return rng.uniform(0.2, 2.0, shape)

    return TriTBHierarchy([field(n3, n2, n1 + 1) for _ in range(4)], [field(n3, n2 + 1, n1) for _ in range(4)],
                          [field(n3 + 1, n2, n1) for _ in range(4)], field(n3, n2, n1), field(n3, n2, n1), None,
                          ref_level=ref_level, **COEFS)


def _entries(n3, n2, n1, ref_level):
    half = lambda n, l: -(-n // 2 ** l)  # noqa: E731
    return [(half(n3, a), half(n2, b), half(n1, b)) for a in range(ref_level) for b in range(a, ref_level)]


@pytest.mark.parametrize("shape,ref_level", [((1, 1, 1), 1), ((5, 9, 7), 3)])
def test_factors_on_first_use(built_lib, shape, ref_level):
    levels = len(_entries(*shape, ref_level))
    rng = np.random.default_rng(2)
    b = rng.standard_normal(shape + (2,))
    count = lambda h: h.lib.asam_launch_count()  # noqa: E731
    with _hierarchy(*shape, ref_level) as h:  # the library is loaded
        n0 = count(h)
    with _hierarchy(*shape, ref_level) as h:
        assert count(h) - n0 == 3 * levels
        n0 = count(h)
        h.set_zebra(False)
        assert count(h) == n0
        first = h.vcycle(b)
        n0 = count(h)
        h.set_zebra(True)
        assert count(h) - n0 == levels
        zebra = h.vcycle(b)
        n0 = count(h)
        h.set_zebra(False)
        np.testing.assert_array_equal(h.vcycle(b), first)
        h.set_zebra(True)
        np.testing.assert_array_equal(h.vcycle(b), zebra)
        with _hierarchy(*shape, ref_level) as other:
            other.set_zebra(True)
            np.testing.assert_array_equal(other.vcycle(b), zebra)


def test_memory_of_the_sequential_order(built_lib):
    torch = pytest.importorskip("torch")
    shape, ref_level = (48, 96, 80), 4
    with _hierarchy(2, 2, 2, 1):
        pass
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    with _hierarchy(*shape, ref_level) as h:
        used = free0 - torch.cuda.mem_get_info()[0]
        # per entry five 2x2 blocks and three vectors of two; couplings of 2x2 blocks between the planes of a level
        n = [a * b * c for a, b, c in _entries(*shape, ref_level)]
        own = [a * b * c for a, b, c in ((48, 96, 80), (24, 48, 40), (12, 24, 20), (6, 12, 10))]
        assert used <= 8 * (26 * sum(n) + 8 * sum(own)) + (8 << 20)
        h.set_zebra(True)
        more = free0 - torch.cuda.mem_get_info()[0] - used
        assert more >= 8 * 14 * sum(n) - (8 << 20)
