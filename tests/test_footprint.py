"""The memory estimate of a solve counts the FP64 tensor-core sigma's buffers where that kernel runs and nowhere else
(the exactness bound of its digit sums, csrc/oz.cu: oz_lead)."""
from math import comb

import pytest

from forte2_gb300.batch import footprint_bytes


def without_digits(n, na, nb, nroot):
    return footprint_bytes(n + 1, na, nb, nroot)  # 17 orbitals and more: no digits, and larger in everything else


@pytest.mark.parametrize("na,nb", [(4, 4), (5, 3), (6, 3), (4, 3)])
def test_spaces_with_too_many_holes(na, nb):
    assert (16 - na + 1) * (16 - nb + 1) > 146
    assert footprint_bytes(16, na, nb, 1) < without_digits(16, na, nb, 1)


@pytest.mark.parametrize("n,na,nb", [(14, 7, 7), (16, 8, 8), (13, 6, 5)])
def test_spaces_on_the_digits(n, na, nb):
    elements = comb(n, na - 1) * comb(n, nb - 1) * (n - na + 1) * (n - nb + 1)
    lower = 2 * min(8 * elements, 2 << 30)  # E of one vector, both sets
    plain = 8 * comb(n, na) * comb(n, nb)
    assert footprint_bytes(n, na, nb, 1) > lower + plain
