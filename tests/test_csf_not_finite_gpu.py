"""Infinities and NaN in determinant vectors: only the CSFs that contain such a determinant are not finite,
in the tiles and in the kernel of large tables (csrc/csf.cu)."""
import numpy as np
import pytest

from forte2_gb300.synthetic import random_ci_vector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,na,nb", [(6, 3, 3), (8, 4, 4), (9, 5, 4), (10, 5, 5)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_det_to_csf(cuda, n, na, nb, bad):
    from forte2_gb300.ci_helpers import CISpinAdapter, CIStrings

    s = CIStrings(na, nb, 0, [[0] * n], [], [])
    sa = CISpinAdapter(na - nb, na - nb, n)
    sa.prepare_couplings(s)
    ncsf = sa.ncsf
    x = random_ci_vector(s.ndet, 2)
    ref = np.zeros(ncsf)
    sa.det_C_to_csf_C(x, ref)
    # determinants with a zero coefficient in some CSF of their configuration, with few and with many open shells
    bounds, dets, coeff, ranges = sa.couplings()
    chosen = {}
    for u0, u1 in ranges:
        per = [set(dets[bounds[u]:bounds[u + 1]][coeff[bounds[u]:bounds[u + 1]] != 0.0]) for u in range(u0, u1)]
        missing = set.union(*per) - set.intersection(*per) if per else set()
        if missing and len(set.union(*per)) not in chosen:
            chosen[len(set.union(*per))] = int(min(missing))
    assert chosen
    for at in [0, *chosen.values()]:
        y = x.copy()
        y[at] = bad
        got = np.zeros(ncsf)
        sa.det_C_to_csf_C(y, got)
        one = np.zeros(s.ndet)
        one[at] = 1.0
        member = np.zeros(ncsf)
        sa.det_C_to_csf_C(one, member)
        member = member != 0.0
        assert member.any() and not member.all()
        assert (np.isfinite(got) == ~member).all()
        assert (got[~member] == ref[~member]).all()
