"""Spaces whose orbital irreps are not closed under products: strings of the missing irreps have their classes too
(host enumeration, csrc/blocks.cu)."""
from itertools import combinations

import numpy as np
import pytest


def irrep(mask, orbsym):
    h = 0
    for p, x in enumerate(orbsym):
        if mask >> p & 1:
            h ^= x
    return h


@pytest.mark.parametrize("orbsym,sym", [([0, 1, 2, 0, 1], 0), ([0, 2, 5, 0, 2, 5], 0), ([0, 3, 5, 3], 0), ([1, 2, 1], 0),
                                        ([1, 2, 4, 1], 0), ([0, 1, 2, 2, 1], 1)])
def test_all_determinants_of_the_irrep(orbsym, sym):
    from forte2_gb300.ci_helpers import enumerate_blocks

    n = len(orbsym)
    strings = {k: [sum(1 << p for p in c) for c in combinations(range(n), k)] for k in range(n + 1)}
    for na in range(n + 1):
        for nb in range(n + 1):
            want = {(a, b) for a in strings[na] for b in strings[nb] if irrep(a, orbsym) ^ irrep(b, orbsym) == sym}
            e = enumerate_blocks(na, nb, sym, [orbsym], [], [])
            got = set()
            a0 = np.concatenate([[0], np.cumsum(np.bincount(e["alpha_class"], minlength=e["nirrep"]))])
            b0 = np.concatenate([[0], np.cumsum(np.bincount(e["beta_class"], minlength=e["nirrep"]))])
            for ca, cb, size, off, nia, nib in e["blocks"]:
                assert size == nia * nib
                got |= {(int(a), int(b)) for a in e["alpha"][a0[ca]:a0[ca] + nia] for b in e["beta"][b0[cb]:b0[cb] + nib]}
            assert got == want and e["ndet"] == len(want)


def test_number_of_irreps():
    from forte2_gb300.ci_helpers import enumerate_blocks

    for orbsym, count in (([0, 1], 2), ([0, 3], 4), ([0, 4], 5), ([0, 1, 2], 4), ([0, 2, 5], 8), ([0, 7], 8)):
        assert enumerate_blocks(1, 1, 0, [orbsym], [], [])["nirrep"] == count


@pytest.mark.gpu
@pytest.mark.parametrize("orbsym,na,nb", [([0, 1, 2, 0, 1, 2, 0, 1], 4, 4), ([0, 2, 5, 0, 2, 5, 0], 3, 4),
                                          ([0, 1, 2] * 4, 6, 6)])
def test_sigma_equals_that_of_the_whole_space(cuda, orbsym, na, nb):
    torch = cuda
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings
    from forte2_gb300.synthetic import make_integrals, random_ci_vector, symmetrize_integrals

    n = len(orbsym)
    ints = symmetrize_integrals(make_integrals(n, 6), orbsym)
    s, c1 = CIStrings(na, nb, 0, [orbsym], [], []), CIStrings(na, nb, 0, [[0] * n], [], [])
    place = {(int(a), int(b)): i for i, (a, b) in enumerate(np.asarray(c1.make_determinants().masks()))}
    at = np.array([place[int(a), int(b)] for a, b in np.asarray(s.make_determinants().masks())])
    x = random_ci_vector(s.ndet, 2)
    full = np.zeros(c1.ndet)
    full[at] = x
    out = []
    for strings, v in ((s, x), (c1, full)):
        sb = CISigmaBuilder(strings, ints.E, ints.H, ints.V, 0)
        d = torch.as_tensor(v, device="cuda")
        y = torch.empty_like(d)
        sb.Hamiltonian(d, y)
        out.append(y.cpu().numpy())
    assert np.linalg.norm(out[0] - out[1][at]) <= 1e-13 * np.linalg.norm(out[1])
    rest = np.delete(out[1], at)
    assert np.abs(rest).max(initial=0.0) <= 1e-13 * np.linalg.norm(out[1])
