"""The tensor-core Gram kernel of the RDMs (csrc/rdm_gram.cu) against FP64 Gram matrices of numpy at
the edges of its tiles: 16 to 128 slots, two tiles (their off-diagonal pair included), one row of the
other spin, partial K steps, one vector (shared operands) and two, rows of very different scale.

Tolerance: 1e-13 of the product of the vectors' norms. The digits drop parts below 2^-62 of a row's
largest element and products below 2^-63, at most sqrt(rows) 2^-60 of the norms; the sums are exact
per hole string and added in FP64 as a tree (2^-53 a step, at most 130 steps)."""

from itertools import combinations

import numpy as np
import pytest

from forte2_gb300.synthetic import make_integrals, random_ci_vector

pytestmark = pytest.mark.gpu


def strings(n, k):
    return [sum(1 << i for i in c) for c in combinations(range(n), k)][::-1]


def holes(n, k, h):
    """for every string K of k - h electrons: (set index, address of K + set, sign)"""
    at = {m: i for i, m in enumerate(strings(n, k))}
    sets = [sum(1 << i for i in c) for c in sorted(combinations(range(n), h), key=lambda c: c[::-1])]
    out = []
    for K in strings(n, k - h):
        row = []
        for o, s in enumerate(sets):
            if not K & s:
                par = sum(bin(K & ((1 << i) - 1)).count("1") for i in range(n) if s >> i & 1)
                row.append((o, at[K | s], -1.0 if par & 1 else 1.0))
        out.append(row)
    return out, len(sets)


def gram(n, k, h, kin, X, Y):
    """sum_K sum_R of the outer strings' h holes and (kin electrons) the inner strings' one hole"""
    outer, D = holes(n, k, h)
    inner, E = holes(n, kin, 1) if kin is not None else (None, 1)
    g = np.zeros((D * E, D * E))
    if inner:
        r, v, J, t = (np.array(c) for c in zip(*((r, *e) for r, R in enumerate(inner) for e in R)))

    def rows(M, K):
        d = np.zeros((len(inner) if inner else M.shape[1], D, E))
        for o, I, s in K:
            if inner:
                d[r, o, v] = s * t * M[I, J]
            else:
                d[:, o, 0] = s * M[I]
        return d.reshape(len(d), D * E)

    for K in outer:
        g += rows(X, K).T @ rows(Y, K)
    return g


def kinds(n, na, nb):
    """kind -> (outer spin, holes, inner spin's hole)"""
    out = {"ab_2rdm": (0, 1, True), "aa_2rdm": (0, 2, False), "bb_2rdm": (1, 2, False), "a_1rdm": (0, 1, False)}
    if n <= 9:
        out.update({"aab_3rdm": (0, 2, True), "abb_3rdm": (1, 2, True), "aaa_3rdm": (0, 3, False)})
    return out


@pytest.mark.parametrize("n,na,nb", [
    (2, 1, 1),   # one row, four slots
    (4, 2, 2),   # 12 slots: eight digits in one tile
    (6, 4, 3),   # 18
    (8, 3, 2),   # 48; 3-RDMs in two tiles
    (9, 4, 4),   # 54; 189 slots
    (9, 2, 5),   # 72: one digit per tile
    (12, 4, 2),  # 108; 45 pairs
    (8, 1, 8),   # 64; the other spin full
    (13, 3, 2),  # 143: two tiles of 80
    (16, 1, 3),  # 256: two tiles of 128
    (14, 1, 7),  # 1-RDM rows of 3,432
])
def test_gram_edges(cuda, n, na, nb):
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings

    ints = make_integrals(n, 3)
    s = CIStrings(na, nb, 0, [[0] * n], [], [])
    sb = CISigmaBuilder(s, ints.E, ints.H, ints.V, 0)
    x, y = random_ci_vector(s.ndet, 1), random_ci_vector(s.ndet, 2)
    y = y * 10.0 ** (-8 * np.random.default_rng(5).random(y.size))  # rows of mixed scale
    for kind, (spin, h, inner) in kinds(n, na, nb).items():
        k, kin = (na, nb) if spin == 0 else (nb, na)
        if k < h or (inner and kin < 1):
            continue
        def shape(v):
            return v.reshape(len(strings(n, na)), -1) if spin == 0 else v.reshape(len(strings(n, na)), -1).T

        tiny = y * 2.0 ** -480
        for a, b, scale in ((x, x, 1.0), (x, y, 1.0), (tiny, tiny, 2.0 ** 480)):
            ref = gram(n, k, h, kin if inner else None, shape(a * scale), shape(b * scale))
            got = np.asarray(getattr(sb, kind)(a, b))
            D = len(list(combinations(range(n), h)))
            if kind == "abb_3rdm":  # [p][Q][s][T]: the outer (beta) pairs are the faster index
                got = got.reshape(n, D, n, D).transpose(1, 0, 3, 2)
            got = got.reshape(ref.shape) * scale * scale
            tol = 1e-13 * np.linalg.norm(a * scale) * np.linalg.norm(b * scale)
            assert np.abs(got - ref).max(initial=0.0) <= tol, (kind, scale)
    assert sb.tensor_core_error() == 0


def test_gram_not_a_number(cuda):
    """a vector with a NaN or an infinity gives results that say so"""
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings

    n = 6
    ints = make_integrals(n, 3)
    s = CIStrings(3, 3, 0, [[0] * n], [], [])
    sb = CISigmaBuilder(s, ints.E, ints.H, ints.V, 0)
    for bad in (np.nan, np.inf):
        x = random_ci_vector(s.ndet, 1)
        x[7] = bad
        g = np.asarray(sb.ab_2rdm(x, x))
        assert not np.isfinite(g).all()
