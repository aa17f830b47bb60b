"""FP64 digit sigma (csrc/oz.cu) against the FP64 multiply-add kernels element by element, on vectors over twenty decades and
with integrals of zero, within the stated bound.

Bound of a sigma element. Per product of a hole string (pair): 2^-55 of the largest coefficient of its row times the
largest integral of its output pair for each operand's cut, and 6 products of digits of 2^14 in the first group left out,
2^-53.4: 2^-52 in all. Per output of a hole string: its sum's last group is rounded (2^-55) and the sum aligned with
seven others', less three bits (2^-51 of the largest of them): 2^-50. The FP64 sums of both sides: at most 300 roundings
of 2^-53 of the sum of all absolute products."""
from itertools import combinations

import numpy as np
import pytest

from forte2_gb300.synthetic import make_integrals, random_ci_vector, symmetrize_integrals

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def strings(n, k):
    return [sum(1 << i for i in c) for c in combinations(range(n), k)]


def bounds(n, na, nb, a, b, E, h, V, c):
    """digit bound + rounding bound of every sigma element; a, b: masks of the strings in address order"""
    at = ({int(m): i for i, m in enumerate(a)}, {int(m): i for i, m in enumerate(b)})
    C = np.abs(c).reshape(len(a), len(b))
    cut, chain = np.zeros_like(C), np.zeros_like(C)
    largest, terms = np.zeros_like(C), na * nb
    vmax = np.abs(V).max(axis=(2, 3))
    for Ka in strings(n, na - 1):
        p = [o for o in range(n) if not Ka >> o & 1]
        ia = [at[0][Ka | 1 << o] for o in p]
        for Kb in strings(n, nb - 1):
            r = [o for o in range(n) if not Kb >> o & 1]
            ib = [at[1][Kb | 1 << o] for o in r]
            D = C[np.ix_(ia, ib)]
            big = D.max() * vmax[np.ix_(p, r)]
            cut[np.ix_(ia, ib)] += D.size * 2.0 ** -52 * big
            chain[np.ix_(ia, ib)] += np.einsum("prqs,qs->pr", np.abs(V[np.ix_(p, r, p, r)]), D)
            largest[np.ix_(ia, ib)] = np.maximum(largest[np.ix_(ia, ib)], big)
    cut += terms * 2.0 ** -50 * largest
    for spin, k in ((0, na), (1, nb)):
        M = C if spin == 0 else C.T
        mcut, mchain, mlarge = np.zeros_like(M), np.zeros_like(M), np.zeros_like(M)
        pairs = [(x, y) for x in range(n) for y in range(x)]
        one = np.zeros((n,) * 4)
        for x in range(n):
            one[:, x, :, x] += h
            one[:, x, x, :] -= h
            one[x, :, :, x] -= h
            one[x, :, x, :] += h
        g = np.abs(V - V.transpose(0, 1, 3, 2) + one / (k - 1))
        parts = np.abs(V) + np.abs(V.transpose(0, 1, 3, 2)) + np.abs(one) / (k - 1)
        X, Y = (np.array(z) for z in zip(*pairs))
        g, parts = g[X[:, None], Y[:, None], X, Y], parts[X[:, None], Y[:, None], X, Y]
        off = g - np.diag(np.diag(g))
        gmax = off.max(axis=1)
        for K in strings(n, k - 2):
            q = [i for i, (x, y) in enumerate(pairs) if not K >> x & 1 and not K >> y & 1]
            rows = [at[spin][K | 1 << pairs[i][0] | 1 << pairs[i][1]] for i in q]
            D = M[rows]
            big = gmax[q][:, None] * D.max(axis=0)
            mcut[rows] += len(q) * 2.0 ** -52 * big
            mchain[rows] += parts[np.ix_(q, q)] @ D
            mlarge[rows] = np.maximum(mlarge[rows], big)
        mcut += k * (k - 1) / 2 * 2.0 ** -50 * mlarge
        cut += mcut if spin == 0 else mcut.T
        chain += mchain if spin == 0 else mchain.T
    chain += abs(E) * C
    return cut, 300 * U * chain


@pytest.mark.parametrize("n,na,nb", [(6, 3, 3), (7, 3, 4), (8, 5, 2)])
@pytest.mark.parametrize("zeros", [False, True])
def test_every_element_within_its_bound(cuda, n, na, nb, zeros):
    torch = cuda
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings

    ints = make_integrals(n, 9)
    if zeros:  # a molecule with symmetry treated without it
        ints = symmetrize_integrals(ints, [(3 * p) % 4 for p in range(n)])
    s = CIStrings(na, nb, 0, [[0] * n], [], [])
    sb = CISigmaBuilder(s, 0.5, ints.H, ints.V, 0)
    a, b = s.alpha_masks(), s.beta_masks()
    rng = np.random.default_rng(n)
    c = random_ci_vector(s.ndet, 7)
    one = 1e-8 * c
    one[s.ndet // 3] = 1.0
    X = torch.as_tensor(np.stack([c, c * 10.0 ** rng.uniform(-20, 0, s.ndet), one]), device="cuda")
    out = {}
    for digits in (0, 1):
        sb.set_variant("digit_fp64", digits)
        y = torch.empty_like(X)
        sb.Hamiltonian(X, y)
        out[digits] = y.cpu().numpy()
    for x, plain, digit in zip(X.cpu().numpy(), out[0], out[1]):
        cut, chain = bounds(n, na, nb, a, b, 0.5, np.asarray(ints.H), np.asarray(ints.V), x)
        d = np.abs(plain - digit).reshape(cut.shape)
        assert (d <= cut + chain).all()
