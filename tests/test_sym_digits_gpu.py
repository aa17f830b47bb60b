"""The tensor-core opposite-spin sigma of point-group-blocked spaces (csrc/sym_digits.cu) against the
C1 kernel on the embedding: 16 to 64 orbital pairs per hole pair, more than 64 (left to the FP64
kernel), tiles of 128 strings with a remainder, unequal electrons, several vectors, vectors of very
different scale, and solves in captured graphs.

Tolerance: 1e-13 of the result's norm, as for the FP64 kernel in test_blocks_gpu.py. The digits drop
parts below 2^-62 of the largest element of vector and integrals; an element of E is rounded once and
at most n^2 of them are added in FP64."""

import numpy as np
import pytest

from forte2_gb300.synthetic import make_integrals, random_ci_vector, symmetrize_integrals

pytestmark = pytest.mark.gpu

SPACES = [
    (5, 5, 0, [0, 1] * 5),                       # 30 pairs
    (6, 6, 5, [0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3]),  # 14 pairs
    (7, 5, 1, [0, 1, 2, 3] * 3),                 # 18 pairs
    (6, 5, 0, [0] * 9 + [1] * 3),                # 54 to 64 pairs
    (4, 4, 1, [0] * 9 + [1] * 3),                # 72 pairs and more: the FP64 kernel
    (6, 6, 3, [0, 1, 2, 3, 4, 5, 6, 7, 0, 3, 5, 6, 6]),
]


def builder(na, nb, sym, orbsym, symmetric=True):
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings

    ints = make_integrals(len(orbsym), 40 + len(orbsym))
    if symmetric:
        ints = symmetrize_integrals(ints, orbsym)
    s = CIStrings(na, nb, sym, [orbsym], [], [])
    return s, CISigmaBuilder(s, ints.E, ints.H, ints.V, 0)


@pytest.mark.parametrize("na,nb,sym,orbsym", SPACES)
def test_blocked_sigma_equals_c1(cuda, na, nb, sym, orbsym):
    torch = cuda
    s, sb = builder(na, nb, sym, orbsym, symmetric=na != nb)
    rng = np.random.default_rng(3)
    x = np.stack([random_ci_vector(s.ndet, 1), random_ci_vector(s.ndet, 2) * 10.0 ** (-9 * rng.random(s.ndet)),
                  random_ci_vector(s.ndet, 3) * 2.0 ** -400])
    X = torch.as_tensor(x, device="cuda")
    got, ref = torch.empty_like(X), torch.empty_like(X)
    sb.Hamiltonian(X, got)
    sb.set_variant("irrep_blocks", 0)
    sb.Hamiltonian(X, ref)
    scale = torch.tensor([1.0, 1.0, 2.0 ** 400], dtype=torch.float64, device="cuda")[:, None]
    got, ref = got * scale, ref * scale
    assert (torch.linalg.vector_norm(got - ref, dim=1) < 1e-13 * torch.linalg.vector_norm(ref, dim=1)).all()
    assert sb.tensor_core_error() == 0


def test_blocked_sigma_not_a_number(cuda):
    torch = cuda
    s, sb = builder(6, 6, 5, [0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3])
    x = torch.as_tensor(random_ci_vector(s.ndet, 1), device="cuda")
    x[11] = float("inf")
    out = torch.empty_like(x)
    sb.Hamiltonian(x, out)
    assert not torch.isfinite(out).all()


def test_blocked_solve_in_graphs(cuda):
    from forte2_gb300.ci import CASCISolver
    from forte2_gb300.params import DavidsonLiuParams

    orbsym = [0, 1] * 5
    ints = symmetrize_integrals(make_integrals(10, 50), orbsym)
    e = []
    for graph in (False, True):
        sol = CASCISolver(norb=10, na=5, nb=5, multiplicity=1, nroot=2, E=ints.E, H=ints.H, V=ints.V, symmetry=0,
                          orbital_symmetry=[orbsym], gas_min=[], gas_max=[], use_graph=graph,
                          davidson_liu_params=DavidsonLiuParams(e_tol=1e-12, maxiter=400)).run()
        assert sol.converged
        e.append(np.asarray(sol.evals))
    assert np.abs(e[0] - e[1]).max() < 1e-10
