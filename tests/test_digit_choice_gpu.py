"""The digit_fp64 variant as the caller's choice between the digit kernels (FP64 accuracy in the norm of a row) and the
FP64 multiply-add kernels (FP64 accuracy element by element): sigma of C1 and of blocked spaces, density matrices."""
from itertools import combinations

import numpy as np
import pytest

from forte2_gb300.batch import uses_digits
from forte2_gb300.synthetic import make_integrals, random_ci_vector, symmetrize_integrals
from test_rdm_gram_gpu import gram, kinds, strings

pytestmark = pytest.mark.gpu


def builder(n, na, nb, irreps=None):
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings

    ints = make_integrals(n, 4)
    if irreps is not None:
        ints = symmetrize_integrals(ints, irreps)
    s = CIStrings(na, nb, 0, [[0] * n if irreps is None else irreps], [], [])
    return s, CISigmaBuilder(s, ints.E, ints.H, ints.V, 0)


@pytest.mark.parametrize("n,na,nb,irreps", [
    (10, 5, 5, None), (12, 6, 6, [0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3])])
def test_small_elements_of_sigma(cuda, n, na, nb, irreps):
    torch = cuda
    s, sb = builder(n, na, nb, irreps)
    at = s.ndet // 3
    x = 1e-30 * random_ci_vector(s.ndet, 3)
    zero = x.copy()
    x[at], zero[at] = 1.0, 0.0
    X = torch.as_tensor(np.stack([x, zero]), device="cuda")

    def apply():
        out = torch.empty_like(X)
        sb.Hamiltonian(X, out)
        return out

    det = np.asarray(s.make_determinants().masks())
    away = sum(np.array([bin(int(m)).count("1") for m in det[:, k] ^ det[at, k]]) for k in (0, 1)) > 4
    away = torch.as_tensor(away, device="cuda")
    default = apply()
    sb.set_variant("digit_fp64", 0)
    plain = apply()
    # more than two excitations away sigma is a sum over the small elements: the same with and without the large one
    assert torch.equal(plain[0][away], plain[1][away])
    assert torch.linalg.vector_norm(plain[0] - default[0]) <= 1e-13 * torch.linalg.vector_norm(plain[0])
    sb.set_variant("digit_fp64", 2)
    assert torch.equal(apply(), default)


@pytest.mark.parametrize("n,na,nb,digits", [(4, 2, 2, 0), (6, 4, 3, 0), (8, 3, 2, 0), (9, 4, 4, 0), (8, 1, 8, 0),
                                            (4, 2, 2, 1), (5, 4, 2, 1), (8, 7, 2, 1),  # too small to gain
                                            (6, 5, 2, 2), (7, 6, 3, 2), (8, 8, 3, 2)])  # by block
def test_density_matrices(cuda, n, na, nb, digits):
    s, sb = builder(n, na, nb)
    sb.set_variant("digit_fp64", digits)
    x, y = random_ci_vector(s.ndet, 1), random_ci_vector(s.ndet, 2)
    for kind, (spin, h, inner) in kinds(n, na, nb).items():
        k, kin = (na, nb) if spin == 0 else (nb, na)
        if k < h or (inner and kin < 1):
            continue

        def shape(v):
            return v.reshape(len(strings(n, na)), -1) if spin == 0 else v.reshape(len(strings(n, na)), -1).T

        for a, b in ((x, x), (x, y)):
            ref = gram(n, k, h, kin if inner else None, shape(a), shape(b))
            got = np.asarray(getattr(sb, kind)(a, b))
            D = len(list(combinations(range(n), h)))
            if kind == "abb_3rdm":
                got = got.reshape(n, D, n, D).transpose(1, 0, 3, 2)
            # sums of at most some thousand products in FP64
            tol = 1e-13 * np.linalg.norm(a) * np.linalg.norm(b)
            assert np.abs(got.reshape(ref.shape) - ref).max(initial=0.0) <= tol, kind


def test_a_kept_solver_captures_its_iterations_again(cuda):
    from forte2_gb300.ci import CASCISolver
    from forte2_gb300.params import CIParams, DavidsonLiuParams

    ints = make_integrals(10, 11)
    solver = CASCISolver(norb=10, na=5, nb=5, multiplicity=1, nroot=1, E=ints.E, H=ints.H, V=ints.V,
                         ci_params=CIParams(), davidson_liu_params=DavidsonLiuParams(e_tol=1e-10, maxiter=200))
    solver.run()
    first = float(solver.evals[0])
    solver.sigma_variants = {"digit_fp64": 0}
    solver.new_problem(ints.E, ints.H, ints.V)
    solver.run()
    assert len(solver.eigensolver._graphs) == 2
    assert abs(float(solver.evals[0]) - first) < 1e-9


@pytest.mark.parametrize("n,na,nb,fast", [(11, 2, 8, False), (12, 2, 9, True), (14, 2, 12, False), (13, 10, 11, False),
                                          (14, 3, 12, True), (10, 4, 8, True), (12, 11, 7, True)])
def test_default_kernels_of_spaces_with_few_beta_holes(cuda, n, na, nb, fast):
    torch = cuda
    s, sb = builder(n, na, nb)
    c = torch.as_tensor(random_ci_vector(s.ndet, 3), device="cuda")
    got = {}
    for digits in (2, 0, 1):
        sb.set_variant("digit_fp64", digits)
        got[digits] = torch.empty_like(c)
        sb.Hamiltonian(c, got[digits])
    assert torch.equal(got[2], got[1 if fast else 0])
    assert uses_digits(n, na, nb) == fast
    assert torch.linalg.vector_norm(got[1] - got[0]) <= 1e-13 * torch.linalg.vector_norm(got[0])
