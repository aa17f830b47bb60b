"""The digit kernels with work buffers so small that they run in parts: ranges of alpha hole strings and steps of tiles
(csrc/oz.cu), parts of positions and of alpha hole strings (csrc/sym_digits.cu), parts of the other spin's strings
(csrc/rdm_gram.cu), each with a remainder."""
import numpy as np
import pytest

from forte2_gb300.synthetic import make_integrals, random_ci_vector, symmetrize_integrals

pytestmark = pytest.mark.gpu


def builder(n, na, nb, irreps=None):
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings

    ints = make_integrals(n, 4)
    if irreps is not None:
        ints = symmetrize_integrals(ints, irreps)
    s = CIStrings(na, nb, 0, [[0] * n if irreps is None else irreps], [], [])
    return s, CISigmaBuilder(s, ints.E, ints.H, ints.V, 0)


@pytest.mark.parametrize("n,na,nb", [(8, 4, 4), (11, 4, 6), (12, 6, 6)])
def test_sigma_in_parts_has_the_same_bits(cuda, n, na, nb):
    torch = cuda
    s, sb = builder(n, na, nb)
    sb.set_variant("digit_fp64", 1)
    X = torch.as_tensor(np.stack([random_ci_vector(s.ndet, v) for v in range(3)]), device="cuda")

    def apply():
        out = torch.full_like(X, float("nan"))
        sb.Hamiltonian(X, out)
        return out

    whole = apply()
    for size in (1, 1_500_000, 7_000_000):  # one hole string and one tile at a time; some of them
        sb.set_variant("digit_buffer_bytes", size)
        # every element is summed over its alpha hole strings in one order, whatever parts they come in
        assert torch.equal(apply(), whole), size
    sb.set_variant("digit_buffer_bytes", 0)
    assert torch.equal(apply(), whole)
    assert sb.tensor_core_error() == 0


@pytest.mark.parametrize("irreps,na,nb", [([0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3], 6, 6), ([0, 1] * 6, 5, 6)])
def test_blocked_sigma_in_parts(cuda, irreps, na, nb):
    torch = cuda
    n = len(irreps)
    s, sb = builder(n, na, nb, irreps)
    X = torch.as_tensor(np.stack([random_ci_vector(s.ndet, v) for v in range(2)]), device="cuda")

    def apply():
        out = torch.full_like(X, float("nan"))
        sb.Hamiltonian(X, out)
        return out

    whole = apply()
    sb.set_variant("irrep_blocks", 0)
    plain = apply()
    sb.set_variant("irrep_blocks", 1)
    for size in (1, 3_000_000, 40_000_000):
        sb.set_variant("digit_buffer_bytes", size)
        out = apply()
        assert (torch.linalg.vector_norm(out - plain, dim=1) < 1e-13 * torch.linalg.vector_norm(plain, dim=1)).all(), size
        assert torch.equal(out, apply())
    sb.set_variant("digit_buffer_bytes", 0)
    assert torch.equal(apply(), whole)
    assert sb.tensor_core_error() == 0


@pytest.mark.parametrize("n,na,nb", [(9, 4, 4), (11, 5, 6), (14, 1, 7)])
def test_density_matrices_in_parts(cuda, n, na, nb):
    s, sb = builder(n, na, nb)
    x, y = random_ci_vector(s.ndet, 1), random_ci_vector(s.ndet, 2)
    tol = 1e-13 * np.linalg.norm(x) * np.linalg.norm(y)
    for kind in ("a_1rdm", "b_1rdm", "ab_2rdm", "aa_2rdm", "bb_2rdm") + (("aab_3rdm", "bbb_3rdm") if n <= 11 else ()):
        sb.set_variant("digit_buffer_bytes", 0)
        whole = np.asarray(getattr(sb, kind)(x, y))
        for size in (1, 600_000):
            sb.set_variant("digit_buffer_bytes", size)
            assert np.abs(np.asarray(getattr(sb, kind)(x, y)) - whole).max(initial=0.0) <= tol, (kind, size)
    assert sb.tensor_core_error() == 0


def test_a_limit_set_before_a_solve(cuda):
    from forte2_gb300.ci import CASCISolver
    from forte2_gb300.params import CIParams, DavidsonLiuParams

    ints = make_integrals(10, 11)
    e = []
    for variants in (None, {"digit_buffer_bytes": 500_000}):
        solver = CASCISolver(norb=10, na=5, nb=5, multiplicity=1, nroot=2, E=ints.E, H=ints.H, V=ints.V,
                             ci_params=CIParams(), sigma_variants=variants,
                             davidson_liu_params=DavidsonLiuParams(e_tol=1e-10, maxiter=200))
        solver.run()
        e.append(np.array(solver.evals))
        solver.new_problem(ints.E, ints.H, ints.V)  # the same limit again: allowed beside captured graphs
        solver.run()
        assert (np.asarray(solver.evals) == e[-1]).all()
        if variants:
            with pytest.raises(ValueError, match="captured graphs"):
                solver.sigma_builder.set_variant("digit_buffer_bytes", 1)
    assert (e[0] == e[1]).all()  # the same sigma bits, so the same iterations
