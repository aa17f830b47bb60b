"""New integrals while the FP64 tensor-core variant is off: turned on again, or replayed by a graph captured before,
sigma is the new integrals' (bitwise that of a builder made with them)."""
import numpy as np
import pytest

from forte2_gb300.synthetic import make_integrals, random_ci_vector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("update", ["set_Hamiltonian", "update_integrals"])
@pytest.mark.parametrize("n,na,nb", [(8, 4, 4), (10, 5, 5)])  # digits on request, by default
def test_integrals_change_while_the_variant_is_off(cuda, n, na, nb, update):
    torch = cuda
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings

    def make(E, ints):
        s = CIStrings(na, nb, 0, [[0] * n], [], [])
        sb = CISigmaBuilder(s, E, ints.H, ints.V, 0)
        sb.set_variant("digit_fp64", 1)
        return s, sb

    def apply(sb):
        out = torch.empty_like(c)
        sb.Hamiltonian(c, out)
        return out

    old, new = make_integrals(n, 1), make_integrals(n, 2)
    s, sb = make(0.5, old)
    c = torch.as_tensor(random_ci_vector(s.ndet, 3), device="cuda")
    before = apply(sb)
    sb.set_variant("digit_fp64", 0)
    getattr(sb, update)(-0.25, new.H, new.V)
    sb.set_variant("digit_fp64", 1)
    after = apply(sb)
    assert torch.equal(after, apply(make(-0.25, new)[1]))
    assert not torch.equal(after, before)


def test_graph_captured_before_the_variant_is_turned_off(cuda):
    from forte2_gb300.ci import CASCISolver
    from forte2_gb300.params import CIParams, DavidsonLiuParams

    n, nroot = 10, 2

    def make(ints):
        return CASCISolver(norb=n, na=5, nb=5, multiplicity=1, nroot=nroot, E=ints.E, H=ints.H, V=ints.V,
                           ci_params=CIParams(), davidson_liu_params=DavidsonLiuParams(e_tol=1e-10, maxiter=200))

    problems = [make_integrals(n, seed) for seed in (11, 12, 13)]
    kept = make(problems[0])
    kept.run()
    assert kept.eigensolver.used_graph
    kept.sigma_variants = {"digit_fp64": 0}
    for ints in problems[1:]:
        kept.new_problem(ints.E, ints.H, ints.V)
        kept.run()
        fresh = make(ints)
        fresh.run()
        # both converged to 1e-10 in the energy
        assert np.abs(np.asarray(kept.evals) - np.asarray(fresh.evals)).max() < 1e-9
