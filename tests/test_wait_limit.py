"""Bounded waits of the digit kernels (csrc/oz.cu, rdm_gram.cu, sym_digits.cu) that run out: the results are NaN, the
caller is told, the device stays usable and the next build is the usual one, to the bit."""
import itertools

import numpy as np
import pytest

from forte2_gb300.synthetic import make_integrals, random_ci_vector, symmetrize_integrals


def waits_end(totals, nbuf, fill):
    """Ring of nbuf slots filled by three warps each, which stopped after `totals` steps: do the waits for the last
    copies of every slot end? fill: a warp arrives without a copy in the steps that others have copied and it has not."""
    most = max(totals)
    arrivals = [sum(1 for t in totals if step < (most if fill else t)) for step in range(most)]
    waited = [range(max(0, (most if fill else t) - nbuf), most if fill else t) for t in totals]
    return all(arrivals[step] == 3 for steps in waited for step in steps)


def test_copies_are_waited_for_when_one_warp_stops_early():
    for nbuf in (2, 3, 8):
        for totals in itertools.product(range(2 * nbuf + 2), repeat=3):
            if max(totals) - min(totals) > nbuf:
                continue  # a step is copied once its slot's last use is complete, for which all three have copied it
            assert waits_end(totals, nbuf, True)
            assert waits_end(totals, nbuf, False) == (len(set(totals)) == 1)


def _builder(n, na, nb, irreps=None):
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings

    ints = make_integrals(n, 4)
    if irreps is not None:
        ints = symmetrize_integrals(ints, irreps)
    s = CIStrings(na, nb, 0, [[0] * n if irreps is None else irreps], [], [])
    return s, CISigmaBuilder(s, ints.E, ints.H, ints.V, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("n,na,nb,irreps", [
    (8, 4, 4, None), (11, 5, 4, None), (12, 6, 6, [0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3])])
def test_sigma(cuda, n, na, nb, irreps):
    torch = cuda
    s, sb = _builder(n, na, nb, irreps)
    if irreps is None:
        sb.set_variant("digit_fp64", 1)
    c = torch.as_tensor(random_ci_vector(s.ndet, 3), device="cuda")
    ref = torch.empty_like(c)
    sb.Hamiltonian(c, ref)
    sb.check()
    sb.set_variant("tc_wait_limit", 1)  # one try: the first wait for a copy gives up
    out = torch.zeros_like(c)
    sb.Hamiltonian(c, out)
    torch.cuda.synchronize()
    assert torch.isnan(out).all()
    assert sb.tensor_core_error() == 1
    with pytest.raises(RuntimeError, match="gave up"):
        sb.Hamiltonian(c, out)
    host = np.zeros(s.ndet)
    with pytest.raises(RuntimeError, match="gave up"):
        sb.Hamiltonian(c.cpu().numpy(), host)
    sb.set_variant("tc_wait_limit", 0)
    sb.Hamiltonian(c, out)
    assert torch.equal(out, ref)
    assert sb.tensor_core_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["ab_2rdm", "sf_2rdm", "sf_3rdm"])
def test_rdm(cuda, kind):
    torch = cuda
    s, sb = _builder(8, 4, 4)
    c = torch.as_tensor(random_ci_vector(s.ndet, 3), device="cuda")
    ref = getattr(sb, kind)(c, c)
    sb.set_variant("tc_wait_limit", 1)
    out = getattr(sb, kind)(c, c)
    torch.cuda.synchronize()
    assert torch.isnan(out).any()
    with pytest.raises(RuntimeError, match="gave up"):
        sb.check()
    with pytest.raises(RuntimeError, match="gave up"):
        getattr(sb, kind)(c.cpu().numpy(), c.cpu().numpy())
    sb.set_variant("tc_wait_limit", 0)
    again = getattr(sb, kind)(c, c)
    # partial results are added by atomics in any order
    assert (again - ref).abs().max().item() <= 1e-14


@pytest.mark.gpu
@pytest.mark.parametrize("use_graph", [True, False])
def test_solve(cuda, use_graph):
    from forte2_gb300.ci import CASCISolver
    from forte2_gb300.params import CIParams, DavidsonLiuParams

    ints = make_integrals(10, 5)
    solver = CASCISolver(norb=10, na=5, nb=5, multiplicity=1, nroot=1, E=ints.E, H=ints.H, V=ints.V,
                         ci_params=CIParams(), davidson_liu_params=DavidsonLiuParams(e_tol=1e-10, maxiter=200),
                         use_graph=use_graph, sigma_variants={"tc_wait_limit": 1})
    with pytest.raises(RuntimeError, match="gave up"):
        solver.run()
