"""FP64 digit sigma (csrc/oz.cu) of so many vectors in one call that their column tiles are more than a grid takes."""
import pytest

from forte2_gb300.synthetic import make_integrals

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,na,nb,nvec", [(4, 2, 2, 65535), (6, 3, 3, 20000), (8, 4, 8, 40000)])
def test_many_vectors(cuda, n, na, nb, nvec):
    torch = cuda
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings

    ints = make_integrals(n, 4)
    s = CIStrings(na, nb, 0, [[0] * n], [], [])
    sb = CISigmaBuilder(s, ints.E, ints.H, ints.V, 0)
    sb.set_variant("digit_fp64", 1)
    g = torch.Generator(device="cuda").manual_seed(3)
    X = torch.randn(nvec, s.ndet, generator=g, dtype=torch.float64, device="cuda")
    out = torch.empty_like(X)
    sb.Hamiltonian(X, out)
    for i in (0, 16383, 16384, nvec - 1):
        if i < nvec:
            one = torch.empty_like(X[i])
            sb.Hamiltonian(X[i].contiguous(), one)
            assert torch.equal(out[i], one)
    sb.set_variant("digit_fp64", 0)
    plain = torch.empty_like(X)
    sb.Hamiltonian(X, plain)
    assert (torch.linalg.vector_norm(out - plain, dim=1) <= 1e-13 * torch.linalg.vector_norm(plain, dim=1)).all()
