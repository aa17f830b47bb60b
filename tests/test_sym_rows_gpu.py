"""The tensor-core opposite-spin sigma of point-group-blocked spaces (csrc/sym_digits.cu) scales the vector row by row:
rows that the largest one does not reach are as accurate as if it were not there."""
import numpy as np
import pytest

from forte2_gb300.synthetic import make_integrals, random_ci_vector, symmetrize_integrals

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("orbsym,na,nb", [([0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3], 6, 6), ([0, 1, 2, 3] * 3, 7, 5),
                                          ([0] * 9 + [1] * 3, 6, 5)])
@pytest.mark.parametrize("small", [1e-12, 1e-200])
def test_rows_out_of_reach_of_a_large_one(cuda, orbsym, na, nb, small):
    torch = cuda
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings

    n = len(orbsym)
    ints = symmetrize_integrals(make_integrals(n, 21), orbsym)
    s = CIStrings(na, nb, 0, [orbsym], [], [])
    sb = CISigmaBuilder(s, ints.E, ints.H, ints.V, 0)
    alpha = np.asarray(s.make_determinants().masks())[:, 0]
    large = alpha == alpha[s.ndet // 3]
    apart = np.array([bin(int(a) ^ int(alpha[s.ndet // 3])).count("1") for a in alpha]) >= 6  # three excitations
    assert apart.sum() > 100
    x = random_ci_vector(s.ndet, 5)
    x = np.where(large, x, small * x)
    # two vectors: every one has scales of its own
    X = torch.as_tensor(np.stack([x, random_ci_vector(s.ndet, 6)]), device="cuda")
    got, ref = torch.empty_like(X), torch.empty_like(X)
    sb.Hamiltonian(X, got)
    sb.set_variant("irrep_blocks", 0)
    sb.Hamiltonian(X, ref)
    rows = torch.as_tensor(apart, device="cuda")
    d, r = (got - ref)[0][rows] / small, ref[0][rows] / small
    # sums of some thousand FP64 terms, as for whole vectors
    assert torch.linalg.vector_norm(d) < 1e-13 * torch.linalg.vector_norm(r)
    assert torch.linalg.vector_norm(got[1] - ref[1]) < 1e-13 * torch.linalg.vector_norm(ref[1])
