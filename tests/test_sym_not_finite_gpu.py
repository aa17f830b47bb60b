"""Infinities and NaN in the vector of a point-group-blocked space (csrc/sym_digits.cu): sigma is not finite in the
elements that H couples to them and in no other, and the others are what they are without them."""
import numpy as np
import pytest

from forte2_gb300.synthetic import make_integrals, random_ci_vector, symmetrize_integrals

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("orbsym,na,nb", [([0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3], 6, 6), ([0] * 9 + [1] * 3, 6, 5)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_only_coupled_elements(cuda, orbsym, na, nb, bad):
    torch = cuda
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings

    n = len(orbsym)
    ints = symmetrize_integrals(make_integrals(n, 21), orbsym)
    s = CIStrings(na, nb, 0, [orbsym], [], [])
    sb = CISigmaBuilder(s, ints.E, ints.H, ints.V, 0)
    det = np.asarray(s.make_determinants().masks())
    x = random_ci_vector(s.ndet, 5)
    at = [s.ndet // 3, s.ndet // 3 + 1, s.ndet - 7]
    zero = x.copy()
    zero[at] = 0.0
    x[at] = [bad, -bad, bad]

    def excitations(i):
        d = [np.array([bin(int(m)).count("1") for m in det[:, k] ^ det[i, k]]) // 2 for k in (0, 1)]
        return d[0] + d[1]

    near = np.min([excitations(i) for i in at], axis=0)
    X = torch.as_tensor(np.stack([x, zero]), device="cuda")
    out = torch.empty_like(X)
    sb.Hamiltonian(X, out)
    got, ref = out.cpu().numpy()
    assert np.isfinite(ref).all()
    # more than two excitations away nothing is touched (rows of the zeroed vector keep their scale but for the three)
    far = near > 2
    assert np.isfinite(got[far]).all()
    assert np.linalg.norm(got[far] - ref[far]) <= 1e-13 * np.linalg.norm(ref[far])
    sb.set_variant("irrep_blocks", 0)  # the FP64 kernels on the embedding
    sb.Hamiltonian(X, out)
    plain = out[0].cpu().numpy()
    assert (np.isfinite(got) == np.isfinite(plain)).all()
    if np.isinf(bad):
        both = np.isinf(got) & np.isinf(plain)
        assert both.any() and (got[both] == plain[both]).all()
