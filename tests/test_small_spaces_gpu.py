"""One-launch sigma of small spaces (csrc/small.cu) and the subspace eigensolver at close eigenvalues."""
import numpy as np
import pytest

from forte2_gb300.synthetic import make_integrals, random_ci_vector

pytestmark = pytest.mark.gpu


# one alpha or beta electron, unequal spins, lists that are no multiple of the four lanes, the most
# determinants of the one-launch path (7,056), and a space whose integrals do not fit it
@pytest.mark.parametrize("n,na,nb", [(2, 1, 1), (5, 1, 4), (5, 5, 2), (7, 3, 2), (9, 3, 3), (11, 2, 1), (13, 1, 1)])
def test_small_sigma_matches_oracle(n, na, nb):
    import torch

    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings
    from oracle.port import PortCI

    ints = make_integrals(n, 11)
    strings = CIStrings(na, nb, 0, [[0] * n], [], [])
    sb = CISigmaBuilder(strings, -1.5, ints.H, ints.V, 0)
    sb.set_algorithm("hz")
    port = PortCI(n, na, nb)
    port.set_hamiltonian(-1.5, ints.H, ints.V)
    c = np.stack([random_ci_vector(strings.ndet, s) for s in range(3)])
    x = torch.as_tensor(c, device="cuda")
    s = torch.full_like(x, float("nan"))
    sb.Hamiltonian(x, s)
    for i in range(3):
        ref = port.sigma(c[i])
        # some hundred FP64 terms per element
        assert np.linalg.norm(s[i].cpu().numpy() - ref) <= 1e-13 * max(np.linalg.norm(ref), 1e-3)
        one = torch.empty_like(x[i])
        sb.Hamiltonian(x[i].contiguous(), one)
        assert torch.equal(one, s[i])


@pytest.mark.parametrize("m", [2, 8, 9, 32, 40])
@pytest.mark.parametrize("split", [0.0, 1e-13, 1e-9, 1e-6, 1e-3])
def test_eigh_of_close_eigenvalues(m, split):
    import torch

    from forte2_gb300._lib import check, lib, stream_handle

    rng = np.random.default_rng(m)
    Q, _ = np.linalg.qr(rng.normal(size=(m, m)))
    w = np.sort(-70.0 + rng.uniform(0, 5, m))
    w[1] = w[0] + split  # below what FP32 separates for the first splits: the FP64 sweeps
    A = (Q * w) @ Q.T
    A = 0.5 * (A + A.T)
    G = torch.as_tensor(A, device="cuda")
    ev = torch.empty(m, dtype=torch.float64, device="cuda")
    V = torch.empty((m, m), dtype=torch.float64, device="cuda")
    check(lib().f2g_dav_eigh(m, G.data_ptr(), ev.data_ptr(), V.data_ptr(), stream_handle()))
    X, e = V.cpu().numpy(), ev.cpu().numpy()
    eps = np.finfo(float).eps
    assert np.abs(e - np.linalg.eigvalsh(A)).max() <= 8 * eps * m * 75
    assert np.abs(X.T @ X - np.eye(m)).max() <= 8 * eps * m
    assert np.abs(A @ X - X * e).max() <= 8 * eps * m * 75
