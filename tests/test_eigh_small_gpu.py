"""The subspace eigensolver (csrc/davidson.cu) for the one or two vectors a solve starts with."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("g", [
    [[3.0]], [[-1e-300]], [[0.0]],
    [[1.0, 0.0], [0.0, -2.0]], [[0.0, 0.0], [0.0, 0.0]], [[1.0, 1e-9], [1e-9, 1.0]], [[2.0, 1.0], [1.0, 2.0]],
    [[-20.0, 1e-3], [1e-3, -19.5]], [[1e200, 3e199], [3e199, -1e200]], [[-7.0, 1e-18], [1e-18, -8.0]],
    [[1.0, 0.3], [0.1, 2.0]],  # its symmetric part
])
def test_small_matrices(cuda, g):
    torch = cuda
    from forte2_gb300._lib import check, lib, stream_handle

    g = np.array(g)
    m = len(g)
    G = torch.as_tensor(g, device="cuda")
    ev = torch.zeros(m, dtype=torch.float64, device="cuda")
    V = torch.zeros((m, m), dtype=torch.float64, device="cuda")
    check(lib().f2g_dav_eigh(m, G.data_ptr(), ev.data_ptr(), V.data_ptr(), stream_handle()))
    a = (g + g.T) / 2
    w, v, size = ev.cpu().numpy(), V.cpu().numpy(), max(np.abs(a).max(), 1e-300)
    assert (np.diff(w) >= 0).all()
    # a few roundings of the largest element
    assert np.abs(w - np.linalg.eigvalsh(a)).max() <= 1e-15 * size
    assert np.abs(v.T @ v - np.eye(m)).max() <= 1e-15
    assert np.abs((a / size) @ v - v * (w / size)).max() <= 1e-15
