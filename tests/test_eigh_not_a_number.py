"""The subspace eigensolver (csrc/davidson.cu) on matrices that hold a NaN or an infinity: its output order stays a
permutation, so that nothing outside its arrays is read, and the result says what it is."""
import itertools

import numpy as np
import pytest

NAN = float("nan")


def rank_order(w):
    """The kernel's output order: rank of every eigenvalue, ties by index, NaN last."""
    order = [-1] * len(w)
    for i, a in enumerate(w):
        r = sum(1 for j, x in enumerate(w)
                if x < a or (a != a and x == x) or ((x == a or (x != x and a != a)) and j < i))
        order[r] = i
    return order


def test_order_is_a_permutation():
    for w in itertools.product([NAN, 1.0, -2.0, float("inf")], repeat=4):
        order = rank_order(w)
        assert sorted(order) == [0, 1, 2, 3]
        v = [w[i] for i in order]
        numbers = [x for x in v if x == x]
        assert numbers == sorted(numbers) and all(x != x for x in v[len(numbers):])


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("m", [1, 5, 8, 12, 40, 64])
def test_matrix_with_a_bad_element(cuda, m, bad):
    torch = cuda
    from forte2_gb300._lib import check, lib, stream_handle

    g = np.random.default_rng(m).normal(size=(m, m))
    g = g + g.T
    g[m // 2, m // 3] = g[m // 3, m // 2] = bad
    G = torch.as_tensor(g, device="cuda")
    ev = torch.zeros(m, dtype=torch.float64, device="cuda")
    V = torch.zeros((m, m), dtype=torch.float64, device="cuda")
    check(lib().f2g_dav_eigh(m, G.data_ptr(), ev.data_ptr(), V.data_ptr(), stream_handle()))
    assert not torch.isfinite(ev).all()
    two = torch.eye(m, dtype=torch.float64, device="cuda") * 2.0
    check(lib().f2g_dav_eigh(m, two.data_ptr(), ev.data_ptr(), V.data_ptr(), stream_handle()))
    assert (ev == 2.0).all()
