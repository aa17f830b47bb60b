"""FP64 sigma by digit splitting on the tensor cores (csrc/oz.cu) against the oracle port, at the edges of
its tiles (128 rows, 48 columns, K steps of 16), of its digit bounds and of its buffers."""
import numpy as np
import pytest

from forte2_gb300.synthetic import make_integrals, random_ci_vector

pytestmark = pytest.mark.gpu

# norb, na, nb: one tile and remainders of 128; unequal spins; 12 and 14 alpha holes (the kept integers of a
# tile just fit, and do not fit, shared memory); 81, 98, 120, 132, 144 non-zero rows per output (no
# slack, slack in one operand, in both); two chunks of output pairs
SIZES = [(4, 2, 2), (6, 3, 3), (7, 2, 5), (8, 4, 4), (9, 4, 3), (10, 5, 5), (11, 5, 4), (12, 3, 4), (13, 2, 2),
         (13, 2, 4), (14, 3, 4), (15, 2, 9), (12, 6, 6)]


def _builder(n, na, nb, seed=5, scale=1.0):
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings

    ints = make_integrals(n, seed)
    strings = CIStrings(na, nb, 0, [[0] * n], [], [])
    sb = CISigmaBuilder(strings, 0.75, ints.H * scale, ints.V * scale, 0)
    sb.set_algorithm("hz")
    sb.set_variant("digit_fp64", 1)
    return ints, strings, sb


def _apply(sb, c):
    import torch

    c = torch.as_tensor(c, device="cuda")
    s = torch.full_like(c, float("nan"))
    sb.Hamiltonian(c, s)
    assert sb.tensor_core_error() == 0
    return s


@pytest.mark.parametrize("n,na,nb", SIZES)
def test_sigma_matches_oracle(n, na, nb):
    from oracle.port import PortCI

    ints, strings, sb = _builder(n, na, nb)
    port = PortCI(n, na, nb)
    port.set_hamiltonian(0.75, ints.H, ints.V)
    rng = np.random.default_rng(n)
    c = random_ci_vector(strings.ndet, 7)
    # a second vector whose elements span twenty decades, a third that is zero but for one element
    wide = c * 10.0 ** rng.uniform(-20, 0, strings.ndet)
    one = np.zeros_like(c)
    one[strings.ndet // 3] = 1.0
    got = _apply(sb, np.stack([c, wide, one, np.zeros_like(c)])).cpu().numpy()
    for x, s in zip((c, wide, one), got):
        ref = port.sigma(x)
        # FP64 sums of some thousand terms: sqrt(terms) 2^-53 of the norm, far below 1e-13
        assert np.linalg.norm(s - ref) <= 1e-13 * np.linalg.norm(ref)
    assert not got[3].any()


@pytest.mark.parametrize("n,na,nb", [(9, 4, 3), (12, 6, 6)])
def test_bitwise_equal_in_any_batch_and_grid(n, na, nb):
    import torch

    _, strings, sb = _builder(n, na, nb)
    c = np.stack([random_ci_vector(strings.ndet, s) for s in range(5)])
    all5 = _apply(sb, c)
    for i in range(5):
        assert torch.equal(all5[i], _apply(sb, c[i]))
    sb.set_max_blocks(7)
    assert torch.equal(all5, _apply(sb, c))


def test_scales_and_non_finite_elements():
    import torch

    ints, strings, sb = _builder(8, 4, 4)
    c = random_ci_vector(strings.ndet, 3)
    ref = _apply(sb, c)
    # powers of two commute with every rounding
    for e in (-900, 700):
        assert torch.equal(_apply(sb, c * 2.0 ** e), ref * 2.0 ** e)
    _, _, small = _builder(8, 4, 4, scale=2.0 ** -600)
    sb0 = _builder(8, 4, 4)[2]
    sb0.set_Hamiltonian(0.0, ints.H, ints.V)
    small.set_Hamiltonian(0.0, ints.H * 2.0 ** -600, ints.V * 2.0 ** -600)
    assert torch.equal(_apply(small, c) * 2.0 ** 600, _apply(sb0, c))
    for bad in (float("nan"), float("inf")):
        d = c.copy()
        d[17] = bad
        s = _apply(sb, d)
        sb.set_variant("digit_fp64", 0)
        plain = _apply(sb, d)
        sb.set_variant("digit_fp64", 1)
        assert torch.equal(torch.isfinite(s), torch.isfinite(plain))


def test_refused_where_the_sizes_rule_it_out():
    from forte2_gb300.ci_helpers import CISigmaBuilder, CIStrings

    for n, na, nb in [(16, 2, 2), (8, 1, 4), (17, 2, 2)]:
        ints = make_integrals(n, 1)
        sb = CISigmaBuilder(CIStrings(na, nb, 0, [[0] * n], [], []), 0.0, ints.H, ints.V, 0)
        with pytest.raises(ValueError, match="digit splitting"):
            sb.set_variant("digit_fp64", 1)
