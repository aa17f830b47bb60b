"""Integer model of the digit splitting of csrc/oz.cu: what the kernel relies on for exactness."""
from fractions import Fraction

import numpy as np
import pytest

DIGITS = 7


def digits(x, e):
    """Signed base-256 digits of x = X 2^(e - 1078), X truncated to 56 bits (the first digit holds 9)."""
    X = int(abs(Fraction(x)) / Fraction(2) ** (e - 1078))
    X = X if x >= 0 else -X
    Z = X + 0x808080808080
    return [Z >> 48] + [((Z >> (8 * (5 - i))) & 255) - 128 for i in range(6)], X


def exponent(x):
    return int(np.frexp(abs(x))[1]) + 1022 if x else 64


@pytest.mark.parametrize("slack", [0, 1])
def test_digits_reconstruct_and_stay_in_range(slack):
    rng = np.random.default_rng(slack)
    xs = np.concatenate([rng.normal(size=400), 10.0 ** rng.uniform(-18, 0, 400), [1.0, -1.0, 1 - 2.0 ** -53, -1 + 2.0 ** -53,
                                                                                 0.0, 0.50196078431372548]])
    e = exponent(np.abs(xs).max()) + slack
    for x in xs:
        d, X = digits(x, e)
        assert sum(v * 256 ** (6 - i) for i, v in enumerate(d)) == X
        assert abs(d[0]) <= (256 >> slack) and all(-128 <= v <= 127 for v in d[1:])
        assert abs(Fraction(x) - X * Fraction(2) ** (e - 1078)) < Fraction(2) ** (e - 1078)


@pytest.mark.parametrize("nk,slack_a,slack_b", [(101, 0, 0), (126, 0, 1), (146, 1, 1)])
def test_group_sums_fit(nk, slack_a, slack_b):
    a = [256 >> slack_a] + [128] * 6
    b = [256 >> slack_b] + [128] * 6
    S = [nk * sum(a[i] * b[g - i] for i in range(g + 1)) for g in range(DIGITS)]
    assert max(S) <= 2 ** 24                       # FP32 accumulation of integers is exact
    assert S[5] + S[6] / 256 < 2 ** 24             # and so is the conversion of S_5 + S_6 / 256
    assert 256 * S[0] + S[1] < 2 ** 31 and 256 * S[2] + S[3] < 2 ** 31
    T = sum(S[g] * 256 ** (5 - g) for g in range(6)) + S[6] // 256
    assert T < 2 ** 63 and 8 * (T >> 3) < 2 ** 63  # one term, and eight of them after the shift by 3


def test_sigma_sum_error_is_below_fp64():
    """Digit-split dot products against exact rational arithmetic, and an FP64 chain of the same terms."""
    rng = np.random.default_rng(3)
    worst = [0.0, 0.0]
    for _ in range(60):
        a = rng.normal(size=81) * 10.0 ** rng.uniform(-3, 0, 81)
        b = rng.normal(0, 0.1, 81)
        ea, eb = exponent(np.abs(a).max()), exponent(np.abs(b).max())
        da = np.array([digits(x, ea)[0] for x in a], dtype=object)
        db = np.array([digits(x, eb)[0] for x in b], dtype=object)
        S = [sum(int((da[:, i] * db[:, g - i]).sum()) for i in range(g + 1)) for g in range(DIGITS)]
        T = sum(S[g] * 256 ** (5 - g) for g in range(6)) + (S[6] + 128 >> 8)
        got = Fraction(T) * Fraction(2) ** (ea + eb - 2100)
        exact = sum(Fraction(x) * Fraction(y) for x, y in zip(a, b))
        chain = 0.0
        for x, y in zip(a, b):
            chain = float(Fraction(x) * Fraction(y) + Fraction(chain))  # a fused multiply-add
        size = float(np.sqrt(((a * b) ** 2).sum()))
        worst[0] += (float(got - exact) / size) ** 2
        worst[1] += (float(Fraction(chain) - exact) / size) ** 2
    assert worst[0] < worst[1]
