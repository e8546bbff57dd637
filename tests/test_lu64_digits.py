"""The trailing update of the FP64 LU (csrc/lu64.cu) restated with Python
integers: entries split into seven digits of eight bits relative to the largest
of their row (L21) or column (U12), the 34 digit products of the highest
weights, sums kept as integers.  The bound checked is the one the kernel
claims: every group of products stays below 2^24 (exact in FP32 accumulation),
the two lowest groups fit 32-bit integers together, and the product is within
(K / 2 + 1) 2^-54 of (largest of the row) x (largest of the column): half a unit
2^-55 from the splitting of either factor, half a unit 2^-54 from the rounding
of the lowest groups, less than that from the products left out."""
import numpy as np
import pytest

S = 7


def digits(v, e):
    """v = I 2^(e - 55) rounded; I as seven digits in [-128, 128], highest first."""
    I = int(np.rint(np.ldexp(np.longdouble(v), 55 - e)))
    d = []
    for _ in range(S - 1):
        low = ((I + 128) & 255) - 128
        d.append(low)
        I = (I - low) >> 8
    d.append(I)
    assert -128 <= I <= 128
    return d[::-1]


def exponent(v):
    return int(np.frexp(np.max(np.abs(v)))[1])


@pytest.mark.parametrize("kind", ["normal", "uniform", "graded", "ones", "equal"])
def test_digit_products(kind):
    rng = np.random.default_rng(11)
    K = 64
    for trial in range(20):
        a, b = rng.normal(size=K), rng.normal(size=K)
        if kind == "uniform":
            a, b = rng.uniform(0.5, 1, K), rng.uniform(0.5, 1, K)
        elif kind == "graded":
            a, b = a * 10.0 ** rng.uniform(-12, 0, K), b * 10.0 ** rng.uniform(-12, 0, K)
        elif kind == "ones":
            a, b = np.ones(K), np.full(K, 1 - 2.0 ** -53)
        elif kind == "equal":
            a, b = np.full(K, rng.uniform()), np.full(K, rng.uniform())
        ea, eb = exponent(a), exponent(b)
        da, db = [digits(x, ea) for x in a], [digits(x, eb) for x in b]
        G = [sum(da[k][s] * db[k][g - s] for k in range(K) for s in range(g + 1)) for g in range(S)]
        G.append(sum(da[k][s] * db[k][7 - s] for k in range(K) for s in range(1, S)))
        assert max(abs(x) for x in G) < 2 ** 24
        assert abs(G[6] * 256 + G[7] + 32768) < 2 ** 31
        T = sum(G[g] << (8 * (5 - g)) for g in range(6)) + ((G[6] * 256 + G[7] + 32768) >> 16)
        assert abs(T) < 2 ** 62
        from fractions import Fraction
        exact = sum(Fraction(x) * Fraction(y) for x, y in zip(a, b))
        got = Fraction(T) * Fraction(2) ** (ea + eb - 54)
        bound = (Fraction(K, 2) + 1) * Fraction(2) ** (ea + eb - 54)
        assert abs(got - exact) <= bound
