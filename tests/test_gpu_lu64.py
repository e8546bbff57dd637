"""The FP64 LU (csrc/lu64.cu) at the sizes where its tiles, panels and clusters
end: blocks of 32 columns, clusters of up to 16 CTAs with 32 rows each, narrower
panels above 1024 rows, row blocks and column tiles of 64.

The measure is the normwise backward error ||A x - b|| / (||A||_F ||x||), which
for partial pivoting is at most a small multiple of n u (u = 2^-53); the bound
below is 16 (n + 8) u, fixed beforehand (complex products count for 2 sqrt 2, the
growth of random matrices for about n^(1/4))."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
bem = pytest.importorskip("cc_abstemious_gb300")
U = 2.0 ** -53


def matrix(n, seed, kind="plain"):
    rng = np.random.default_rng(seed)
    A = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    if kind == "graded":  # rows and columns over many orders of magnitude
        A = 10.0 ** rng.uniform(-6, 6, n)[:, None] * A * 10.0 ** rng.uniform(-3, 3, n)[None, :]
    elif kind == "tiny":  # products outside the range of normal numbers
        A = A * 1e-160
    elif kind == "pivots":  # every pivot is the last row
        A = A + 1e3 * np.eye(n)[::-1]
    return A, rng.normal(size=n) + 1j * rng.normal(size=n)


def backward(A, x, b):
    return np.linalg.norm(A @ x - b) / (np.linalg.norm(A) * np.linalg.norm(x))


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 95, 97, 127, 129, 161, 255, 257, 511, 513, 545, 1023,
                               1025, 1057, 1217, 2433])
def test_sizes(n):
    A, b = matrix(n, n)
    assert backward(A, bem.solve_lu(A, b), b) <= 16 * (n + 8) * U


@pytest.mark.parametrize("kind", ["graded", "tiny", "pivots"])
@pytest.mark.parametrize("n", [33, 97, 300, 1100])
def test_scales_and_exchanges(n, kind):
    A, b = matrix(n, 7 * n, kind)
    s = 1.0 if kind != "tiny" else 1e160
    x = bem.solve_lu(A, b * (1e-160 if kind == "tiny" else 1.0))
    assert backward(A * s, x, b) <= 16 * (n + 8) * U


def test_graded_rows_keep_their_digits():
    """Row by row: a row scaled by 1e-9 has the residual of its own scale."""
    A, b = matrix(300, 3)
    d = 10.0 ** np.random.default_rng(4).uniform(-9, 0, 300)
    x = bem.solve_lu(d[:, None] * A, d * b)
    r = np.abs(A @ x - b) / (np.linalg.norm(A, axis=1) * np.linalg.norm(x))
    assert r.max() <= 16 * 308 * U


def test_zero_pivot_is_singular_and_nothing_sticks():
    A, b = matrix(200, 1)
    A[:, 77] = 0
    with pytest.raises(bem.BemError):
        bem.solve_lu(A, b)
    A, b = matrix(200, 1)
    assert backward(A, bem.solve_lu(A, b), b) <= 16 * 208 * U


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_non_finite_entries_end_in_non_finite_results(value):
    A, b = matrix(150, 2)
    A[140, 3] = value
    try:
        x = bem.solve_lu(A, b)
    except bem.BemError:
        return
    assert not np.all(np.isfinite(x))
    A, b = matrix(150, 2)
    assert backward(A, bem.solve_lu(A, b), b) <= 16 * 158 * U


@pytest.mark.parametrize("n", [2, 31, 33, 95, 545, 1057])
def test_repeated_solves_are_bit_identical(n):
    """The panels' CTAs and warps hand results to one another; every hand-over has
    its barrier, so that a solve does not depend on which of them is ahead."""
    A, b = matrix(n, 5 * n)
    x = bem.solve_lu(A, b)
    for _ in range(10):
        assert np.array_equal(bem.solve_lu(A, b), x)


def rowwise(A, x, b):
    """Largest |b - A x|_i / (|A| |x|)_i, which for partial pivoting is a small
    multiple of n u whatever the scale of row i or of the columns."""
    return float(np.max(np.abs(A @ x - b) / (np.abs(A) @ np.abs(x))))


@pytest.mark.parametrize("scale", [1e6, 1e9, 1e12])
@pytest.mark.parametrize("count", [1, 15, 17, 24, 31, 56])
@pytest.mark.parametrize("n", [300, 1100, 2100])
def test_a_few_rows_of_another_scale(n, count, scale):
    """The large rows are the first pivots and end inside a block; where its panels
    are narrower than it, the rows exchanged by a later panel leave the columns
    of an earlier one small."""
    A, b = matrix(n, n + count)
    rows = np.random.default_rng(count).permutation(n)[:count]
    A[rows] *= scale
    b[rows] *= scale
    assert rowwise(A, bem.solve_lu(A, b), b) <= 16 * (n + 8) * U


@pytest.mark.parametrize("count", [17, 24, 56])
@pytest.mark.parametrize("n", [300, 1100, 2100])
def test_a_few_columns_of_another_scale(n, count):
    A, b = matrix(n, 2 * n + count)
    A[:, np.random.default_rng(count).permutation(n)[:count]] *= 1e9
    assert rowwise(A, bem.solve_lu(A, b), b) <= 16 * (n + 8) * U


@pytest.mark.parametrize("n", [300, 1100, 1500])
def test_rows_over_many_decades(n):
    A, b = matrix(n, n + 5)
    d = 10.0 ** np.random.default_rng(n).uniform(-9, 9, n)
    A, b = d[:, None] * A, d * b
    assert rowwise(A, bem.solve_lu(A, b), b) <= 16 * (n + 8) * U


@pytest.mark.parametrize("n", [12833, 25665])
def test_panels_of_eight_and_of_four_columns(n):
    """Above 12800 and 25600 rows the cluster's shared memory holds panels of 8 and
    of 4 columns; twenty-four rows a billion times the others, as above."""
    import torch
    ctx = bem.Context()
    g = torch.Generator(device="cuda").manual_seed(n)
    At = torch.randn(n, n, dtype=torch.complex128, device="cuda", generator=g)  # its transpose, column-major
    b = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
    rows = torch.randperm(n, device="cuda", generator=g)[:24]
    At[:, rows] *= 1e9
    b[rows] *= 1e9
    x = b.clone()
    torch.cuda.synchronize()
    ctx.check(ctx.lib.bem_solve_lu(ctx.h, n, At.data_ptr(), n, x.data_ptr(), 1))
    size = torch.empty(n, dtype=torch.float64, device="cuda")
    for i in range(0, n, 2048):
        size[i:i + 2048] = x.abs() @ At[:, i:i + 2048].abs()
    r = ((x @ At - b).abs() / size).max().item()
    del At, size, ctx
    torch.cuda.empty_cache()
    assert r <= 16 * (n + 8) * U


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1j * np.inf])
@pytest.mark.parametrize("first,last", [(40, 41), (40, 44), (92, 96), (32, 96)])
def test_zeros_of_l21_meet_non_finite_columns_of_u12(first, last, value):
    """0 x infinity is NaN in elimination: rows of L21 that are zero throughout carry
    it into the trailing matrix, and from there into every unknown (four columns at
    a time in the kernel: alone, in a whole group of four, everywhere)."""
    A, b = matrix(96, 9)
    A[32:, :32] = 0
    A[3, first:last] = value
    try:
        x = bem.solve_lu(A, b)
    except bem.BemError:
        return
    assert not np.isfinite(x).any()
