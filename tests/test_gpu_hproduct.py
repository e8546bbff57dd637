"""H-matrix products (csrc/hmatrix.cu, hm_leaf_mv_kernel) over the leaf sizes where
the sharing of rows and columns among its four warps changes: leaves of up to 32,
64 and more rows, of more than 512 columns, dense and compressed, and ranks that
are no multiple of four, against the same operator expanded to a matrix.

Both sums run over the same stored entries in another order, so they differ by
rounding of sums of up to n products: below 1e-12 of the largest value for n <= 900,
with u = 1.1e-16 and the growth from U (V^T x) instead of (U V^T) x."""
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
bem = pytest.importorskip("cc_abstemious_gb300")
from cc_abstemious_gb300 import workloads  # noqa: E402


@pytest.mark.parametrize("leaf,eta", [(1, 4.0), (7, 2.0), (31, 4.0), (33, 1.0), (64, 4.0), (65, 2.0), (150, 4.0),
                                      (600, 4.0), (1000, 1.0)])
def test_leaf_sizes(leaf, eta):
    inp = workloads.perturbed_sphere_input(tempfile.mkdtemp(prefix="bem_hprod_"), leaf, 900, [2.0])
    inp["solver"] = {"Hierarchical": {"tolerance": 1e-6, "max_iterations": 1000, "leaf_size": leaf, "eta": eta,
                                      "aca_tolerance": 1e-5}}
    pd = bem.PreData.from_dict(inp, ctx=bem.Context.default())
    H = bem.HMatrix(pd, bem.EqnSide.LHS)
    F = H.to_full()
    rng = np.random.default_rng(leaf)
    x, b = (rng.normal(size=pd.n) + 1j * rng.normal(size=pd.n) for _ in range(2))
    for alpha, beta in ((1.0 + 0j, 0.0 + 0j), (0.5 - 1j, 2.0 + 0.5j)):
        ref = alpha * (F @ x) + beta * b
        assert np.max(np.abs(H.gemv(alpha, x, beta, b) - ref)) <= 1e-12 * np.max(np.abs(ref))
