"""Building an H-matrix (csrc/hmatrix.cu): pivots of the compression, recompression."""
import numpy as np
import pytest

from conftest import sphere_input

pytestmark = pytest.mark.gpu
bem = pytest.importorskip("cc_abstemious_gb300")


def test_repeated_builds_are_bit_identical():
    """Every leaf's pivots, ranks and factors are a sequence of their own, whichever
    of its warps is ahead."""
    solver = {"Hierarchical": {"max_iterations": 1000, "tolerance": 1e-6, "leaf_size": 16, "eta": 1.0,
                               "aca_tolerance": 1e-5}}
    inp = sphere_input("refined_sphere.vtk", solver=solver, method_type="BurtonMiller")
    pd = bem.PreData.from_dict(inp, ctx=bem.Context.default())
    rng = np.random.default_rng(1)
    x, b = (rng.normal(size=pd.n) + 1j * rng.normal(size=pd.n) for _ in range(2))
    first = None
    for _ in range(200):
        H = bem.HMatrix(pd, bem.EqnSide.LHS)
        got = (H.stats(), H.gemv(0.7 - 0.2j, x, 0.3 + 0.1j, b))
        first = first or got
        assert got[0] == first[0] and np.array_equal(got[1], first[1])
