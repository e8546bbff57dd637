"""Building an H-matrix (csrc/hmatrix.cu): pivots of the compression, recompression."""
import tempfile

import numpy as np
import pytest

from conftest import sphere_input
from oracle import oracle as O

pytestmark = pytest.mark.gpu
bem = pytest.importorskip("cc_abstemious_gb300")
from cc_abstemious_gb300 import workloads  # noqa: E402


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


@pytest.mark.parametrize("n,ka,leaf,eta,tol,ranks", [
    (500, 1.0, 30, 4.0, 1e-6, [12, 13, 20, 21, 29]),
    (900, 2.0, 33, 2.0, 1e-8, [23, 24, 25, 26, 31, 32, 33, 34]),   # both sides of 24 and of 32
    (700, 6.0, 40, 4.0, 1e-10, [15, 28, 32, 42, 49]),
    (700, 3.0, 60, 4.0, 1e-13, [29, 30, 47, 49]),                   # leaves of full rank, down to rounding
    (1400, 15.0, 150, 6.0, 1e-9, [61, 83, 84, 90]),                 # above 64, odd and even
])
def test_compressed_leaves(n, ka, leaf, eta, tol, ranks):
    """Every compressed leaf against its dense block and the ranks against the oracle's,
    at the ranks where the recompression takes other numbers of warps (24 / 25, 32 / 33),
    device instead of shared memory (32 / 33) and a bye in its pairing (odd ranks).

    The iteration ends at steps of tol / 50; what the truncation drops are singular
    values below tol times the sum of the larger ones, at most r of them: within
    (4 + r) tol of the block's norm."""
    inp = workloads.perturbed_sphere_input(tempfile.mkdtemp(prefix="bem_hb_"), 3, n, [ka])
    inp["solver"] = {"Hierarchical": {"tolerance": 1e-6, "max_iterations": 1000, "leaf_size": leaf, "eta": eta,
                                      "aca_tolerance": tol}}
    P = O.Problem(inp)
    H, G = P.dense_surface()
    al, be = P.lhs_factors()
    A = al * H + be * G
    pd = bem.PreData.from_dict(inp, ctx=bem.Context.default())
    built = bem.HMatrix(pd, bem.EqnSide.LHS)
    F, bl = built.to_full(), O.block_list(P.cpts, leaf, eta)
    seen = []
    for i in np.flatnonzero(bl["admissible"]):
        ix = np.ix_(bl["rows"][bl["row_off"][i]:bl["row_off"][i + 1]], bl["cols"][bl["col_off"][i]:bl["col_off"][i + 1]])
        r = O.aca(A[ix], tol)[0].shape[1]
        seen.append(r)
        assert np.linalg.norm(F[ix] - A[ix]) <= (4 + r) * tol * np.linalg.norm(A[ix])
    assert built.stats()["admissible"] == len(seen)
    assert abs(built.stats()["rank_sum"] - sum(seen)) <= max(2, sum(seen) // 200)
    assert set(ranks) <= set(seen)


def flat_box(path, m):
    """A cube of 6 m^2 quads with flat faces: between two elements of a face the
    classical kernel's derivative along the normal is exactly zero."""
    from cc_abstemious_gb300 import meshgen
    nodes, cells = [], []
    t = np.linspace(-1.0, 1.0, m + 1)
    for axis in range(3):
        for side in (-1.0, 1.0):
            base = len(nodes)
            for i in range(m + 1):
                for j in range(m + 1):
                    p = np.zeros(3)
                    p[axis], p[(axis + 1) % 3], p[(axis + 2) % 3] = side, t[i], t[j]
                    nodes.append(p)
            for i in range(m):
                for j in range(m):
                    q = base + i * (m + 1) + j
                    c = [q, q + m + 1, q + m + 2, q + 1]
                    cells.append(c if side > 0 else c[::-1])
    meshgen.write_vtk(path, np.array(nodes), np.array(cells), 9)


@pytest.mark.parametrize("form", ["plain", "mixed"])
def test_blocks_of_zeros_end_in_no_result_and_nothing_sticks(tmp_path, form):
    """A block of zeros has no pivot (the reference divides by it and ends in an index
    out of range): no result is claimed, and the next build is what it was."""
    good = workloads.perturbed_sphere_input(str(tmp_path), 4, 400, [2.0])
    good["solver"] = {"Hierarchical": {"tolerance": 1e-6, "max_iterations": 1000, "leaf_size": 8, "eta": 4.0}}
    path = str(tmp_path / "box.vtk")
    flat_box(path, 8)
    flat = workloads.base_input(path, [100.0], method="Classical", solver=good["solver"],
                                field_points=np.array([[3.0, 0.0, 0.0]]))
    P = O.Problem(flat)
    A, bl = P.dense_surface()[0], O.block_list(P.cpts, 8, 4.0)
    blocks = [np.ix_(bl["rows"][bl["row_off"][i]:bl["row_off"][i + 1]], bl["cols"][bl["col_off"][i]:bl["col_off"][i + 1]])
              for i in np.flatnonzero(bl["admissible"])]
    assert any(not A[ix].any() for ix in blocks)
    ctx = bem.Context.default()

    def solve(inp):
        a = bem.Analysis(ctx)
        a.set_input(inp)
        a.run(form=form)
        return a.get_result()[0].scattered, a.reports[0]

    first = solve(good)
    for _ in range(2):
        try:
            got, rep = solve(flat)
        except bem.BemError:
            continue
        assert rep["flag"] == 2 or not np.isfinite(got).all()
    again = solve(good)
    assert np.array_equal(first[0], again[0]) and again[1]["flag"] == 1
