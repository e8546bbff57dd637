"""The FP64 kernel functions (csrc/kernels.cuh: root, phase, sine and cosine in
64-bit integers) against extended precision, across the ranges where their parts
change over: phases of 2^-10 turns and below (the FP64 path), quarter turns, many
turns, bodies of very small and very large scale.

Bounds, fixed beforehand: the separation enters with a relative error of 2 u, the
phase k r with that of r and k, so an entry is within (8 + 4 k r) u of its modulus
(u = 2^-53); factors for the cancellation in the direction cosines are avoided by
comparing G of the classical kernel, whose modulus has none."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
bem = pytest.importorskip("cc_abstemious_gb300")
from cc_abstemious_gb300 import meshgen, workloads  # noqa: E402

U = 2.0 ** -53


@pytest.mark.parametrize("scale", [1e-12, 1.0, 1e9])
@pytest.mark.parametrize("ka", [1e-9, 1e-3, 0.0245, 0.3, math.pi / 2, 7.0, 60.0, 3000.0])
def test_green_function(tmp_path, ka, scale):
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no extended precision on this machine")
    nodes, tris = meshgen.perturbed_sphere(120, 3)
    path = str(tmp_path / "body.vtk")
    meshgen.write_vtk(path, nodes * scale, tris, 5)
    inp = workloads.base_input(path, [ka * 343.0 / (2 * math.pi * scale)], method="Classical", field_points=np.zeros((0, 3)))
    pd = bem.PreData.from_dict(inp)
    H, G = bem.get_dense_surface_matrices(pd)
    cp = pd.get_cpts()
    q = np.longdouble
    x, wa = cp[:, :3].astype(q), (cp[:, 6] * cp[:, 7]).astype(q)
    pi = q(3.14159265358979323846) + q(2.6433832795028842e-19) * (np.finfo(q).nmant > 63)
    k = q(2.0 * 3.14159265358979323846 * float(pd.frequencies[0]) / 343.0)
    d = x[None] - x[:, None]
    r = np.sqrt((d ** 2).sum(axis=2))
    off = ~np.eye(len(x), dtype=bool)
    r[~off] = 1
    g = wa / (4 * pi * r)
    re, im = g * np.cos(k * r), g * np.sin(k * r)
    err = np.hypot((G.real - re).astype(float), (G.imag - im).astype(float)) / np.abs(g).astype(float)
    bound = (8 + 4 * (k * r).astype(float)) * U
    assert np.all(err[off] <= bound[off])
    # the imaginary part keeps its own digits where the phase is small
    small = off & ((k * r).astype(float) < 1e-2)
    rel = np.abs((G.imag - im).astype(float)) / np.abs(im).astype(float)
    assert np.all(rel[small] <= 16 * U)
