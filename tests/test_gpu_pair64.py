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


def extended(pd, ka_value):
    """Collocation points, unit normals, weights and wavenumber in extended precision."""
    q = np.longdouble
    cp = pd.get_cpts()
    normal = cp[:, 3:6].astype(q)
    normal /= np.sqrt((normal ** 2).sum(axis=1))[:, None]
    return cp[:, :3].astype(q), normal, (cp[:, 6] * cp[:, 7]).astype(q), \
        q(2.0 * 3.14159265358979323846 * ka_value / 343.0)


PI = np.longdouble(3.14159265358979323846) + np.longdouble(2.6433832795028842e-19)


@pytest.mark.parametrize("method", ["Classical", "BurtonMiller"])
@pytest.mark.parametrize("ka", [1e-3, 0.0245, 0.3, 7.0, 60.0])
def test_surface_matrices(tmp_path, ka, method):
    """G and H with all their terms.  Counted over the operations of a pair (root 2,
    weight 2, sine and cosine 2, direction cosines 8 each relative to one, products
    and sums) no term is further off than 40 u of its modulus with the direction
    cosines set to one, and 4 k r u for the phase."""
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no extended precision on this machine")
    nodes, tris = meshgen.perturbed_sphere(160, 5)
    path = str(tmp_path / "body.vtk")
    meshgen.write_vtk(path, nodes, tris, 5)
    inp = workloads.base_input(path, [ka * 343.0 / (2 * math.pi)], method=method, field_points=np.zeros((0, 3)))
    pd = bem.PreData.from_dict(inp)
    H, G = bem.get_dense_surface_matrices(pd)
    x, nr, wa, k = extended(pd, float(pd.frequencies[0]))
    d = x[None] - x[:, None]
    r = np.sqrt((d ** 2).sum(axis=2))
    off = ~np.eye(len(x), dtype=bool)
    r[~off] = 1
    m = wa / (4 * PI * r)
    g = m * (np.cos(k * r) + 1j * np.sin(k * r))
    f = -1 / r + 1j * k
    cy = (d * nr[:, None, :]).sum(axis=2) / r
    h, size_g, size_h = -g * f * cy, m, m * (1 / r + k)
    if method == "BurtonMiller":
        cx = (d * nr[None]).sum(axis=2) / r
        b = 1 / k
        t = (k * k * r - 3 / r + 3j * k) * cx * cy
        h = h + 1j * b * (g / r) * (-f * (nr @ nr.T) - t)
        g = g + 1j * b * g * f * cx
        size_g = size_g + b * m * (1 / r + k)
        size_h = size_h + b * m / r * (1 / r + k + k * k * r + 3 / r + 3 * k)
    u = (40 + 4 * (k * r)) * U
    assert np.all((np.abs(G - g) <= u * size_g)[off])
    assert np.all((np.abs(H - h) <= u * size_h)[off])


@pytest.mark.parametrize("n", [100, 700])
@pytest.mark.parametrize("ka", [1e-3, 0.3, 7.0, 60.0])
def test_field(tmp_path, ka, n):
    """The field's fused term: 40 + 4 k r units of its modulus with the direction cosine
    set to one, and the sums (n / 256 in turn, then eight in a tree)."""
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no extended precision on this machine")
    nodes, tris = meshgen.perturbed_sphere(n, 7)
    path = str(tmp_path / "body.vtk")
    meshgen.write_vtk(path, nodes, tris, 5)
    points = meshgen.fibonacci_points(37, 3.0)
    inp = workloads.base_input(path, [ka * 343.0 / (2 * math.pi)], field_points=points)
    pd = bem.PreData.from_dict(inp)
    rng = np.random.default_rng(n)
    phi, vn = (rng.normal(size=pd.n) + 1j * rng.normal(size=pd.n) for _ in range(2))
    out = bem.evaluate_field(pd, phi, vn)
    x, nr, wa, k = extended(pd, float(pd.frequencies[0]))
    d = np.asarray(points).astype(np.longdouble)[:, None] - x[None]
    r = np.sqrt((d ** 2).sum(axis=2))
    m = wa / (4 * PI * r)
    g = m * (np.cos(k * r) + 1j * np.sin(k * r))
    h = -g * (-1 / r + 1j * k) * (d * nr[None]).sum(axis=2) / r
    ref = (g * vn - h * phi).sum(axis=1)
    size = m * (np.abs(vn) + (1 / r + k) * np.abs(phi))
    bound = (size * (40 + 4 * k * r + n / 256 + 8)).sum(axis=1) * U
    assert np.all(np.abs(out - ref) <= bound)
