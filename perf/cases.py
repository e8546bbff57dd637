"""The calls that users of this framework spend their time in, for measuring it.

A case is one call (or the short sequence that belongs together) through the
public entry points of `cc_abstemious_gb300`, on synthetic seeded bodies: the
seed changes the shape of the body, the direction of the wave and the surface
values.  Sizes are those of the workloads, tests and benchmark of this
repository: 324 triangles is the reference's own verification body, 6144 quads
and 40960 triangles are the benchmark's bodies, 500 to 5000 triangles its batch.

The kinds:

  analysis   Analysis: JSON input and VTK file on the host -> every frequency ->
             pressures at the field points and the surface solution on the host
  surface    solve_for_surface on a parsed problem (assembly and solver)
  lu         solve_lu of the caller's own dense matrix
  product    HMatrix.gemv, the compressed operator applied to a vector
  matrices   get_dense_surface_matrices into the caller's device tensors
  field      evaluate_field, a surface solution carried to a map of points
  batch      run_batch, several bodies and all their frequencies at once

The network of the learned preconditioner is trained once per family of bodies
and is not a call that a user repeats, so no case stands for it.
"""
import math
import os
import tempfile

import numpy as np
import torch

import cc_abstemious_gb300 as bem
from cc_abstemious_gb300 import meshgen

SOUND_SPEED = 343.0
DENSITY = 1.21
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def _case(name, kind, **more):
    c = {"name": name, "kind": kind, "form": "plain", "solver": "Direct", "precond": "none", "method": "BurtonMiller",
         "bc": "rigid", "shape": "tri", "elements": 0, "frequencies": 1, "ka_lo": 1.0, "ka_hi": 1.0, "points": 0,
         "waves": 1, "total": False, "tolerance": 1e-8}
    c.update(more)
    return c


def listed():
    return [
        # the smallest whole call: the reference's verification body, one
        # frequency, the default Direct solver in FP64, one field point
        _case("direct_324", "analysis", method="Classical", elements=324, ka_lo=0.2, ka_hi=0.2, points=1),
        # a small body in the batched form with a radiating surface (nonzero
        # normal velocity) and the cheap preconditioner, a few frequencies
        _case("mixed_1280x4", "analysis", form="mixed", precond="block_jacobi", bc="velocity", elements=1280,
              frequencies=4, ka_lo=0.5, ka_hi=3.0, points=100, tolerance=1e-10),
        # the default Direct solver on the benchmark's body with an absorbing
        # surface: assembly and the dense FP64 LU of a large matrix
        _case("direct_6144", "surface", bc="impedance", shape="quad", elements=6144, ka_lo=4.0, ka_hi=4.0),
        # the dense FP64 solver alone on a caller's matrix of an odd size
        _case("lu_2001", "lu", elements=2001),
        # the reference's Iterative solver in FP64 on the benchmark's body
        _case("iterative_6144", "surface", solver="Iterative", shape="quad", elements=6144, ka_lo=5.5, ka_hi=5.5),
        # the reference's Hierarchical solver with its default tree and ACA
        # settings: building the H-matrix and iterating on it
        _case("hierarchical_2560", "surface", solver="Hierarchical", method="Classical", elements=2560, ka_lo=1.0,
              ka_hi=1.0, tolerance=1e-6),
        # products with a compressed operator (the benchmark's tree settings)
        _case("product_10240", "product", solver="HierarchicalFine", elements=10240, ka_lo=5.0, ka_hi=5.0),
        # both FP64 influence matrices for the caller's own algebra
        _case("matrices_4002", "matrices", elements=4002, ka_lo=3.0, ka_hi=3.0),
        # a pressure map around a solved body, far more points than elements
        _case("field_20000", "field", shape="quad", elements=6144, ka_lo=6.0, ka_hi=6.0, points=20000, total=True,
              bc="velocity"),
        # the headline: 16 frequencies of the benchmark's body in one batch
        _case("mixed_6144x16", "analysis", form="mixed", solver="Iterative", shape="quad", elements=6144,
              frequencies=16, ka_lo=1.0, ka_hi=10.0, points=100),
        # a fleet of uneven absorbing bodies with the strong preconditioner
        _case("batch_12x8", "batch", form="mixed", precond="lu", bc="impedance", elements=5000, bodies=12,
              frequencies=8, ka_lo=0.5, ka_hi=8.0, points=100, tolerance=1e-10),
        # the largest: the benchmark's ellipsoid under a plane wave and a
        # point source, rounded operators and the strong preconditioner
        _case("ellipsoid_40960x2", "analysis", form="mixed_rounded", precond="lu", shape="ellipsoid", elements=40960,
              frequencies=2, ka_lo=5.0, ka_hi=17.5, points=100, waves=2, tolerance=1e-10),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["direct", "direct", "lu", "lu", "iterative", "hierarchical", "product", "matrices", "field",
                       "mixed", "mixed", "batch"])
    ka = round(rng.uniform(0.3, 6.0), 3)
    if kind == "direct":
        c = _case("", rng.choice(["analysis", "surface"]), method=rng.choice(["Classical", "BurtonMiller"]),
                  bc=rng.choice(["rigid", "velocity", "impedance"]), elements=_size(rng, 200, 4000), ka_lo=ka,
                  ka_hi=ka, points=_size(rng, 1, 300), total=rng.random() < 0.5)
    elif kind == "lu":
        c = _case("", "lu", elements=_size(rng, 50, 3500))
    elif kind == "iterative":
        c = _case("", "surface", solver="Iterative", shape="quad", elements=_size(rng, 400, 6144), ka_lo=ka, ka_hi=ka)
    elif kind == "hierarchical":
        c = _case("", "surface", solver="Hierarchical", method="Classical", elements=_size(rng, 400, 4000),
                  ka_lo=ka / 3, ka_hi=ka / 3, tolerance=1e-6)
    elif kind == "product":
        c = _case("", "product", solver=rng.choice(["Hierarchical", "HierarchicalFine"]),
                  elements=_size(rng, 800, 10240), ka_lo=ka, ka_hi=ka)
    elif kind == "matrices":
        c = _case("", "matrices", method=rng.choice(["Classical", "BurtonMiller"]), shape=rng.choice(["tri", "quad"]),
                  elements=_size(rng, 300, 6000), ka_lo=ka, ka_hi=ka)
    elif kind == "field":
        c = _case("", "field", shape=rng.choice(["tri", "quad"]), elements=_size(rng, 300, 6144), ka_lo=ka, ka_hi=ka,
                  points=_size(rng, 50, 20000), total=rng.random() < 0.5, bc=rng.choice(["velocity", "impedance"]))
    elif kind == "mixed":
        c = _case("", "analysis", form=rng.choice(["mixed", "mixed", "mixed_rounded", "refined"]),
                  precond=rng.choice(["none", "block_jacobi", "lu"]), solver=rng.choice(["Direct", "Iterative"]),
                  bc=rng.choice(["rigid", "velocity", "impedance"]), shape=rng.choice(["tri", "quad"]),
                  elements=_size(rng, 300, 5000), frequencies=rng.randint(1, 16), ka_lo=0.5,
                  ka_hi=round(rng.uniform(1.0, 6.0), 3), points=_size(rng, 1, 300), waves=rng.choice([1, 1, 2, 3]),
                  tolerance=1e-10)
    else:
        c = _case("", "batch", form="mixed", precond=rng.choice(["lu", "block_jacobi"]), bc="impedance",
                  elements=_size(rng, 700, 5000), bodies=rng.randint(2, 12), frequencies=rng.randint(1, 8), ka_lo=0.5,
                  ka_hi=round(rng.uniform(1.0, 8.0), 3), points=_size(rng, 1, 200), tolerance=1e-10)
    del c["name"]
    return c


# ---- inputs ------------------------------------------------------------------
def _mesh(shape, elements, seed):
    """(nodes, cells, VTK cell type) of a body of about `elements` elements."""
    if shape == "tri":
        nodes, cells = meshgen.perturbed_sphere(elements, seed)
        return nodes, cells, 5
    rng = np.random.default_rng(seed)
    if shape == "ellipsoid":
        lon = 2 * max(2, int(round(math.sqrt(elements / 2.5) / 2)))
        nodes, cells = meshgen.uv_ellipsoid((2.0, 1.0, 0.5), lon, elements // (2 * lon) + 1)
        return nodes * (1.0 + 0.1 * rng.random(3)), cells, 5
    nodes, cells = meshgen.cube_sphere(max(2, int(round(math.sqrt(elements / 6.0)))))
    r = 1.0
    for _ in range(3):  # a few smooth bumps, unlike on every seed
        d = rng.normal(size=3)
        r = r + 0.03 * (nodes @ (d / np.linalg.norm(d))) ** 2
    return nodes * np.asarray(r)[:, None], cells, 9


def _input(case, path, seed):
    rng = np.random.default_rng(seed + 7)
    d = rng.normal(size=3)
    d /= np.linalg.norm(d)
    wave = {"PlaneWave": {"direction": d.tolist(), "amplitude": [1.0, 0.0]}}
    point = {"SphericalWave": {"origin": [0.0, 0.0, 3.0], "amplitude": [1.0, 0.0]}}
    turned = {"PlaneWave": {"direction": (-d).tolist(), "amplitude": [0.5, 0.5]}}
    tol = {"tolerance": case["tolerance"], "max_iterations": 2500}
    solver = {"Direct": {"Direct": {}}, "Iterative": {"Iterative": tol},
              "Hierarchical": {"Hierarchical": tol},
              "HierarchicalFine": {"Hierarchical": dict(tol, leaf_size=64, eta=1.0, aca_tolerance=1e-5)}}
    bc = {"rigid": ("NormalVelocity", [0.0, 0.0]), "velocity": ("NormalVelocity", [1.0, 0.2]),
          "impedance": ("Impedance", [DENSITY * SOUND_SPEED, 0.2 * DENSITY * SOUND_SPEED])}[case["bc"]]
    radius = 2.0 if case["shape"] == "ellipsoid" else 1.0
    kas = np.linspace(case["ka_lo"], case["ka_hi"], case["frequencies"])
    inp = {"mesh_file": path, "body_index": 1,
           "frequency": {"List": {"values": [float(k) * SOUND_SPEED / (2 * math.pi * radius) for k in kas]}},
           "sound_speed": SOUND_SPEED, "mass_density": DENSITY, "problem_type": "Exterior",
           "method_type": case["method"], "solver": solver[case["solver"]], "incident_wave": wave,
           "surface_bc": {"bc_type": bc[0], "value": bc[1]},
           "output": {"o_type": "Total" if case["total"] else "Scattered", "field": "Pressure", "file": "",
                      "field_points": (meshgen.fibonacci_points(case["points"], 5.0) * (1.0 + rng.random((
                          case["points"], 1)))).tolist() if case["points"] else []}}
    if case["waves"] > 1:
        inp["additional_incident_waves"] = [point, turned][:case["waves"] - 1]
    return inp


def _body_sizes(case, seed):
    """Element counts of the bodies of a batch: 500 up to `elements`, the largest among them."""
    rng = np.random.default_rng(seed + 3)
    return [case["elements"]] + [int(t) for t in rng.integers(500, case["elements"] + 1, size=case["bodies"] - 1)]


def _matrix(case, seed):
    g = torch.Generator().manual_seed(seed)
    n = case["elements"]
    return (torch.randn(n, n, dtype=torch.complex128, generator=g),
            torch.randn(n, dtype=torch.complex128, generator=g))


def _vectors(count, n, seed):
    rng = np.random.default_rng(seed + 11)
    return [rng.normal(size=n) + 1j * rng.normal(size=n) for _ in range(count)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "lu":
        A, b = _matrix(case, seed)
        return {"kind": kind, "A": np.asfortranarray(A.numpy()), "b": b.numpy()}
    folder = tempfile.TemporaryDirectory(prefix="bem_case_")
    state = {"kind": kind, "case": case, "folder": folder}
    if kind == "batch":
        inputs = []
        for b, t in enumerate(_body_sizes(case, seed)):
            path = os.path.join(folder.name, "body_%d.vtk" % b)
            nodes, cells, cell_type = _mesh("tri", t, 100 * seed + b)
            meshgen.write_vtk(path, nodes, cells, cell_type)
            inputs.append(_input(case, path, seed + b))
        state["problems"] = [bem.PreData.from_dict(i) for i in inputs]
        return state
    path = os.path.join(folder.name, "body.vtk")
    nodes, cells, cell_type = _mesh(case["shape"], case["elements"], seed)
    meshgen.write_vtk(path, nodes, cells, cell_type)
    inp = _input(case, path, seed)
    if kind == "analysis":
        state["input"] = inp
        return state
    pd = state["problem"] = bem.PreData.from_dict(inp)
    if kind == "surface":
        state["rhs"] = bem.get_incident_surface(pd)
    elif kind == "product":
        state["operator"] = bem.HMatrix(pd)
        state["x"], state["b"] = _vectors(2, pd.n, seed)
    elif kind == "matrices":
        # column-major n x n matrices, as the entry point fills them
        state["out"] = tuple(torch.empty((pd.n, pd.n), dtype=torch.complex128, device=DEVICE).t() for _ in range(2))
    elif kind == "field":
        state["phi"], state["vn"] = _vectors(2, pd.n, seed)
        state["incident"] = bem.get_incident_field(pd)
    return state


def run(state):
    kind = state["kind"]
    if kind == "lu":
        return bem.solve_lu(state["A"], state["b"])
    if kind == "analysis":
        case = state["case"]
        a = bem.Analysis()
        a.set_input(state["input"])
        a.run(form=case["form"], precond=case["precond"])
        phi, vn = a.surface_solution()
        return {"scattered": np.stack([r.scattered for w in a.results_by_rhs for r in w]),
                "incident": np.stack([r.incident for w in a.results_by_rhs for r in w]), "phi": phi, "vn": vn}
    if kind == "batch":
        out = bem.run_batch(state["problems"], precond=state["case"]["precond"])
        return {"scattered": np.stack([r.scattered for results, _ in out for r in results]),
                "incident": np.stack([r.incident for results, _ in out for r in results])}
    pd = state["problem"]
    if kind == "surface":
        phi, vn, _ = bem.solve_for_surface(pd, state["rhs"])
        return {"phi": phi, "vn": vn}
    if kind == "product":
        return state["operator"].gemv(0.7 - 0.2j, state["x"], 0.3 + 0.1j, state["b"])
    if kind == "matrices":
        return dict(zip("HG", bem.get_dense_surface_matrices(pd, out=state["out"])))
    return bem.evaluate_field(pd, state["phi"], state["vn"], state["incident"])


# ---- what a pass cannot do without ------------------------------------------------
def _count(case):
    if case["shape"] == "quad":
        return 6 * max(2, int(round(math.sqrt(case["elements"] / 6.0)))) ** 2
    return case["elements"] + case["elements"] % 2


def work(case):
    """Real arithmetic: 8 n^3 / 3 for a dense complex LU, 8 for a complex
    multiply-add, about 60 for one pair of the Green's function and its
    derivatives.  Bytes: geometry and vectors in, results out; no operator,
    which a path may form again and need not store."""
    kind, n = case["kind"], _count(case)
    pair = 60.0
    if kind == "lu":
        n = case["elements"]
        return {"bytes": 16.0 * n * n + 32.0 * n, "flops": 8.0 * n ** 3 / 3}
    if kind == "matrices":
        return {"bytes": 72.0 * n + 32.0 * n * n, "flops": pair * n * n}
    if kind == "field":
        m = case["points"]
        return {"bytes": 104.0 * n + 56.0 * m, "flops": (pair + 16.0) * n * m}
    if kind == "product":
        # stored entries of 16 bytes: 27 million of 10240 rows at the benchmark's
        # tree settings, fewer at the reference's
        stored = (200.0 if case["solver"] == "HierarchicalFine" else 60.0) * math.log2(n) * n
        return {"bytes": 16.0 * stored + 48.0 * n, "flops": 8.0 * stored}
    sizes = [n]
    if kind == "batch":  # the mean of the sizes drawn from the seed
        sizes = [case["elements"]] + [(500 + case["elements"]) // 2] * (case["bodies"] - 1)
    flops = nbytes = 0.0
    for s in sizes:
        systems = case["frequencies"] * case["waves"]
        flops += case["frequencies"] * pair * s * s + systems * (2 * 8.0 * s * s + 76.0 * s * case["points"])
        if case["solver"] == "Direct" and case["form"] == "plain" or case["precond"] == "lu":
            flops += case["frequencies"] * 8.0 * s ** 3 / 3
        nbytes += 72.0 * s + systems * (48.0 * s + 32.0 * case["points"])
    if case["solver"] == "Hierarchical" and kind == "surface":  # near blocks only, then a product per step
        flops = 400.0 * n * (pair + 10 * 8.0)
    return {"bytes": nbytes, "flops": flops}


# ---- the same results in plain FP64 --------------------------------------------------
def _collocation(nodes, cells, cell_type):
    """Points, unit normals, areas and the one-point rule's weight."""
    p = torch.as_tensor(np.asarray(nodes)[cells], dtype=torch.float64, device=DEVICE)
    x = p.mean(dim=1)
    if cell_type == 5:
        normal = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
        size = torch.linalg.vector_norm(normal, dim=1)
        return x, normal / size[:, None], 0.5 * size, 1.0
    u = 0.25 * (p[:, 1] + p[:, 2] - p[:, 0] - p[:, 3])
    v = 0.25 * (p[:, 2] + p[:, 3] - p[:, 0] - p[:, 1])
    normal = torch.linalg.cross(u, v)
    size = torch.linalg.vector_norm(normal, dim=1)
    return x, normal / size[:, None], 0.25 * size, 4.0


def _green(src, src_n, obs, obs_n, k, coupling):
    """G and H of every (observation row, source column): the Helmholtz kernel
    and its derivative along the observation normal, plus `coupling` times
    their derivatives along the source normal (Burton-Miller)."""
    d = src[None, :, :] - obs[:, None, :]
    r = torch.linalg.vector_norm(d, dim=2)
    inv = torch.where(r > 0, 1.0 / r, torch.zeros_like(r))
    g = torch.polar(inv / (4 * math.pi), k * r)
    f = torch.complex(-inv, torch.full_like(inv, k))
    along_obs = (d * obs_n[:, None, :]).sum(dim=2) * inv
    gf = g * f
    h = -gf * along_obs
    if coupling:
        along_src = (d * src_n[None, :, :]).sum(dim=2) * inv
        nn = obs_n @ src_n.T
        t = torch.complex(k * k * r - 3 * inv, torch.full_like(r, 3 * k)) * (along_src * along_obs)
        h = h + coupling * (g * inv) * (-f * nn - t)
        g = g + coupling * gf * along_src
    return g, h


def _surface_matrices(case, geometry, k):
    x, normal, area, wt = geometry
    n = len(area)
    coupling = 1j / k if case["method"] == "BurtonMiller" else 0.0
    H = torch.empty((n, n), dtype=torch.complex128, device=DEVICE)
    G = torch.empty_like(H)
    for i in range(0, n, 1024):
        g, h = _green(x, normal, x[i:i + 1024], normal[i:i + 1024], k, coupling)
        G[i:i + 1024], H[i:i + 1024] = g * (wt * area), h * (wt * area)
    b = torch.sqrt(area / math.pi)
    own_g = (wt * area / (2 * math.pi * b)).to(torch.complex128)
    own_h = torch.full_like(own_g, -0.5)
    if coupling:
        own_h = own_h - coupling * wt * area / (2 * math.pi * b ** 3)
        own_g = own_g + 0.5 * coupling
    i = torch.arange(n, device=DEVICE)
    G[i, i], H[i, i] = own_g, own_h
    return H, G


def _incident(wave, x, normal, k, omega, coupling):
    kind, w = next(iter(wave.items()))
    v = torch.tensor(w["direction" if kind == "PlaneWave" else "origin"], dtype=torch.float64, device=DEVICE)
    v = v / torch.linalg.vector_norm(v)
    amp = complex(*w["amplitude"]) / (1j * omega * DENSITY)
    if kind == "PlaneWave":
        phi = amp * torch.polar(torch.ones(len(x), dtype=torch.float64, device=DEVICE), k * (x @ v))
        slope = 1j * k * phi * (normal @ v) if normal is not None else None
    else:
        d = x - v
        r = torch.linalg.vector_norm(d, dim=1)
        phi = amp * torch.polar(1.0 / (4 * math.pi * r), k * r)
        slope = phi * torch.complex(-1.0 / r, torch.full_like(r, k)) * (d * normal).sum(1) / r if normal is not None \
            else None
    return phi + coupling * slope if coupling and slope is not None else phi


def _solve(case, inp, geometry, values, waves):
    """Surface potential and normal velocity of every wave at one frequency."""
    x, normal, _, _ = geometry
    omega = 2 * math.pi * values
    k = omega / SOUND_SPEED
    coupling = 1j / k if case["method"] == "BurtonMiller" else 0.0
    H, G = _surface_matrices(case, geometry, k)
    value = complex(*inp["surface_bc"]["value"])
    rhs = torch.stack([-_incident(w, x, normal, k, omega, coupling) for w in waves], dim=1)
    if case["bc"] == "impedance":
        factor = -1j * omega * DENSITY / value
        H += factor * G
    elif value:
        rhs += value * G.sum(dim=1, keepdim=True)
    del G
    phi = torch.linalg.solve(H, rhs).T.contiguous()
    vn = factor * phi if case["bc"] == "impedance" else torch.full_like(phi, value)
    return phi, vn


def _field(inp, geometry, points, phi, vn, wave, frequency):
    x, normal, area, wt = geometry
    omega = 2 * math.pi * frequency
    k = omega / SOUND_SPEED
    inc = _incident(wave, points, None, k, omega, 0.0)
    out = []
    for i in range(0, len(points), 1024):
        # the field point is the source of the kernel, the element's normal the observer's
        g, h = _green(points[i:i + 1024], None, x, normal, k, 0.0)
        g, h = g * (wt * area)[:, None], h * (wt * area)[:, None]
        out.append(vn @ g - phi @ h)
    out = torch.cat(out) if out else inc
    return (inc + out if inp["output"]["o_type"] == "Total" else out), inc


def _analysis_exact(case, inp, mesh):
    geometry = _collocation(*mesh)
    waves = [inp["incident_wave"]] + inp.get("additional_incident_waves", [])
    points = torch.as_tensor(inp["output"]["field_points"], dtype=torch.float64, device=DEVICE).reshape(-1, 3)
    frequencies = inp["frequency"]["List"]["values"]
    parts = {}
    for f, hz in enumerate(frequencies):
        phi, vn = _solve(case, inp, geometry, hz, waves)
        for r, w in enumerate(waves):
            sc, inc = _field(inp, geometry, points, phi[r], vn[r], w, hz)
            pressure = 2j * math.pi * hz * DENSITY
            parts[r, f] = (pressure * sc, pressure * inc, phi[r], vn[r])
    rows = [parts[r, f] for r in range(len(waves)) for f in range(len(frequencies))]
    return [torch.stack([row[q] for row in rows]).cpu().numpy() for q in range(4)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "lu":
        A, b = _matrix(case, seed)
        return torch.linalg.solve(A.to(DEVICE), b.to(DEVICE)).cpu().numpy()
    if kind == "batch":
        sizes = _body_sizes(case, seed)
        if case["frequencies"] * sum(8.0 * t ** 3 / 3 for t in sizes) > 1e13:
            return None
        rows = []
        for b, t in enumerate(sizes):
            mesh = _mesh("tri", t, 100 * seed + b)
            rows.append(_analysis_exact(case, _input(case, "", seed + b), mesh))
        return {"scattered": np.concatenate([r[0] for r in rows]), "incident": np.concatenate([r[1] for r in rows])}
    if kind in ("analysis", "surface") and case["frequencies"] * 8.0 * _count(case) ** 3 / 3 > 1.5e13:
        return None
    mesh = _mesh(case["shape"], case["elements"], seed)
    inp = _input(case, "", seed)
    if kind == "analysis":
        return dict(zip(("scattered", "incident", "phi", "vn"), _analysis_exact(case, inp, mesh)))
    geometry = _collocation(*mesh)
    hz = inp["frequency"]["List"]["values"][0]
    if kind == "surface":
        phi, vn = _solve(case, inp, geometry, hz, [inp["incident_wave"]])
        return {"phi": phi[0].cpu().numpy(), "vn": vn[0].cpu().numpy()}
    if kind == "matrices":
        return dict(zip("HG", _surface_matrices(case, geometry, 2 * math.pi * hz / SOUND_SPEED)))
    n = len(geometry[2])
    u, v = (torch.as_tensor(t, device=DEVICE) for t in _vectors(2, n, seed))
    if kind == "product":
        H, _ = _surface_matrices(case, geometry, 2 * math.pi * hz / SOUND_SPEED)
        return ((0.7 - 0.2j) * (H @ u) + (0.3 + 0.1j) * v).cpu().numpy()
    points = torch.as_tensor(inp["output"]["field_points"], dtype=torch.float64, device=DEVICE)
    return _field(inp, geometry, points, u, v, inp["incident_wave"], hz)[0].cpu().numpy()
