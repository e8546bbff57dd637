"""GMRES (csrc/gmres.cu, csrc/precond.cu) at the sizes where its tiles end: row
blocks of 64 and 512, column chunks of 512, Gram-Schmidt chunks of 64 to 512 rows,
preconditioner blocks of up to 64 in halves of 32, Arnoldi clusters of up to 16
CTAs with 128 rows each.

FP64: the stopping test gives ||r|| <= tol (||A||_F ||x|| + ||b||), so the error
against a direct solution is at most tol ||A^-1|| (||A||_F + ||A||) ||x||; with the
matrices below (||A^-1|| < 1, ||A||_F < 2.2 sqrt(n) + 1 < 60) it is under 1e-11 for
tol = 1e-13."""
import tempfile

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
bem = pytest.importorskip("cc_abstemious_gb300")
from cc_abstemious_gb300 import workloads  # noqa: E402


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 129, 511, 512, 513, 577, 700, 1023, 1025, 2047, 2049, 2600])
def test_fp64_sizes(n):
    rng = np.random.default_rng(n)
    A = 0.25 * (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))) / np.sqrt(n) + 2 * np.eye(n)
    b = rng.normal(size=n) + 1j * rng.normal(size=n)
    x, rep = bem.gmres(A, b, 1000, 1e-13)
    ref = np.linalg.solve(A, b)
    # the reported backward error is x's own
    err = np.linalg.norm(A @ x - b) / (np.linalg.norm(A) * np.linalg.norm(x) + np.linalg.norm(b))
    assert abs(err - rep["backward_error"]) <= (n + 8) * 2.0 ** -53 + 1e-12 * err
    # the reference allows n iterations in cycles of sqrt(n): too few for n = 1, 2
    assert rep["flag"] == 1 or n <= 2
    if n <= 2:
        return
    assert np.linalg.norm(x - ref) <= 2e-11 * np.linalg.norm(ref)


@pytest.mark.parametrize("form", ["mixed", "refined"])
@pytest.mark.parametrize("precond", [None, "block_jacobi"])
@pytest.mark.parametrize("n", [60, 64, 66, 130, 510, 514, 578])
def test_mixed_sizes(n, precond, form):
    """The stated accuracy of the forms against FP64 LU of the same operator."""
    inp = workloads.perturbed_sphere_input(tempfile.mkdtemp(prefix="bem_tiles_"), n, n, [1.0, 2.0], tol=1e-8)
    a = bem.Analysis(bem.Context.default())
    a.set_input(inp)
    a.run(form=form, precond=precond, check_vs_lu=True)
    for rep in a.reports:
        assert rep["flag"] == 1
        assert 0 <= rep["rel_err_vs_lu"] < 1e-6, rep


@pytest.mark.parametrize("waves", [2, 3])
@pytest.mark.parametrize("n", [2570, 3100])
def test_waves_share_an_operator(n, waves):
    """Sizes and counts at which the mixed form's products take the wide tiles, two
    right-hand sides per pass and, with three, one left over (8 or 12 systems of 36
    or 49 tiles): every wave to the form's accuracy, and converged by itself."""
    inp = workloads.perturbed_sphere_input(tempfile.mkdtemp(prefix="bem_waves_"), n, n, [1.0, 2.0, 3.0, 4.0], tol=1e-8)
    inp["incident_wave"] = {"PlaneWave": {"direction": [0.0, 0.0, 1.0], "amplitude": [1.0, 0.0]}}
    inp["additional_incident_waves"] = [
        {"SphericalWave": {"origin": [0.0, 0.0, 3.0], "amplitude": [0.5, 0.2]}},
        {"PlaneWave": {"direction": [1.0, 1.0, 0.0], "amplitude": [0.0, 1.0]}}][:waves - 1]
    a = bem.Analysis(bem.Context.default())
    a.set_input(inp)
    a.run(form="mixed", check_vs_lu=True)
    reports = [rep for r in a.reports_by_rhs for rep in r]
    assert len(reports) == 4 * waves
    for rep in reports:
        assert rep["flag"] == 1
        assert 0 <= rep["rel_err_vs_lu"] < 1e-6, rep
