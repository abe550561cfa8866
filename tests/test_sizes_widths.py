"""Polydisperse spread of one to nine vectors: passes of one, two, four and eight vectors, full and not.  Tolerances: 1e-11
(float64) and 2e-5 (float32) relative (max-norm), the operator's bars."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("fp32", 2e-5)])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 4, 5, 9])
def test_widths(nrhs, precision, tol):
    from mutual_polarization_slab_gb300 import sizes as gs
    from mutual_polarization_slab_gb300.workloads import rsa
    from oracle import polydisperse_oracle as po
    n, xi, grid, P = 41, 0.6, (30, 31, 33), 7
    x, box, _ = rsa(n, 0.1, seed=9)
    rng = np.random.default_rng(nrhs)
    radii, lam = rng.uniform(0.6, 1.0, n), rng.uniform(3.0, 9.0, n)
    p = rng.standard_normal((nrhs, n, 3)) * 10.0 ** rng.integers(-3, 4, (nrhs, 1, 1))
    ref = po.PolyGeometry(x, radii, lam, box, xi, 1e-2, Ngrid=grid, P=P)
    with gs.PolydisperseSystem(x, radii, lam, box, xi, 1e-2, Ngrid=grid, P=P, max_rhs=nrhs) as s:
        out = s.matvec(p, precision=precision).cpu().numpy()
    for r in range(nrhs):
        want = ref.field(p[r])
        assert np.abs(out[r] - want).max() <= tol * np.abs(want).max(), r
