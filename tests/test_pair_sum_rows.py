"""Pair sums where a row's lanes change.  Float64: vectors in and beyond full groups of four, rows of few and many pairs, on
both sides of the rule.  Float32: one to seven vectors, rows on both sides of the wide form's limit, a last warp with rows
missing, rows without pairs.  Tolerances: 1e-12 and 2e-5 relative (max-norm), the operators' bars."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compare(n, rc, nrhs, precision, tol, spacing=2.3):
    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    from oracle import ewald_oracle as ew
    rng = np.random.default_rng(n + nrhs)
    k = max(5, int(np.ceil(n ** (1 / 3))))
    box = np.full(3, spacing * k)
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x = np.mod(spacing * g[rng.permutation(len(g))[:n]] + rng.uniform(-0.1, 0.1, (n, 3)), box)
    xi, eps = 0.5, np.full(n, 7.0)
    grid = (30, 32, 36) if precision == "fp64" else (40, 42, 44)
    m = rng.standard_normal((nrhs, n, 3))
    with SpectralEwaldSystem(x, eps, box, xi, rc, grid, 8, *gcap.default_table(xi), slab_factor=1.0, max_rhs=nrhs) as s:
        out = s.matvec(m, precision=precision).cpu().numpy()
    geo = ew.Geometry(x, eps, box, xi, rc, grid, 8, *ew.default_table(xi), slab_factor=1.0)
    for r in sorted({0, nrhs // 2, nrhs - 1}):
        ref = geo.field_real(m[r])
        assert np.abs(out[r] - ref).max() <= tol * np.abs(ref).max(), r


@pytest.mark.parametrize("n,rc,nrhs", [(800, 3.0, 7), (800, 3.0, 8), (800, 3.0, 12), (800, 5.2, 12), (800, 5.2, 20),
                                       (1700, 3.0, 6)])
def test_float64(n, rc, nrhs):
    _compare(n, rc, nrhs, "fp64", 1e-12)


@pytest.mark.parametrize("n", [1, 5, 5000, 5003])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 7])
def test_float32(n, nrhs):
    _compare(n, 3.0, nrhs, "fp32", 2e-5)


@pytest.mark.parametrize("nrhs", [1, 3])
def test_float32_rows_without_pairs(nrhs):
    _compare(5501, 2.45, nrhs, "fp32", 2e-5, spacing=2.5)
