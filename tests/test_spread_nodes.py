"""The float64 and double-float node spread and the contractions against the oracle where their tiles could go wrong:
grids that are no multiple of the 8-node tile, of exactly one or two tiles, smaller than stencil plus tile, tile lists of
0, 1, 32, 96, 97 and several hundred particles, one to seven vectors (groups of three), the largest support, both tile
depths.  Tolerance: 1e-12 relative (max-norm), the float64 operators' bar.  The double-float grids keep eta below 1:
above it the Green's coefficient grows with k and amplifies the grid's rounding (by 1e5 on 16^3 with P = 16)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(grid, P, n, nrhs, clustered, precision):
    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    from oracle import ewald_oracle as ew
    rng = np.random.default_rng(n + P)
    box = np.array([60.0, 55.0, 65.0])
    # positions only have to be distinct here; clustered ones crowd a few tiles, and wrap round the box
    g = np.stack(np.meshgrid(*[np.arange(14)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x = (g[rng.permutation(len(g))[:n]] + rng.uniform(-0.3, 0.3, (n, 3))) * (box / 14 if not clustered else 0.9)
    x = np.mod(x - 3.0, box)
    xi, rc = 0.5, 0.3
    eps = rng.uniform(3.0, 9.0, n)
    m = rng.standard_normal((nrhs, n, 3))
    with SpectralEwaldSystem(x, eps, box, xi, rc, grid, P, *gcap.default_table(xi), slab_factor=0.0, max_rhs=nrhs) as s:
        out = s.matvec(m, precision=precision).cpu().numpy()
        again = s.matvec(m, precision=precision).cpu().numpy()
    np.testing.assert_array_equal(out, again)          # fixed summation order
    pn, pa, rvn = ew.default_table(xi)
    geo = ew.Geometry(x, eps, box, xi, rc, grid, P, pn, pa, rvn, slab_factor=0.0)
    ref = np.stack([geo.field_real(v) for v in m])
    assert np.abs(out - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("grid,P,n,nrhs", [
    ((8, 8, 8), 6, 97, 1), ((16, 16, 16), 16, 33, 2), ((17, 9, 25), 9, 1, 3), ((24, 33, 10), 10, 96, 4),
    ((40, 40, 40), 5, 500, 7), ((96, 96, 96), 8, 300, 1), ((72, 64, 80), 10, 400, 3), ((12, 12, 13), 12, 700, 2),
])
@pytest.mark.parametrize("clustered", [False, True])
def test_float64_nodes(grid, P, n, nrhs, clustered):
    _check(grid, P, n, nrhs, clustered, "fp64")


@pytest.mark.parametrize("grid,P,n,nrhs", [
    ((40, 40, 48), 4, 500, 7), ((96, 96, 96), 8, 300, 1), ((72, 64, 80), 10, 400, 3), ((90, 45, 50), 5, 97, 4),
    ((54, 75, 60), 6, 1, 2), ((96, 90, 100), 16, 33, 1),
])
@pytest.mark.parametrize("clustered", [False, True])
def test_double_float_nodes(grid, P, n, nrhs, clustered):
    _check(grid, P, n, nrhs, clustered, "df")
