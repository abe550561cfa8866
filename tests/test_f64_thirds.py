"""Float64 transforms of axes whose prime factors split into thirds (31, 43, 61, 67, 79, 97, 103): as x, y and z axis, alone
(no twiddles), twice and with other factors, against the oracle's complex pipeline.  Tolerance: 1e-12 relative (max-norm),
the float64 operators' bar; grids with eta below 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(31, 8, 10), (8, 43, 9), (9, 10, 61), (67, 6, 8), (6, 79, 8), (8, 6, 97), (103, 8, 6),
                                  (62, 86, 31), (961, 6, 7), (8, 7, 806), (43, 31, 122), (6, 93, 129)])
@pytest.mark.parametrize("nrhs", [1, 4])
def test_against_oracle(grid, nrhs):
    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    from oracle import ewald_oracle as ew
    rng = np.random.default_rng(sum(grid))
    box, xi, P, n, rc = 0.8 * np.array(grid), 0.6, 6, 40, 0.3
    x, m, eps = rng.uniform(0, 1, (n, 3)) * box, rng.standard_normal((nrhs, n, 3)), np.full(n, 5.0)
    with SpectralEwaldSystem(x, eps, box, xi, rc, grid, P, *gcap.default_table(xi), slab_factor=0.0, max_rhs=nrhs) as s:
        out = s.matvec(m, precision="fp64").cpu().numpy()
    pn, pa, rvn = ew.default_table(xi)
    g = ew.Geometry(x, eps, box, xi, rc, grid, P, pn, pa, rvn, slab_factor=0.0)
    ref = np.stack([g.field_real(v) for v in m])
    assert np.abs(out - ref).max() <= 1e-12 * np.abs(ref).max()
