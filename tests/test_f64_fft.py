"""The float64 operator on its own transforms (precision 'fp64'): every radix, prime axes, odd lengths (no Nyquist bin),
even ones in each axis (its coupling rule, the two-line and three-line columns), blocks that are cut short, odd row
counts, and the cuFFT fallback above the largest prime, all against the oracle's complex pipeline.  Tolerance: 1e-12
relative (max-norm), the float64 operators' bar."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(24, 24, 24), (25, 25, 25), (31, 26, 27), (86, 22, 36), (64, 48, 40), (45, 50, 32), (16, 17, 254), (127, 16, 18),
         (131, 16, 16), (108, 18, 20), (22, 33, 49), (17, 19, 23), (20, 16, 96)]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("nrhs", [1, 4])
def test_fp64_matvec_against_oracle(grid, nrhs):
    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    from mutual_polarization_slab_gb300.workloads import rsa
    from oracle import ewald_oracle as ew
    x, box, _ = rsa(60, 0.1, seed=5)
    xi, rc, P = 0.7, 0.45 * box[0], 7
    eps = np.full(60, 12.0)
    with SpectralEwaldSystem(x, eps, box, xi, rc, grid, P, *gcap.default_table(xi), slab_factor=0.0, max_rhs=nrhs) as s:
        m = np.random.default_rng(1).standard_normal((nrhs, 60, 3))
        out = s.matvec(m, precision="fp64").cpu().numpy()
    pn, pa, rvn = ew.default_table(xi)
    g = ew.Geometry(x, eps, box, xi, rc, grid, P, pn, pa, rvn, slab_factor=0.0)
    ref = np.stack([g.field_real(v) for v in m])
    assert np.abs(out - ref).max() <= 1e-12 * np.abs(ref).max()
