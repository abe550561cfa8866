"""Pair sums of the float64 and double-float operators on both sides of the rule between a warp a row and vector and eight
lanes a row: particles and vectors just below and above it, rows of few and many pairs.  Tolerance: 1e-12 relative
(max-norm), the float64-accurate operators' bar."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rc,nrhs", [(1450, 3.0, 3), (1600, 3.0, 3), (1600, 5.2, 2), (2560, 5.2, 1), (240, 3.0, 24),
                                       (260, 3.0, 24), (260, 5.2, 24), (1, 3.0, 4)])
def test_pair_sums(n, rc, nrhs):
    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    from oracle import ewald_oracle as ew
    rng = np.random.default_rng(n)
    k = max(5, int(np.ceil(n ** (1 / 3))))
    box = np.full(3, 2.3 * k)
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x = np.mod(2.3 * g[rng.permutation(len(g))[:n]] + rng.uniform(-0.1, 0.1, (n, 3)), box)
    xi, grid, P, eps = 0.5, (30, 32, 36), 8, np.full(n, 7.0)
    m = rng.standard_normal((nrhs, n, 3))
    with SpectralEwaldSystem(x, eps, box, xi, rc, grid, P, *gcap.default_table(xi), slab_factor=1.0, max_rhs=nrhs) as s:
        out = {p: s.matvec(m, precision=p).cpu().numpy() for p in ("fp64", "df")}
    geo = ew.Geometry(x, eps, box, xi, rc, grid, P, *ew.default_table(xi), slab_factor=1.0)
    for r in sorted({0, nrhs - 1}):
        ref = geo.field_real(m[r])
        for p in out:
            assert np.abs(out[p][r] - ref).max() <= 1e-12 * np.abs(ref).max(), (p, r)
