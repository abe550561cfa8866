"""Float32 polydisperse matvecs of many vectors on both sides of the rules between the kernels that take a group of vectors
at a time and the others: spread and contraction each by itself, groups that are not full, grids below and above the spread's
limits, particles just below and above the contraction's.  Tolerance: 2e-5 relative (max-norm), the bar of the operator's
other tests; grids with eta below 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,P,n,nrhs", [
    ((34, 33, 37), 8, 840, 48),      # both
    ((34, 33, 37), 8, 833, 48),      # spread only: one particle too few
    ((24, 25, 26), 8, 840, 48),      # contraction only: too few tiles
    ((33, 35, 38), 7, 620, 65),      # both, last group of one vector
    ((40, 36, 32), 16, 2400, 17),    # both, largest support, second group of one vector
    ((34, 33, 37), 8, 2500, 16),     # both, one group
    ((54, 53, 53), 6, 60, 16),       # neither: large and sparse
    ((54, 53, 53), 6, 1400, 16),     # spread only, above the limit for large grids
])
def test_rules(grid, P, n, nrhs):
    from mutual_polarization_slab_gb300 import sizes as gs
    from oracle import polydisperse_oracle as po
    rng = np.random.default_rng(n + nrhs)
    xi, tol, box = 0.55, 1e-2, 0.72 * np.array(grid)
    k = [int(v / 1.7) for v in box]
    g = np.stack(np.meshgrid(*[np.arange(v) for v in k], indexing="ij"), -1).reshape(-1, 3)
    x = np.mod((g[rng.permutation(len(g))[:n]] + 0.5) / k * box + rng.uniform(-0.05, 0.05, (n, 3)) - 1.0, box)
    assert len(x) == n
    radii, eps = rng.uniform(0.5, 0.8, n), rng.uniform(3.0, 9.0, n)
    m = rng.standard_normal((nrhs, n, 3))
    ref = po.PolyGeometry(x, radii, eps, box, xi, tol, Ngrid=grid, P=P)
    with gs.PolydisperseSystem(x, radii, eps, box, xi, tol, Ngrid=grid, P=P, max_rhs=nrhs) as s:
        out = s.matvec(m, precision="fp32").cpu().numpy()
    for r in sorted({0, 15, nrhs - 1}):
        want = ref.field(m[r])
        assert np.abs(out[r] - want).max() <= 2e-5 * np.abs(want).max(), r
