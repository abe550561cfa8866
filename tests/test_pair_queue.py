"""The float64 pair list where a row's queue fills exactly, by one less and by one more (rows of 0 to 97 pairs), and the
polydisperse couplings of such rows.  Tolerance: 1e-11 relative (max-norm), the float64 polydisperse operator's bar."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 32, 33, 34, 64, 65, 66, 98])
def test_cluster_rows(n):
    from mutual_polarization_slab_gb300 import sizes as gs
    from oracle import polydisperse_oracle as po
    rng = np.random.default_rng(n)
    box, xi, tol = np.array([26.0, 28.0, 30.0]), 0.4, 1e-4          # cutoff 7.6: every sphere of the cluster sees all others
    g = np.stack(np.meshgrid(*[np.arange(-3, 4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    g = g[np.argsort((g ** 2).sum(1), kind="stable")][:n]
    x = np.concatenate((1.3 * g + rng.uniform(-0.04, 0.04, (n, 3)), [[13.0, 14.0, 15.0]]))
    x = np.mod(x[rng.permutation(n + 1)], box)                      # the cluster sits across the box's corner
    radii, eps = rng.uniform(0.4, 0.6, n + 1), rng.uniform(3.0, 9.0, n + 1)
    p = rng.standard_normal((n + 1, 3))
    ref = po.PolyGeometry(x, radii, eps, box, xi, tol)
    with gs.PolydisperseSystem(x, radii, eps, box, xi, tol, max_rhs=1) as s:
        assert s.n_pairs == ref.p1.size
        out = s.matvec(p[None]).cpu().numpy()[0]
    E = ref.field(p)
    assert np.abs(out - E).max() <= 1e-11 * np.abs(E).max()
