"""The polydisperse operator for one to many vectors (separate and interleaved float32 grids) against the oracle where the
kernels could go wrong: numbers of vectors around the groups of 4 and 16, grids that are no multiple of the 32-node
transposition tile, stencils that wrap, small and large supports.  Tolerances: 1e-11 (float64) and 2e-5 (float32)
relative (max-norm), the bars of the operator's other tests; grids with eta below 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,P,n", [((13, 12, 11), 11, 1), ((34, 33, 37), 8, 90), ((31, 39, 33), 5, 70),
                                      ((40, 36, 32), 16, 33), ((32, 30, 40), 6, 500), ((16, 50, 48), 10, 1)])
@pytest.mark.parametrize("nrhs", [1, 3, 11, 12, 13, 16, 17, 48, 65])
def test_vectors(grid, P, n, nrhs):
    from mutual_polarization_slab_gb300 import sizes as gs
    from oracle import polydisperse_oracle as po
    rng = np.random.default_rng(n + nrhs)
    xi, tol, box = 0.55, 1e-2, 0.72 * np.array(grid)
    g = np.stack(np.meshgrid(*[np.arange(int(v / 2.1)) for v in box], indexing="ij"), -1).reshape(-1, 3)
    x = np.mod(g[rng.permutation(len(g))[:n]] * 2.1 + rng.uniform(-0.05, 0.05, (n, 3)) - 1.0, box)
    radii, eps = rng.uniform(0.6, 1.0, n), rng.uniform(3.0, 9.0, n)
    m = rng.standard_normal((nrhs, n, 3))
    ref = po.PolyGeometry(x, radii, eps, box, xi, tol, Ngrid=grid, P=P)
    with gs.PolydisperseSystem(x, radii, eps, box, xi, tol, Ngrid=grid, P=P, max_rhs=nrhs) as s:
        out = {p: s.matvec(m, precision=p).cpu().numpy() for p in ("fp64", "fp32")}
    for r in sorted({0, nrhs // 2, nrhs - 1}):
        want = ref.field(m[r])
        for p, bar in (("fp64", 1e-11), ("fp32", 2e-5)):
            assert np.abs(out[p][r] - want).max() <= bar * np.abs(want).max(), (p, r)
