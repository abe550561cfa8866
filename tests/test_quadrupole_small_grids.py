"""Float32 quadrupole matvecs of many particles on small grids, spread by nodes (and contracted by home blocks where particles
are many enough), and both sides of the rule's lines: cover, and for one vector particles to a node.  Tolerance: 2e-5 relative (max-norm), the bar of the operator's
other tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,P,n", [((16, 16, 16), 4, 64), ((16, 17, 19), 8, 287), ((16, 17, 19), 8, 288),
                                      ((24, 8, 9), 6, 60), ((7, 24, 24), 5, 60), ((32, 33, 30), 6, 50),
                                      ((32, 33, 30), 6, 51), ((16, 16, 16), 4, 409), ((16, 16, 16), 4, 410),
                                      ((8, 8, 8), 4, 256), ((8, 8, 8), 4, 257)])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_small_grids(grid, P, n, nrhs):
    from mutual_polarization_slab_gb300 import quadrupole as gq
    from oracle import quadrupole_oracle as qo
    rng = np.random.default_rng(n + P)
    # a spacing for which the spheres of a lattice of 2.05 fit the box and the Gaussians the grid
    h = max(0.7, 2.05 * np.ceil((n / np.prod(grid)) ** (1 / 3) * min(grid)) / min(grid))
    box = h * np.array(grid)
    g = np.stack(np.meshgrid(*[np.arange(int(v / 2.05)) for v in box], indexing="ij"), -1).reshape(-1, 3)
    assert len(g) >= n
    x = np.mod(g[rng.permutation(len(g))[:n]] * 2.05 + rng.uniform(-0.02, 0.02, (n, 3)) - 1.0, box)
    xi, rc, lam = 0.4 / h, 0.45 * min(box), rng.uniform(3.0, 9.0, n)
    S, Q = rng.standard_normal((nrhs, n, 3)), rng.standard_normal((nrhs, n, 5))
    tabs, rv = qo.default_quad_tables(xi)
    ref = qo.QuadGeometry(x, lam, box, xi, rc, grid, P, tabs, rv)
    with gq.QuadrupoleSystem(x, lam, box, xi, 1e-4, rc=rc, Ngrid=grid, P=P, max_rhs=nrhs) as s:
        out = s.matvec(s.pack(S, Q), precision="fp32").cpu().numpy()
    for r in range(nrhs):
        for part, want in zip((slice(0, 3), slice(3, 8)), ref.apply(S[r], Q[r], real=True)):
            assert np.abs(out[r][:, part] - want).max() <= 2e-5 * np.abs(want).max(), part
