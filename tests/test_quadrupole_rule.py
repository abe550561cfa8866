"""Float32 quadrupole matvecs on both sides of the spread's rule: particles whose stencils cover just less and just more than
half of the grid, grids just below and above the smallest one that is spread by nodes.  Tolerance: 2e-5 relative (max-norm),
the bar of the operator's other tests; grids with eta below 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,P,n", [((32, 33, 30), 6, 73), ((32, 33, 30), 6, 74), ((31, 31, 31), 8, 500),
                                      ((32, 31, 31), 8, 500), ((30, 32, 47), 5, 181)])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_spread_rule(grid, P, n, nrhs):
    from mutual_polarization_slab_gb300 import quadrupole as gq
    from oracle import quadrupole_oracle as qo
    rng = np.random.default_rng(n + P)
    xi, rc, box = 0.6, 4.0, 0.69 * np.array(grid)
    g = np.stack(np.meshgrid(*[np.arange(int(v / 2.02)) for v in box], indexing="ij"), -1).reshape(-1, 3)
    x = np.mod(g[rng.permutation(len(g))[:n]] * 2.02 + rng.uniform(-0.008, 0.008, (n, 3)) - 1.0, box)
    lam = rng.uniform(3.0, 9.0, n)
    S, Q = rng.standard_normal((nrhs, n, 3)), rng.standard_normal((nrhs, n, 5))
    tabs, rv = qo.default_quad_tables(xi)
    ref = qo.QuadGeometry(x, lam, box, xi, rc, grid, P, tabs, rv)
    with gq.QuadrupoleSystem(x, lam, box, xi, 1e-4, rc=rc, Ngrid=grid, P=P, max_rhs=nrhs) as s:
        out = s.matvec(s.pack(S, Q), precision="fp32").cpu().numpy()
    for r in range(nrhs):
        for part, want in zip((slice(0, 3), slice(3, 8)), ref.apply(S[r], Q[r], real=True)):
            assert np.abs(out[r][:, part] - want).max() <= 2e-5 * np.abs(want).max(), part
