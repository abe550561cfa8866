"""The dipole + quadrupole operator against the oracle where its kernels could go wrong: grids that are no multiple of the
8-node tile, of exactly one or two, both tile depths, contraction by home blocks and by gather, the smallest and
largest support, rows of no, few and many pairs, several vectors.  Tolerances: 1e-11 (float64) and 2e-5 (float32)
relative (max-norm), the bars of the operator's other tests; grids with eta below 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,P,n,rc,nrhs", [
    ((8, 9, 10), 5, 9, 1.0, 1),            # one pair-free tile
    ((16, 16, 16), 16, 40, 5.0, 2),
    ((40, 41, 30), 8, 1280, 2.6, 1),       # gather, short rows
    ((39, 40, 47), 6, 2500, 6.5, 1),       # home blocks, long rows
    ((40, 40, 40), 16, 2100, 4.0, 2),      # home blocks, largest region
    ((47, 48, 48), 9, 3600, 4.0, 1),       # home blocks, region rows of 16
    ((48, 47, 46), 10, 3500, 4.0, 3),      # home blocks, region rows of 17, three vectors
    ((48, 57, 64), 4, 100, 8.0, 3),        # sparse: gather
    ((39, 40, 46), 7, 2399, 4.0, 1),       # one below the home blocks' rule
])
def test_operator(grid, P, n, rc, nrhs):
    from mutual_polarization_slab_gb300 import quadrupole as gq
    from oracle import quadrupole_oracle as qo
    rng = np.random.default_rng(n + P)
    xi, box = 0.6, 0.69 * np.array(grid)
    g = np.stack(np.meshgrid(*[np.arange(int(v / 2.02)) for v in box], indexing="ij"), -1).reshape(-1, 3)
    x = np.mod(g[rng.permutation(len(g))[:n]] * 2.02 + rng.uniform(-0.008, 0.008, (n, 3)) - 1.0, box)
    lam = rng.uniform(3.0, 9.0, n)
    S, Q = rng.standard_normal((nrhs, n, 3)), rng.standard_normal((nrhs, n, 5))
    tabs, rv = qo.default_quad_tables(xi)
    ref = qo.QuadGeometry(x, lam, box, xi, rc, grid, P, tabs, rv)
    with gq.QuadrupoleSystem(x, lam, box, xi, 1e-4, rc=rc, Ngrid=grid, P=P, max_rhs=nrhs) as s:
        m = s.pack(S, Q)
        out = {p: s.matvec(m, precision=p).cpu().numpy() for p in ("fp64", "fp32")}
    for r in range(nrhs):
        for part, want in zip((slice(0, 3), slice(3, 8)), ref.apply(S[r], Q[r], real=True)):
            for p, tol in (("fp64", 1e-11), ("fp32", 2e-5)):
                assert np.abs(out[p][r, :, part] - want).max() <= tol * np.abs(want).max(), (p, part)
