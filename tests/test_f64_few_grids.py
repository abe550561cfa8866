"""Float64 matvecs of quadrupoles and sizes on axes below 30 nodes, on both sides of the number of grids from which cuFFT
transforms them.  Tolerance: 1e-11 relative (max-norm), the bar of the operators' other tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nrhs", [("quadrupoles", 2), ("quadrupoles", 3), ("sizes", 19), ("sizes", 20)])
@pytest.mark.parametrize("grid", [(16, 18, 20), (22, 29, 31)])
def test_few_grids(kind, nrhs, grid):
    from mutual_polarization_slab_gb300 import quadrupole as gq, sizes as gs
    from mutual_polarization_slab_gb300.workloads import rsa
    from oracle import polydisperse_oracle as po, quadrupole_oracle as qo
    n, xi, P = 40, 0.6, 7
    x, box, _ = rsa(n, 0.1, seed=5)
    rng = np.random.default_rng(nrhs)
    rc, lam = 0.45 * box[0], rng.uniform(3.0, 9.0, n)
    S, Q = rng.standard_normal((nrhs, n, 3)), rng.standard_normal((nrhs, n, 5))
    if kind == "quadrupoles":
        ref = qo.QuadGeometry(x, lam, box, xi, rc, grid, P, *qo.default_quad_tables(xi))
        want = [np.concatenate(ref.apply(S[r], Q[r], real=True), axis=-1) for r in (0, nrhs - 1)]
        with gq.QuadrupoleSystem(x, lam, box, xi, 1e-4, rc=rc, Ngrid=grid, P=P, max_rhs=nrhs) as s:
            out = s.matvec(s.pack(S, Q), precision="fp64").cpu().numpy()
        parts = (slice(0, 3), slice(3, 8))
    else:
        radii = rng.uniform(0.6, 1.0, n)
        ref = po.PolyGeometry(x, radii, lam, box, xi, 1e-2, Ngrid=grid, P=P)
        want = [ref.field(S[r]) for r in (0, nrhs - 1)]
        with gs.PolydisperseSystem(x, radii, lam, box, xi, 1e-2, Ngrid=grid, P=P, max_rhs=nrhs) as s:
            out = s.matvec(S, precision="fp64").cpu().numpy()
        parts = (slice(0, 3),)
    for r, w in zip((0, nrhs - 1), want):
        for part in parts:
            assert np.abs(out[r][:, part] - w[:, part]).max() <= 1e-11 * np.abs(w[:, part]).max()
