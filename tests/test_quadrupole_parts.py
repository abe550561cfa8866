"""Spread of dipole and quadrupole moments by atomics: stencils of one to eleven passes over their rows, few particles (a warp
to a pass) and one.  Tolerance: 1e-11 relative (max-norm), the float64 operator's bar."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,grid", [(3, (16, 17, 18)), (6, (16, 17, 18)), (8, (18, 16, 17)), (13, (20, 19, 21)),
                                    (18, (22, 20, 21))])
@pytest.mark.parametrize("n", [1, 40])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_passes(P, grid, n, nrhs):
    from mutual_polarization_slab_gb300 import quadrupole as gq
    from mutual_polarization_slab_gb300.workloads import rsa
    from oracle import quadrupole_oracle as qo
    x, box, _ = rsa(40, 0.1, seed=3)
    x, box = x[:n], np.asarray(box)
    rng = np.random.default_rng(P + n)
    xi, rc, lam = 0.4, 0.45 * box[0], rng.uniform(3.0, 9.0, n)
    S, Q = rng.standard_normal((nrhs, n, 3)), rng.standard_normal((nrhs, n, 5))
    ref = qo.QuadGeometry(x, lam, box, xi, rc, grid, P, *qo.default_quad_tables(xi))
    with gq.QuadrupoleSystem(x, lam, box, xi, 1e-4, rc=rc, Ngrid=grid, P=P, max_rhs=nrhs) as s:
        out = s.matvec(s.pack(S, Q), precision="fp64").cpu().numpy()
    for r in range(nrhs):
        for part, want in zip((slice(0, 3), slice(3, 8)), ref.apply(S[r], Q[r], real=True)):
            assert np.abs(out[r][:, part] - want).max() <= 1e-11 * np.abs(want).max(), part
