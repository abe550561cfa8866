"""Float64 matvecs on both sides of the rule between the library's own transforms and cuFFT: rods behind a short x axis
(dipoles, field maps), grids with an axis below 30 nodes (quadrupoles, sizes).  Tolerances: 1e-12 (dipoles, field maps) and
1e-11 relative (max-norm), the bars of the operators' other tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _particles():
    from mutual_polarization_slab_gb300.workloads import rsa
    x, box, _ = rsa(60, 0.1, seed=5)
    return x, np.asarray(box), np.random.default_rng(1)


@pytest.mark.parametrize("grid", [(13, 16, 199), (13, 16, 200), (14, 16, 200), (13, 200, 15), (200, 13, 15)])
@pytest.mark.parametrize("nrhs", [1, 4])
def test_dipoles(grid, nrhs):
    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    from oracle import ewald_oracle as ew
    x, box, rng = _particles()
    xi, rc, P, eps, m = 0.7, 0.45 * box[0], 7, np.full(60, 12.0), rng.standard_normal((nrhs, 60, 3))
    with SpectralEwaldSystem(x, eps, box, xi, rc, grid, P, *gcap.default_table(xi), slab_factor=1.0, max_rhs=nrhs) as s:
        out = s.matvec(m, precision="fp64").cpu().numpy()
    g = ew.Geometry(x, eps, box, xi, rc, grid, P, *ew.default_table(xi), slab_factor=1.0)
    for r in range(nrhs):
        ref = g.field_real(m[r])
        assert np.abs(out[r] - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("grid", [(29, 30, 31), (30, 29, 30), (30, 31, 29), (30, 30, 31)])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_quadrupoles_and_sizes(grid, nrhs):
    from mutual_polarization_slab_gb300 import quadrupole as gq, sizes as gs
    from oracle import polydisperse_oracle as po, quadrupole_oracle as qo
    x, box, rng = _particles()
    xi, rc, P, lam = 0.6, 0.45 * box[0], 7, rng.uniform(3.0, 9.0, 60)
    S, Q = rng.standard_normal((nrhs, 60, 3)), rng.standard_normal((nrhs, 60, 5))
    ref = qo.QuadGeometry(x, lam, box, xi, rc, grid, P, *qo.default_quad_tables(xi))
    with gq.QuadrupoleSystem(x, lam, box, xi, 1e-4, rc=rc, Ngrid=grid, P=P, max_rhs=nrhs) as s:
        out = s.matvec(s.pack(S, Q), precision="fp64").cpu().numpy()
    for r in range(nrhs):
        for part, want in zip((slice(0, 3), slice(3, 8)), ref.apply(S[r], Q[r], real=True)):
            assert np.abs(out[r][:, part] - want).max() <= 1e-11 * np.abs(want).max()
    radii = rng.uniform(0.6, 1.0, 60)
    ref = po.PolyGeometry(x, radii, lam, box, xi, 1e-2, Ngrid=grid, P=P)
    with gs.PolydisperseSystem(x, radii, lam, box, xi, 1e-2, Ngrid=grid, P=P, max_rhs=nrhs) as s:
        out = s.matvec(S, precision="fp64").cpu().numpy()
    for r in range(nrhs):
        want = ref.field(S[r])
        assert np.abs(out[r] - want).max() <= 1e-11 * np.abs(want).max()
