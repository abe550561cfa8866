"""Vectors of one batched matvec stay apart: a vector of small moments keeps its own relative accuracy beside a large one,
a zero vector gives zeros, and a vector of NaN leaves the others alone.  Grids whose (y, z) planes hold an odd number of
rows, where the transforms' pairs of rows could reach from one vector's grid into the next.  Tolerances: 1e-12 (dipoles)
and 1e-11 (quadrupoles, sizes) relative to each vector's own largest entry, the bars of the operators' other tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(kind, grid, nrhs):
    from mutual_polarization_slab_gb300 import capacitance as gcap, quadrupole as gq, sizes as gs
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    from mutual_polarization_slab_gb300.workloads import rsa
    x, box, _ = rsa(60, 0.1, seed=5)
    xi, rc, eps = 0.7, 0.45 * box[0], np.full(60, 12.0)
    if kind == "quadrupole":
        return gq.QuadrupoleSystem(x, eps, box, xi, 1e-4, rc=rc, Ngrid=grid, P=7, max_rhs=nrhs)
    if kind == "sizes":
        return gs.PolydisperseSystem(x, np.linspace(0.6, 1.0, 60), eps, box, xi, 1e-4, rc=rc, Ngrid=grid, P=7,
                                     max_rhs=nrhs)
    return SpectralEwaldSystem(x, eps, box, xi, rc, grid, 7, *gcap.default_table(xi), slab_factor=1.0, max_rhs=nrhs)


@pytest.mark.parametrize("kind,precision,grid", [
    ("dipole", "fp64", (25, 25, 25)), ("dipole", "fp64", (24, 27, 31)), ("dipole", "fp64", (24, 24, 25)),
    ("dipole", "df", (24, 25, 27)), ("dipole", "df", (24, 24, 25)), ("quadrupole", "fp64", (30, 31, 27)),
    ("sizes", "fp64", (33, 31, 27)), ("sizes", "fp64", (31, 31, 31))])
def test_vectors_apart(kind, precision, grid):
    scale = np.array([1.0, 1e-12, 0.0, 1e6, 1.0, np.nan, 1e-3])
    ndof, tol = (8, 1e-11) if kind == "quadrupole" else (3, 1e-11 if kind == "sizes" else 1e-12)
    m = np.random.default_rng(3).standard_normal((7, 60, ndof))
    with _system(kind, grid, 7) as s:
        single = np.stack([s.matvec(v, precision=precision).cpu().numpy() for v in m])
        out = s.matvec(m * scale[:, None, None], precision=precision).cpu().numpy()
    for r, k in enumerate(scale):
        if np.isnan(k):
            assert np.isnan(out[r]).all()
        else:
            assert np.abs(out[r] - k * single[r]).max() <= tol * k * np.abs(single[r]).max(), r
