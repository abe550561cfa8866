"""The screened 27-cell walks (point-dipole forces, field maps) against brute force where the screen could go wrong:
positions outside the box, an open z axis with large coordinates, one particle, queues that fill exactly, dense cells."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _close(got, ref, tol):
    # sums of up to a few hundred float64 terms: 1e-12 of the largest entry is > 1e3 roundings of it
    assert np.abs(got - ref).max() <= tol * max(np.abs(ref).max(), 1e-300)


@pytest.mark.parametrize("n,periodic_z,shift", [(1, True, 0), (2, True, 0), (33, False, 0), (65, True, 3), (400, False, 0),
                                                (400, True, 40), (1500, True, 0)])
def test_dipole_forces_screen(n, periodic_z, shift):
    from mutual_polarization_slab_gb300.dipole_forces import compute_forces
    from oracle.dipole_forces_oracle import compute_forces as ref
    rng = np.random.default_rng(n)
    box = np.array([12.0, 9.0, 15.0])
    # distinct lattice points with jitter: separations stay above 0.3, so no single pair dominates the sums
    g = np.stack(np.meshgrid(np.arange(12), np.arange(9), np.arange(15), indexing="ij"), -1).reshape(-1, 3)
    x = g[rng.permutation(len(g))[:n]] + rng.uniform(-0.35, 0.35, (n, 3))
    x += box * rng.integers(-shift, shift + 1, (n, 3)) * np.array([1, 1, 1 if periodic_z else 0])
    if not periodic_z:
        x[:, 2] += 1e4          # an open axis keeps its absolute coordinates
    m = rng.normal(size=(n, 3))
    F, U = compute_forces(x, m, box, 4.4, 1.7, periodic_z)
    Fr, Ur = ref(x, m, box, 4.4, 1.7, periodic_z)
    # images and offsets cost the separations up to 1e4 / 1e-16 = 1e-12 absolute, r^-5 at 0.3 amplifies by ~20
    _close(F, Fr, 1e-10)
    _close(U, Ur, 1e-10)


@pytest.mark.parametrize("n,probes,shift", [(1, 1, 0), (40, 33, 0), (300, 70, 2), (2000, 500, 0)])
def test_field_map_screen(n, probes, shift):
    from mutual_polarization_slab_gb300.fieldmap import field_map
    from oracle import fieldmap_oracle as fo
    rng = np.random.default_rng(n)
    box, xi = np.array([11.0, 13.0, 12.0]), 0.6
    x = rng.uniform(0, 1, (n, 3)) * box + box * rng.integers(-shift, shift + 1, (n, 3))
    u = (np.arange(probes)[:, None] + 0.5) * np.array([0.618, 0.414, 0.732])
    p = np.mod(u, 1.0) * box + box * rng.integers(-shift, shift + 1, (probes, 3))
    m = rng.normal(size=(n, 3))
    _close(field_map(p, x, m, box, xi), np.real(fo.field_map(p, x, m, box, xi)), 1e-9)
