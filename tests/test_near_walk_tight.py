"""The division-free pair terms of the screened walks to rounding: particles inside a periodic box, so that neither images
nor offsets cost digits.  Tolerance 1e-12 of the largest entry: a sum of up to a few hundred terms, each a few roundings
(1.1e-16) of its own size, the terms of a particle up to ten times their sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _close(got, ref):
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("n", [2, 65, 700, 1500])
def test_dipole_forces(n):
    from mutual_polarization_slab_gb300.dipole_forces import compute_forces
    from oracle.dipole_forces_oracle import compute_forces as ref
    rng = np.random.default_rng(n)
    box = np.array([12.0, 9.0, 15.0])
    g = np.stack(np.meshgrid(np.arange(12), np.arange(9), np.arange(15), indexing="ij"), -1).reshape(-1, 3)
    x = g[rng.permutation(len(g))[:n]] + rng.uniform(0.2, 0.8, (n, 3))   # separations above 0.4
    m = rng.normal(size=(n, 3))
    F, U = compute_forces(x, m, box, 4.4, 1.7, True)
    Fr, Ur = ref(x, m, box, 4.4, 1.7, True)
    _close(F, Fr)
    _close(U, Ur)


@pytest.mark.parametrize("n,probes", [(40, 33), (1500, 400)])
def test_field_map(n, probes):
    from mutual_polarization_slab_gb300.fieldmap import field_map
    from oracle import fieldmap_oracle as fo
    rng = np.random.default_rng(n)
    box, xi = np.array([22.0, 26.0, 24.0]), 0.6
    k = (11, 13, 12)
    g = np.stack(np.meshgrid(*[np.arange(v) for v in k], indexing="ij"), -1).reshape(-1, 3)
    x = (g[rng.permutation(len(g))[:n]] + 0.5) * 2.0 + rng.uniform(-0.2, 0.2, (n, 3))
    p = rng.uniform(0.0, 1.0, (probes, 3)) * box
    m = rng.normal(size=(n, 3))
    _close(field_map(p, x, m, box, xi), np.real(fo.field_map(p, x, m, box, xi)))
