"""A cutoff so small that the cells outnumber 32-bit ids (1440 x 1600 x 1920) is refused on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_too_many_cells():
    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.dipole_forces import compute_forces
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    box = np.array([14.4, 16.0, 19.2])
    x = np.random.default_rng(0).uniform(0, 1, (40, 3)) * box
    with pytest.raises(ValueError):
        SpectralEwaldSystem(x, np.full(40, 5.0), box, 0.6, 0.01, (18, 20, 24), 6, *gcap.default_table(0.6))
    with pytest.raises(RuntimeError, match="bad argument"):   # (its errors are all of this class)
        compute_forces(x, np.ones((40, 3)), box, 0.01, 1.0, True)
