"""The double-float (and hand-written float32) transforms against the float64 operator where their tiles could go wrong:
every radix as first and later stage, axes of one stage, odd and even numbers of rows, the longest axes (one column of
three lines to a block), grids with a single partial tile of columns, Nyquist planes of every parity.  Tolerances: 1e-12
and 2e-5 relative (max-norm), the two operators' bars; grids with eta below 1."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(8, 8, 8), (6, 9, 10), (18, 20, 24), (16, 27, 32), (36, 25, 50), (64, 8, 96), (100, 9, 15),
                                  (10, 1000, 8), (8, 9, 1024), (1024, 6, 9), (30, 45, 40), (72, 48, 54)])
@pytest.mark.parametrize("nrhs", [1, 2])
def test_transforms(grid, nrhs):
    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    rng = np.random.default_rng(sum(grid) + nrhs)
    box, xi, P, n = 0.8 * np.array(grid), 0.6, 6, 40
    x = rng.uniform(0, 1, (n, 3)) * box      # positions only have to be distinct: the cutoff leaves few pairs
    m = rng.standard_normal((nrhs, n, 3))
    with SpectralEwaldSystem(x, np.full(n, 5.0), box, xi, 0.3, grid, P, *gcap.default_table(xi), slab_factor=0.0,
                             max_rhs=nrhs) as s:
        ref = s.matvec(m, precision="fp64").cpu().numpy()
        df = s.matvec(m, precision="df").cpu().numpy()
        os.environ["MPS_FFT32"] = "own"
        try:
            f32 = s.matvec(m, precision="fp32").cpu().numpy()
        finally:
            del os.environ["MPS_FFT32"]
    assert np.abs(df - ref).max() <= 1e-12 * np.abs(ref).max()
    assert np.abs(f32 - ref).max() <= 2e-5 * np.abs(ref).max()
