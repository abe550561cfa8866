"""The staged gradient contraction's long regions (one vector, three home blocks to a CTA): bit-identical to the warp gather
on grids staged by 16-byte pieces and by single nodes, with home blocks left over in y."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,P", [((104, 100, 108), 10), ((101, 104, 99), 10), ((96, 112, 104), 8), ((106, 97, 103), 8)])
def test_long_regions(monkeypatch, grid, P):
    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    rng = np.random.default_rng(P)
    n, box = 3000, 0.8 * np.array(grid)
    x, m = rng.uniform(0, 1, (n, 3)) * box, rng.standard_normal((1, n, 3))
    with SpectralEwaldSystem(x, np.full(n, 5.0), box, 0.6, 0.4, grid, P, *gcap.default_table(0.6), slab_factor=0.0,
                             max_rhs=1) as s:
        home = s.matvec(m, precision="fp32grad").cpu().numpy()
        monkeypatch.setenv("MPS_GRAD_CONTRACT", "warp")
        warp = s.matvec(m, precision="fp32grad").cpu().numpy()
    np.testing.assert_array_equal(home, warp)
