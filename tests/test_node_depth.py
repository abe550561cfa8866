"""MPS_TILE_DEPTH fixes the depth of the float64 and double-float spread's tiles; the sums do not depend on it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "df"])
def test_depth_is_fixed(precision, monkeypatch):
    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    from mutual_polarization_slab_gb300.workloads import rsa
    x, box, _ = rsa(200, 0.1, seed=5)
    m = np.random.default_rng(1).standard_normal((4, 200, 3))
    out = {}
    for depth in ("4", "8", "12", None):   # 12: a depth of other tiles only
        if depth:
            monkeypatch.setenv("MPS_TILE_DEPTH", depth)
        else:
            monkeypatch.delenv("MPS_TILE_DEPTH")
        with SpectralEwaldSystem(x, np.full(200, 9.0), box, 0.7, 6.0, (36, 40, 45), 8, *gcap.default_table(0.7),
                                 slab_factor=0.0, max_rhs=4) as s:
            out[depth] = s.matvec(m, precision=precision).cpu().numpy()
            tile = s.tuning()["fp64"]["tile"]
        assert tile[2] == int(depth) if depth in ("4", "8") else tile[2] in (4, 8), (depth, tile)
    for v in out.values():
        assert np.array_equal(v, out["4"])
