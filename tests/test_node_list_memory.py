"""Device memory that a first matvec keeps.  Float64 dipoles: grids, spectra and one list entry per particle and tile, no
second list of the entries (only the tiled contractions read one).  Float32 sizes, few vectors: grids and spectra, no room
for the interleaved grids of many vectors."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pool_used():
    import torch
    rt = ctypes.CDLL("libcudart.so.13")
    pool, used = ctypes.c_void_p(), ctypes.c_uint64()
    torch.cuda.synchronize()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), torch.cuda.current_device()) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(used)) == 0   # cudaMemPoolAttrUsedMemCurrent
    return used.value


def test_first_matvec_memory():
    import torch
    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    g, n, P = 61, 100_000, 10   # no axis is a multiple of the tile's 8 nodes: up to 4 x 4 x 4 tiles a particle
    k = 47
    x = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 2.2 + 0.5
    box = np.full(3, 2.2 * k)
    m = torch.ones((n, 3), dtype=torch.float64, device="cuda")
    with SpectralEwaldSystem(x, np.full(n, 5.0), box, 0.3, 2.3, (g, g, g), P, *gcap.default_table(0.3), slab_factor=0.0,
                             max_rhs=1) as s:
        out, before = torch.empty_like(m), _pool_used()
        s.matvec(m, precision="fp64", out=out)
        kept = _pool_used() - before
        pairs = s.n_pairs
    entries = 64 * n * 4
    grids = 3 * g ** 3 * 8 + 3 * (g // 2 + 1) * g * g * 16
    # beside the lists and grids: the float64 copy of the pair list (six doubles a pair) and a quarter of the lists
    assert kept <= grids + entries + 48 * pairs + entries // 4, (kept, grids, entries, pairs)


@pytest.mark.parametrize("nrhs", [1, 15, 16])
def test_first_sizes_matvec_memory(nrhs):
    import torch
    from mutual_polarization_slab_gb300 import sizes as gs
    g, n = 96, 64
    x = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3) * 5.0 + 1.0
    box = np.full(3, 20.0)
    with gs.PolydisperseSystem(x, np.full(n, 1.0), np.full(n, 5.0), box, 0.5, 1e-2, rc=5.5, Ngrid=(g, g, g), P=6,
                               max_rhs=nrhs) as s:
        m = torch.ones((nrhs, n, 3), dtype=torch.float64, device="cuda")
        out, before = torch.empty_like(m), _pool_used()
        s.matvec(m, precision="fp32", out=out)
        kept = _pool_used() - before
    grids = nrhs * (g ** 3 * 4 + (g // 2 + 1) * g * g * 8)
    # beside them: the transforms' work area (as large again at most), a few lists of the 64 particles
    assert kept <= 2 * grids + (1 << 20), (kept, grids)
