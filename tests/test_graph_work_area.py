"""The transforms' work area grows with the widest matvec so far; the steps that a solve has captured hold the address of the
area of their time.  That area stays allocated, and the next solve launches the captured steps on it."""
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


def _run(monkeypatch, graph, wider):
    """Memory that a wider matvec adds between two equal solves, and the solutions."""
    import torch
    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    monkeypatch.setenv("MPS_GMRES_GRAPH", "1" if graph else "0")
    k, g = 6, 62   # a prime that the double-float transforms do not take: float64 residuals
    x = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3) * 2.5 + 0.4
    n = len(x)
    b = np.tile([0.0, 0.0, 1.0], (1, n, 1))
    m = torch.as_tensor(np.random.default_rng(5).normal(size=(3, n, 3)), device="cuda")
    kw = dict(tol=1e-7, restart=20, maxit=8, precision="mixed")
    with SpectralEwaldSystem(x, np.full(n, 5.0), np.full(3, 2.5 * k), 0.6, 5.0, (g, g, g), 8, *gcap.default_table(0.6),
                             slab_factor=0.0, max_rhs=3) as s:
        first, info = s.solve(b, None, **kw)
        assert info[0].converged and (s.graphs()[0] >= 1) == graph
        before = _pool_used()
        if wider == "vectors":
            out = s.matvec(m, precision="fp32grad")
        else:
            out = s.matvec_complex(m[0])
        added = _pool_used() - before
        second, _ = s.solve(b, None, **kw)
        assert torch.isfinite(torch.view_as_real(out) if out.is_complex() else out).all()
        return added, first.cpu().numpy(), second.cpu().numpy()


@pytest.mark.parametrize("wider", ["vectors", "complex"])
def test_captured_work_area_stays(monkeypatch, wider):
    held, a, b = _run(monkeypatch, True, wider)
    freed, c, d = _run(monkeypatch, False, wider)
    assert held > freed, (held, freed)   # by the smaller area
    np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(c, d)
    np.testing.assert_array_equal(a, c)
