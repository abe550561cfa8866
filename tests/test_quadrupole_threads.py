"""Float32 dipole + quadrupole operators of different supports used by several threads at once: the home-block contraction
asks for shared memory by support, and one thread's request must not undo another's."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_supports_side_by_side():
    import torch
    from mutual_polarization_slab_gb300 import quadrupole as gq
    grid, box, n = (16, 16, 16), 0.69 * np.array([16.0] * 3), 128
    rng = np.random.default_rng(0)
    g = np.stack(np.meshgrid(*[np.arange(6)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x = (g[rng.permutation(216)[:n]] + 0.5) * box / 6
    m = rng.standard_normal((n, 8))
    tables = gq.default_table(0.6)
    errors, results = [], {}

    def work(k, P):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                with gq.QuadrupoleSystem(x, np.full(n, 5.0), box, 0.6, 1e-4, *tables, rc=1.0, Ngrid=grid, P=P,
                                         max_rhs=1) as s:
                    md = torch.as_tensor(m, device="cuda")
                    first, last = s.matvec(md, precision="fp32"), torch.empty_like(md)
                    for _ in range(1000):
                        s.matvec(md, precision="fp32", out=last)
                    results[k] = (first.cpu().numpy(), last.cpu().numpy())
        except Exception as e:   # reported in the main thread
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k, P)) for k, P in enumerate((16, 9, 12, 16))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors
    for first, last in results.values():
        # float32 sums; the spread may add in another order
        assert np.abs(first - last).max() <= 2e-5 * np.abs(first).max()
    assert np.abs(results[0][0] - results[3][0]).max() <= 2e-5 * np.abs(results[0][0]).max()
