"""First use of an axis length from several threads at once, each on a non-blocking stream of its own: the transforms'
tables have to be complete before any of them reads them."""
import glob
import os
import re
import threading

import numpy as np
import pytest


def test_uploads_wait_for_the_device():
    # a plain cudaMemcpy from pageable memory promises only that the data has been staged
    csrc = os.path.join(os.path.dirname(__file__), "..", "mutual_polarization_slab_gb300", "csrc")
    bad = [f for f in glob.glob(os.path.join(csrc, "*.cu")) if re.search(r"\bcudaMemcpy\(", open(f).read())]
    assert not bad


# lengths that no other test takes: 62, 74, 58 (primes 31, 37, 29) in float64, 250, 162, 128 in double-float
@pytest.mark.gpu
@pytest.mark.parametrize("precision,grid", [("fp64", (62, 74, 58)), ("df", (250, 162, 128))])
def test_first_use_on_side_streams(precision, grid):
    import torch
    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    from mutual_polarization_slab_gb300.workloads import rsa
    from oracle import ewald_oracle as ew
    x, box, _ = rsa(60, 0.1, seed=5)
    xi, rc, P = 0.7, 0.45 * box[0], 7
    eps = np.full(60, 12.0)
    tables = gcap.default_table(xi)
    m = np.random.default_rng(1).standard_normal((60, 3))
    torch.cuda.synchronize()
    barrier, out = threading.Barrier(4), [None] * 4

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            with SpectralEwaldSystem(x, eps, box, xi, rc, grid, P, *tables, slab_factor=0.0, max_rhs=1) as s:
                barrier.wait(60)
                out[k] = s.matvec(m, precision=precision).cpu().numpy()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    pn, pa, rvn = ew.default_table(xi)
    ref = ew.Geometry(x, eps, box, xi, rc, grid, P, pn, pa, rvn, slab_factor=0.0).field_real(m)
    # 1e-12 relative (max-norm): the bar of the float64-accurate operators
    for o in out:
        assert np.abs(o - ref).max() <= 1e-12 * np.abs(ref).max()
