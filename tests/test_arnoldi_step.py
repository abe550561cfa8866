"""The Arnoldi step kernels where they change form: systems of up to 2048 unknowns take one block each, larger ones the
split dots (chunks of 2048 unknowns); one pass and two passes of Gram-Schmidt, up to 41 columns (groups of four), one
and several right-hand sides, a zero right-hand side, graph and host-driven.  The solver's residual is checked with the
operator itself: at most the tolerance (the solver ends on a true residual)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 100, 682, 683, 1365, 1366])
@pytest.mark.parametrize("nrhs,restart", [(1, 1), (1, 41), (3, 6), (4, 13)])
def test_residual_of_the_solution(n, nrhs, restart, monkeypatch):
    import torch

    from mutual_polarization_slab_gb300 import capacitance as gcap
    from mutual_polarization_slab_gb300.system import SpectralEwaldSystem
    from mutual_polarization_slab_gb300.workloads import rsa
    x, box, _ = rsa(n, 0.25 if n > 10 else 0.01, seed=n)
    rc = min(5.0, 0.45 * box[0])
    xi = 3.0 / rc
    eps = np.full(n, 28.0)
    rng = np.random.default_rng(n)
    b = torch.as_tensor(rng.standard_normal((nrhs, n, 3)), device="cuda")
    if nrhs == 4:
        b[2] = 0.0
    with SpectralEwaldSystem(x, eps, box, xi, rc, np.full(3, 24), 8, *gcap.default_table(xi), slab_factor=0.0,
                             max_rhs=nrhs) as s:
        tol = 1e-9
        kw = dict(tol=tol, restart=restart, maxit=400, precision="fp64")
        sol, info = s.solve(b, **kw)
        assert all(i.converged for i in info)
        res = b - s.matvec(sol)
        for r in range(nrhs):
            assert float(res[r].norm()) <= 1.0001 * tol * float(b[r].norm())
        monkeypatch.setenv("MPS_GMRES_GRAPH", "0")
        host, hinfo = s.solve(b, **kw)
        assert torch.equal(sol, host)
        assert [i.matvecs_fp64 for i in info] == [i.matvecs_fp64 for i in hinfo]
        # one pass: the mixed solve's inner steps, with the true residual after every correction
        mixed, minfo = s.solve(b, tol=1e-8, restart=max(restart, 10), maxit=10, precision="mixed", residual_policy=1)
        assert all(i.converged for i in minfo)
        res = b - s.matvec(mixed)
        for r in range(nrhs):
            assert float(res[r].norm()) <= 1.0001e-8 * float(b[r].norm())
