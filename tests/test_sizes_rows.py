"""Couplings of the polydisperse pair list, found a pair to a thread: rows without pairs first, last and in between, no pair
at all, a single one, and pairs beyond one block, against the oracle (float64 1e-11, as for the operator elsewhere)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX = np.array([56.0, 52.0, 54.0])
FAR = np.array([[50.0, 45.0, 47.0], [38.0, 45.0, 35.0], [50.0, 30.0, 40.0], [38.0, 30.0, 47.0]])   # apart from all others


def _cluster(k):
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)
    return 3.0 + 2.3 * g + 0.2 * np.random.default_rng(k).uniform(-1, 1, g.shape)


CASES = {
    "one sphere": FAR[:1],
    "no pairs": FAR,
    "one pair": np.vstack((FAR[:1], FAR[:1] + [2.3, 0.0, 0.0])),
    "empty rows around a pair": np.vstack((FAR[1:2], _cluster(2)[:1], FAR[2:3], _cluster(2)[1:2], FAR[3:4])),
    "empty rows around many": np.vstack((FAR[:2], _cluster(4)[:20], FAR[2:3], _cluster(4)[20:], FAR[3:4])),
}


@pytest.mark.parametrize("tables", [False, True])
@pytest.mark.parametrize("case", list(CASES))
def test_rows(case, tables):
    from mutual_polarization_slab_gb300 import sizes as gs
    from oracle import polydisperse_oracle as po
    x, xi, tol = CASES[case], 0.5, 1e-5
    n = len(x)
    eps = np.linspace(3.0, 9.0, n)
    if tables:
        a = np.where(np.arange(n) % 2 == 0, 0.8, 1.0)
        rt = po.default_r_table()
        uniq, _ = po.unique_radii(a)
        perp, para = po.real_space_table(rt, uniq, xi)
        og = po.PolyGeometry(x, a, eps, BOX, xi, tol, tables=(rt, perp, para, uniq))
        sysm = gs.PolydisperseSystem(x, a, eps, BOX, xi, tol, rt, perp, para, max_rhs=1)
    else:
        a = np.linspace(0.7, 1.0, n)
        og = po.PolyGeometry(x, a, eps, BOX, xi, tol)
        sysm = gs.PolydisperseSystem(x, a, eps, BOX, xi, tol, max_rhs=1)
    p = np.random.default_rng(n).normal(size=(n, 3))
    with sysm:
        assert sysm.n_pairs == og.p1.size
        got = sysm.matvec(p).cpu().numpy()
    want = og.field(p)
    assert np.abs(got - want).max() <= 1e-11 * np.abs(want).max()
