"""An infinite diagonal entry (a penalty taken to its limit): its unknown is zero and the
others solve the system without it, on every path a front takes.  Bound: as for the
other systems of condition number below 3 with n + 1 roundings per entry, 18 n u."""
import numpy as np
import pytest
import scipy.sparse as sp

from sylver_gb300 import workloads as w

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [20, 70, 110, 150, 300])
@pytest.mark.parametrize("precision", [0, 1])
def test_infinite_pivot(sylver, gpu, n, precision):
    rng = np.random.default_rng(n)
    a = rng.uniform(-1.0, 1.0, (n, n))
    a = a + a.T
    np.fill_diagonal(a, 2.0 * np.abs(a).sum(axis=1).max())
    k = n // 2
    b = rng.standard_normal((n, 2))
    keep = np.delete(np.arange(n), k)
    xt = np.zeros((n, 2))
    xt[keep] = np.linalg.solve(a[np.ix_(keep, keep)], b[keep])
    a[k, k] = np.inf
    m = w.SymMatrix.from_scipy(sp.csc_matrix(a))
    an = sylver.Analysis(m.n, m.ptr, m.row, order=np.arange(1, n + 1))
    f = sylver.Factor(an, True, m.val, precision=precision)
    assert f.flag == 0
    x = f.solve(f.solve(b, job=1), job=3)
    u = 2.0 ** -24 if precision else 2.0 ** -53
    assert np.abs(x - xt).max() <= 18 * n * u * np.abs(xt).max()
