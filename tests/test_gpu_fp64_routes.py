"""Routes of FP64 Cholesky that the default schedule does not take, and the numbers of
right-hand sides at which the sweeps change their columns per pass, at the sizes where
panels, groups, tiles and blocks end.  Bound as for the other front sizes: a condition
number of at most 3, 18 n u relative to the largest entry of the solution."""
import numpy as np
import pytest
import scipy.sparse as sp

from sylver_gb300 import workloads as w
from test_gpu_front_sizes import _two_leaves

pytestmark = pytest.mark.gpu


def _system(sylver, n1, n2, nb):
    a, d = _two_leaves(n1, n2, nb, n1 + n2 + nb)
    m = w.SymMatrix.from_scipy(sp.csc_matrix(a))
    an = sylver.Analysis(m.n, m.ptr, m.row, order=np.arange(1, m.n + 1))
    assert an.flag >= 0
    return a, d, m, an


def _solves(f, a, d, counts, u):
    n = d.size
    rng = np.random.default_rng(n + 2)
    for nrhs in counts:
        b = np.asfortranarray(rng.standard_normal((n, nrhs)) * d[:, None])
        xt = np.linalg.solve(a / d[:, None] / d[None, :], b / d[:, None])
        x = f.solve(f.solve(b, job=1), job=3) * d[:, None]
        assert np.abs(x - xt).max() <= 18 * n * u * np.abs(xt).max(), nrhs


@pytest.mark.parametrize("n1,n2,nb", [(32, 40, 41), (48, 64, 16), (65, 96, 32), (80, 81, 48),
                                      (127, 200, 65), (255, 257, 140), (256, 320, 63)])
def test_fp64_pipe_route(sylver, gpu, n1, n2, nb):
    """tc_min_cb_rows < 0: panels without digits, updates by FP64 multiply-adds."""
    a, d, m, an = _system(sylver, n1, n2, nb)
    sylver.set_schedule(tc_min_cb_rows=-1, small_front_rows=64)
    try:
        f = sylver.Factor(an, True, m.val)
        assert f.flag == 0
        bad = a.copy()
        bad[-1, -1] = -bad[-1, -1]
        g = sylver.Factor(an, True, w.SymMatrix.from_scipy(sp.csc_matrix(bad)).val)
        assert g.flag == -6
    finally:
        sylver.set_schedule()
    pr = f.profile()
    assert pr["update_tc"]["launches"] == 0 and pr["panel_split"]["launches"] == 0
    if n2 + nb > 64:
        assert pr["panel_trsm"]["launches"] > 0 and pr["update"]["launches"] > 0
    _solves(f, a, d, (1, 3), 2.0 ** -53)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n1,n2,nb", [(33, 48, 47), (95, 128, 129), (255, 257, 140)])
def test_rhs_counts(sylver, gpu, n1, n2, nb, precision):
    """FP64 passes of 1, 2, 4, 6 and 8 columns, whole and ragged, FP32 ones of 4 and 16,
    and calls of more than one pass of 32."""
    a, d, m, an = _system(sylver, n1, n2, nb)
    f = sylver.Factor(an, True, m.val, precision=precision)
    assert f.flag == 0
    _solves(f, a, d, (4, 6, 7, 8, 10, 11, 12, 15, 16, 18, 24, 31, 32, 33, 40),
            2.0 ** -24 if precision else 2.0 ** -53)


@pytest.mark.parametrize("nrhs", [1, 2, 3, 5, 8, 9, 17])
def test_fp64_refinement(sylver, gpu, nrhs):
    """Refinement of an FP64 factorization: the residual by the call's columns."""
    p = w.lognormal27(9, nrhs=nrhs)
    an = sylver.Analysis(p.a.n, p.a.ptr, p.a.row, order=p.order)
    f = sylver.Factor(an, True, p.a.val, ir_max_iter=3, ir_tol=1e-15)
    x = f.solve(p.rhs)
    be = w.backward_error(p.a.to_scipy_full(), x, p.rhs).max()
    assert f.solve_inform.flag == 0 and be <= 1e-15
    assert abs(f.solve_stats()[1] - be) <= 2e-16
