"""Fronts at the sizes where a kernel's blocks, tiles or dispatch rules end: two
dense leaves of n1 and n2 columns under one dense root of nb, so that a leaf is a
front with n1 of n1 + nb rows eliminated, factorised whole in one CTA (at most 80
rows in FP64, 128 in FP32), by panels, or by panels with tensor-core updates, and
the sweeps take every right-hand-side count their passes are cut into.

Bound: the matrices are strictly diagonally dominant (row sums of the off-diagonal
magnitudes at most half the diagonal), so their condition number is at most 3;
Cholesky and two triangular solves commit at most 3 n roundings per entry of
relative size u, the explicit inverses of the solves as much again: 3 * 6 n u
relative to the largest entry of the solution."""
import numpy as np
import pytest
import scipy.sparse as sp

from sylver_gb300 import workloads as w

pytestmark = pytest.mark.gpu


def _two_leaves(n1, n2, nb, seed):
    n = n1 + n2 + nb
    rng = np.random.default_rng(seed)
    a = rng.uniform(-1.0, 1.0, (n, n))
    a = np.tril(a, -1)
    a[n1:n1 + n2, :n1] = 0.0  # the leaves do not touch
    a = a + a.T
    s = np.abs(a).sum(axis=1).max()
    a = a * (0.5 / max(s, 1e-300)) + np.eye(n)
    d = 2.0 ** rng.integers(-8, 9, n)
    return a * d[:, None] * d[None, :], d


@pytest.mark.parametrize("n1,n2,nb", [(1, 1, 1), (7, 8, 1), (9, 15, 23), (16, 17, 31), (31, 33, 32),
                                      (32, 40, 41), (33, 48, 47), (48, 64, 16), (63, 65, 17),
                                      (64, 64, 64), (65, 96, 32), (80, 81, 48), (95, 128, 129),
                                      (127, 200, 65), (255, 257, 140), (256, 320, 63)])
@pytest.mark.parametrize("precision", [0, 1])
def test_front_sizes(sylver, gpu, n1, n2, nb, precision):
    n = n1 + n2 + nb
    a, d = _two_leaves(n1, n2, nb, n)
    m = w.SymMatrix.from_scipy(sp.csc_matrix(a))
    an = sylver.Analysis(m.n, m.ptr, m.row, order=np.arange(1, n + 1))
    assert an.flag >= 0
    f = sylver.Factor(an, True, m.val, precision=precision, ir_max_iter=0)
    assert f.flag == 0
    rng = np.random.default_rng(n + 1)
    u = 2.0 ** -24 if precision else 2.0 ** -53
    for nrhs in (1, 2, 3, 5, 9, 17):
        b = np.asfortranarray(rng.standard_normal((n, nrhs)) * d[:, None])
        xt = np.linalg.solve(a / d[:, None] / d[None, :], b / d[:, None])
        x = f.solve(b, job=1)
        x = f.solve(x, job=3) * d[:, None]
        assert np.abs(x - xt).max() <= 18 * n * u * np.abs(xt).max(), nrhs
    # one non-positive pivot in the last leaf column and one in the root
    for k in (n1 + n2 - 1, n - 1):
        bad = a.copy()
        bad[k, k] = -bad[k, k]
        mb = w.SymMatrix.from_scipy(sp.csc_matrix(bad))
        g = sylver.Factor(an, True, mb.val, precision=precision)
        assert g.flag == -6


@pytest.mark.parametrize("nrhs", [1, 2, 4, 6, 16])
def test_residual_columns(sylver, gpu, nrhs):
    """Refinement of an FP64 factorization takes the residual kernel through each
    number of columns per pass and stops at the 1e-14 backward error."""
    p = w.lognormal27(9, nrhs=nrhs)
    an = sylver.Analysis(p.a.n, p.a.ptr, p.a.row, order=p.order)
    f = sylver.Factor(an, True, p.a.val, precision=sylver.FP32, ir_max_iter=10)
    x = f.solve(p.rhs)
    assert f.solve_inform.flag == 0
    be = w.backward_error(p.a.to_scipy_full(), x, p.rhs).max()
    assert be <= 1e-14
    assert abs(f.solve_stats()[1] - be) <= 1e-15
