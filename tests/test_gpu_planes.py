"""Digit planes of FP64 Cholesky updates: their size is bounded, so that wide levels go
through them in several launches, and a device without room for them takes the
updates on the FP64 pipe.

Bound of the solutions: diagonally dominant matrices of condition number at most 3;
Cholesky, the sweeps and the inverses of their diagonal blocks commit at most 18 n u
relative to the largest entry, n the longest chain of eliminations."""
import numpy as np
import pytest
import scipy.sparse as sp

from sylver_gb300 import workloads as w

pytestmark = pytest.mark.gpu


def _leaves(nleaf, n1, nb, seed):
    """nleaf dense leaves of n1 columns that do not touch, under one dense root of nb."""
    n = nleaf * n1 + nb
    rng = np.random.default_rng(seed)
    i, j = np.tril_indices(n1, -1)
    rows, cols = [], []
    for q in range(nleaf):
        rows += [q * n1 + i, np.repeat(np.arange(n - nb, n), n1)]
        cols += [q * n1 + j, np.tile(np.arange(q * n1, (q + 1) * n1), nb)]
    i, j = np.tril_indices(nb, -1)
    rows.append(n - nb + i)
    cols.append(n - nb + j)
    r, c = np.concatenate(rows), np.concatenate(cols)
    v = rng.uniform(-1.0, 1.0, r.size)
    s = max(np.bincount(r, np.abs(v), n).max(), np.bincount(c, np.abs(v), n).max())
    low = sp.coo_matrix((v * (0.25 / s), (r, c)), shape=(n, n)).tocsc()
    return (low + low.T + sp.eye(n)).tocsc()


def _check(sylver, a, chain, launches):
    m = w.SymMatrix.from_scipy(a)
    an = sylver.Analysis(m.n, m.ptr, m.row, order=np.arange(1, m.n + 1))
    assert an.flag >= 0
    f = sylver.Factor(an, True, m.val)
    assert f.flag == 0
    xt = np.random.default_rng(1).uniform(-1.0, 1.0, (m.n, 2))
    x = f.solve(np.asfortranarray(a @ xt))
    assert np.abs(x - xt).max() <= 18 * chain * 2.0 ** -53 * np.abs(xt).max()
    pr = f.profile()
    for kind, count in launches.items():
        assert pr[kind]["launches"] == count, (kind, pr[kind])


def test_planes_in_several_launches(sylver, gpu):
    # 20 fronts of 1200 rows, planes of 2^22 entries (an eighth of the front storage is
    # less): 17 + 3 fronts' trailing columns behind column 256, 14 + 6 contribution
    # blocks of 300 columns; the root's trailing columns behind 256, 512 and 768
    _check(sylver, _leaves(20, 300, 900, 3), 1200, {"panel_split": 7})


def test_panels_in_several_launches(sylver, gpu):
    # 2000 fronts of 100 rows, of which 68 each are cut behind the first panel: two
    # launches of the first panel step and of its update, one of the second panel step,
    # and two of the contribution blocks (1092 + 908 fronts of 60 rows, 64 columns)
    _check(sylver, _leaves(2000, 40, 60, 4), 100,
           {"panel_trsm": 3, "update_tc": 4, "panel_split": 2})


@pytest.mark.parametrize("posdef,precision", [(True, 0), (True, 1), (False, 0)])
def test_allocation_failures(sylver, gpu, posdef, precision):
    """Every allocation of a first factorization in turn reports out of memory: the call
    fails with the CUDA error flag or gives a correct factor another way, and the next
    call is none the worse for it."""
    lib = sylver.load()
    p = w.lognormal27(9) if posdef else w.shifted_laplace3d(7, nrhs=1)
    an = sylver.Analysis(p.a.n, p.a.ptr, p.a.row, order=p.order)
    full = p.a.to_scipy_full()
    kinds, n = [], 0
    while True:
        n += 1
        assert n < 1000
        lib.sylver_gb300_fail_allocation(n)
        try:
            f = sylver.Factor(an, posdef, p.a.val, precision=precision, ir_max_iter=5)
        finally:
            left = lib.sylver_gb300_fail_allocation(0)
        if f.flag < 0:
            assert f.flag == -51 and left == 0
            continue
        x = f.solve(p.rhs)
        assert w.backward_error(full, x, p.rhs).max() <= 1e-14
        if posdef:
            kinds.append(f.profile()["update_tc"]["launches"] > 0)
        if left:
            break
    assert n > 20
    if posdef and precision == 0:
        # the planes' own allocation: FP64 pipe; nothing failed: digit products
        assert kinds == [False, True]
