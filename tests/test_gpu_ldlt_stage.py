"""Host staging of the LDL^T level tables: growing in the middle of a level, reused at
its final size, and in pageable memory where the host gives no pinned memory.  The
tables are the same, so the factors are bit for bit."""
import numpy as np
import pytest

from sylver_gb300 import workloads as w

pytestmark = pytest.mark.gpu


def test_stage_growth_and_fallback(sylver, gpu):
    # 36^3: the leaf level's entry tables alone exceed the first block of 1 MiB
    p = w.shifted_laplace3d(36, nrhs=2)
    an = sylver.Analysis(p.a.n, p.a.ptr, p.a.row, order=p.order)
    lib = sylver.load()

    def results(f):
        assert f.flag == 0
        d, piv = f.diag(p.a.n)
        return d.view(np.int64), piv, np.array([f.inform.num_neg, f.inform.num_two])

    def same(a, b):
        return all(np.array_equal(u, v) for u, v in zip(a, b))

    f = sylver.Factor(an, False, p.a.val, ir_max_iter=5)
    grown = results(f)
    assert w.backward_error(p.a.to_scipy_full(), f.solve(p.rhs), p.rhs).max() <= 1e-14
    f.refactor(p.a.val)
    assert same(results(f), grown)
    # every allocation of the factorization in turn fails until the last one: those that
    # still succeed are the staging blocks'
    paged = 0
    for nth in range(1, 400):
        lib.sylver_gb300_fail_allocation(nth)
        try:
            g = sylver.Factor(an, False, p.a.val)
        finally:
            left = lib.sylver_gb300_fail_allocation(0)
        if left:
            break
        if g.flag < 0:
            assert g.flag == -51
            continue
        paged += 1
        assert same(results(g), grown)
    assert left and paged >= 2
