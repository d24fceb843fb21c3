"""Tensor-core update of FP64 fronts (operands cut into seven 9-bit digits).

The self-check runs the split + TMA + tcgen05 path of the factorization on a
synthetic panel and compares with a long double host product, relative to the
product of the two row norms in units of 2^-53.  Bound: one unit for the
rounding of the result, plus per term nine units of 2^-10 (the six dropped
products with index sum 9 of at most 2^-63 each, as much again for the
later ones and the rounding of the operands and of the sum together: 9)."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from sylver_gb300 import workloads as w

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,spread,special",
                         [(1, 1, 0, -1), (31, 5, 0, 30), (128, 32, 0, -1), (129, 33, 20, -1),
                          (200, 70, 40, 5), (300, 257, 0, 299), (1000, 96, 60, -1),
                          (2500, 160, 10, -1), (384, 2048, 3, 0)])
def test_tc64_update_selfcheck(sylver, gpu, rows, k, spread, special):
    err = ctypes.c_double(-1.0)
    rc = sylver.load().sylver_gb300_tc64_selfcheck(rows, k, spread, special, ctypes.byref(err))
    assert rc == 0
    assert 0.0 <= err.value <= 1.0 + 9.0 * k / 1024.0, err.value


@pytest.mark.parametrize("n", [97, 128, 255, 256, 257, 289, 513, 700])
def test_fp64_dense_front(sylver, gpu, n):
    """One dense front whose last panel and last group are full, ragged or one
    column: L^-1 against NumPy's through a forward solve.  Bound: Cholesky and
    the substitution are backward stable with n + 1 roundings per entry; the
    matrix has a condition number below 10."""
    rng = np.random.default_rng(n)
    g = rng.standard_normal((n, n))
    d = np.ldexp(1.0, rng.integers(-300, 300, n))  # badly scaled rows and columns
    a = (g @ g.T / n + np.eye(n)) * d[:, None] * d[None, :]
    m = w.SymMatrix.from_scipy(sp.csc_matrix(a))
    an = sylver.Analysis(m.n, m.ptr, m.row)
    f = sylver.Factor(an, True, m.val)
    assert f.flag == 0
    b = rng.standard_normal((n, 3)) * d[:, None]
    x = f.solve(b) * d[:, None]
    xt = np.linalg.solve(g @ g.T / n + np.eye(n), b / d[:, None])
    assert np.abs(x - xt).max() <= 10 * (n + 1) * 2.0 ** -53 * 10 * np.abs(xt).max()
