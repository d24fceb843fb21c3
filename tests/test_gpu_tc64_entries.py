"""FP64 tensor-core update, entry by entry: an FP64 sum of k products and its
subtraction from C commit at most u ((k + 1) (|L| |L^T|)_ij + |C_ij|), u = 2^-53.  An entry d
taken from the digit products adds the rounding of the sum (u |d|) and what the digits
leave out, below (k + 1) 2^-68 of the two scales 2^e; it is only taken where
|d| >= 2^-15 or |C| >= k 2^-12 of the scales, so that this is below u (k + 1) |d| or u |C| / 8:
at most u ((k + 3) (|L| |L^T|)_ij + 9/8 |C_ij|) in all, the unit of the check."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("narrow", [0, 1])
@pytest.mark.parametrize("rows,k,spread,rowexp,special",
                         [(1, 1, 0, 0, -1), (33, 31, 0, 0, -1), (64, 32, 30, 200, 40),
                          (129, 33, 60, 0, -1), (160, 64, 0, 300, -1), (97, 65, 100, 0, 0),
                          (200, 130, 12, 500, -1), (300, 96, 20, 3, 299), (130, 700, 40, 0, -1),
                          (257, 257, 800, 100, -1), (256, 512, 0, 0, -1), (150, 1100, 0, 2, -1)])
def test_tc64_update_entries(sylver, gpu, rows, k, spread, rowexp, special, narrow):
    err, changed = ctypes.c_double(-1.0), ctypes.c_long(-1)
    rc = sylver.load().sylver_gb300_tc64_entrycheck(rows, k, spread, rowexp, narrow, special,
                                                    ctypes.byref(err), ctypes.byref(changed))
    assert rc == 0
    assert changed.value == 0
    assert 0.0 <= err.value <= 1.0, err.value
