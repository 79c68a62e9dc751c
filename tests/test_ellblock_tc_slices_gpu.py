"""The tensor-core ELLBLOCK X^2 with a group's waves shared among CTAs (few
groups): against the ordered FP64 product, blocks that the threshold drops from
the middle of rows included.  The same kept blocks, ascending; values within
2e-5 (FP16 split) and 1e-8 (8-bit split) of the largest entry of X^2, the
bounds that test_ellblock_tc_gpu.py uses and, for the 8-bit split, 32 P 2^-31
of the row and column scales with P the 4 products or fewer of a block here."""
import ctypes as C

import numpy as np
import pytest

import bml_b200 as B
from test_ellblock_f64_gpu import BS, _free, _lists, _product, _random_blocks
from test_ellblock_tc_gpu import from_dense, set_partition, to_dense

pytestmark = [pytest.mark.gpu, pytest.mark.unordered]


@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("nb,per_row", [(1, 1), (4, 2), (5, 3), (30, 3), (61, 4), (130, 3)])
@pytest.mark.parametrize("drop", [False, True])
def test_slices(nb, per_row, drop, split):
    X = _random_blocks(nb, per_row, nb + per_row, True, small=0.5 if drop else 0.0)
    thr = 1.0 if drop else 1e-6
    set_partition(nb, nb)
    x = from_dense(X)
    st, tr, want, lists = _product(x, None, nb, nb, thr, 1)
    assert st == B.OK
    old = B.lib.bml_b200_set_tc_split(split)
    for mb in (nb, max(len(r) for r in lists)):  # room for every touched block column; for the kept ones only
        set_partition(nb, mb)
        y = B.lib.bml_zero_matrix(3, 2, nb * BS, nb * BS, 0)
        t = (C.c_double * 2)()
        B.check(B.lib.bml_b200_ellblock_multiply_x2_tc(x, y, thr, t))
        got = to_dense(y, nb * BS)
        assert [sorted(r) for r in lists] == _lists(y)
        tol = 2e-5 if split == 0 else 1e-8
        assert np.abs(got - want).max() <= tol * np.abs(want).max()
        assert abs(t[0] - tr[0]) <= 1e-12 * np.abs(np.diag(X)).sum()
        assert abs(t[1] - tr[1]) <= tol * (np.abs(X) ** 2).sum()
        _free(y)
    B.lib.bml_b200_set_tc_split(old)
    _free(x)
