"""Touched columns of the unordered product (A*B's width before thresholding;
a negative threshold keeps every touched column), which it tells from the sums
themselves: products that are zero of either sign, sums that cancel to zero,
products that underflow.  Against the ordered form, which counts columns when
they are first touched: the same status, widths, columns and values."""
import numpy as np
import pytest

import bml_b200 as B

pytestmark = [pytest.mark.gpu, pytest.mark.unordered]


def _matrix(N, M, seed, dtype, special):
    rng = np.random.default_rng(seed)
    v, ix, nz = np.zeros((N, M), dtype), np.zeros((N, M), np.int32), rng.integers(0, M + 1, N).astype(np.int32)
    for i in range(N):
        ix[i, :nz[i]] = np.sort(rng.choice(N, nz[i], replace=False))
        v[i, :nz[i]] = rng.choice(special, nz[i])
    return v, ix, nz


def _rows(m, N, M):
    v, ix, nz = m.download()
    v, ix = v.reshape(N, M), ix.reshape(N, M)
    return [sorted(zip(ix[i, :nz[i]].tolist(), v[i, :nz[i]].tolist())) for i in range(N)], nz


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("thr,square,Mc", [(-1.0, True, 200), (-1.0, False, 200), (0.5, False, 200), (0.5, False, 12),
                                           (float("nan"), True, 200)])
def test_touched_columns(thr, square, Mc, dtype):
    N, M = 200, 9
    tiny = np.finfo(dtype).tiny
    special = np.array([1.0, -1.0, 0.0, -0.0, 2.0, -tiny, tiny], dtype)
    a, b = _matrix(N, M, 1, dtype, special), _matrix(N, M, 2, dtype, special)
    prec = "double_real" if dtype == np.float64 else "single_real"
    out = []
    B.lib.bml_b200_set_verbose(0)
    for exact in (0, 1):
        old = B.lib.bml_b200_set_x2_exact(exact)
        A, Bm, Cm = B.Ellpack.from_arrays(*a, N, M, prec), B.Ellpack.from_arrays(*b, N, M, prec), B.Ellpack(N, Mc, prec)
        if square:
            st, _ = B.multiply_x2(A, Cm, thr)
        else:
            B.lib.bml_multiply_AB(A.h, Bm.h, Cm.h, thr)
            st = B.last_error()
        B.clear_error()
        out.append((st, *_rows(Cm, N, Mc)))
        B.lib.bml_b200_set_x2_exact(old)
    B.lib.bml_b200_set_verbose(1)
    (st0, r0, n0), (st1, r1, n1) = out
    assert st0 == st1 == (B.ERR_ROW_OVERFLOW if Mc == 12 else B.OK)
    assert np.array_equal(n0, n1)
    if Mc == 200:
        for x, y in zip(r0, r1):
            assert [k for k, _ in x] == [k for k, _ in y]
            # sums of small integers are exact in any order; the smallest normal numbers beside them come and go
            assert all(abs(p - q) <= 1e-30 for (_, p), (_, q) in zip(x, y))
