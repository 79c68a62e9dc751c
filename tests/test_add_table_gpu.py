"""bml_add through the direct column table against its definition, bit for bit:
A's entries in A's order as alpha*a (+ beta*b), then B's new columns in B's
order as beta*b, each step rounded as the reference rounds it
(ellpack/bml_add_ellpack_typed.c:50-216), kept when |x| > threshold.  Rows at
the edges of the tables (2048 columns of B where M is at most 512, else 32768),
wider ones beside them (found by a hash), rows longer than one round of a CTA
(128 and 1024 entries), columns that are multiples of a table apart, empty
rows, zero scalars; and tr(A B^T) of matrices large enough to be sized by their
rows."""
import numpy as np
import pytest

import bml_b200 as B

pytestmark = pytest.mark.gpu


def _random(N, M, ncols, widths, span, seed, dtype):
    rng = np.random.default_rng(seed)
    v, ix, nz = np.zeros((N, M), dtype), np.zeros((N, M), np.int32), np.zeros(N, np.int32)
    for i in range(N):
        n, s = widths[i % len(widths)], min(span[i % len(span)], ncols)
        lo = int(rng.integers(0, ncols - s + 1))
        c = rng.choice(s, size=min(n, s), replace=False) + lo
        if len(c) >= 2:  # the whole span, ends included
            c[0], c[1] = lo, lo + s - 1
            c = np.unique(c)
            rng.shuffle(c)
        v[i, :len(c)], ix[i, :len(c)], nz[i] = rng.standard_normal(len(c)), c, len(c)
    return v, ix, nz


def _sum(a, b, alpha, beta, thr, dtype):
    out = []
    for av, ai, an, bv, bi, bn in zip(*a, *b):
        x = {}
        if alpha:
            for k, y in zip(ai[:an], av[:an]):
                x[int(k)] = dtype(0.0 + alpha * float(y))
        if beta:
            for k, y in zip(bi[:bn], bv[:bn]):
                x[int(k)] = dtype(float(x.get(int(k), 0.0)) + beta * float(y))
        out.append([(k, y) for k, y in x.items() if abs(y) > dtype(thr)])
    return out


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("alpha,beta,thr", [(2.0, -1.0, 1e-1), (1.0, 1.0, 0.0), (0.0, 0.7, 0.3), (1.3, 0.0, 0.3)])
@pytest.mark.parametrize("ncols,M,wide_a,wide_b,span", [
    (40, 40, (0, 1, 7, 40), (40, 0, 3), (40,)),
    (70000, 600, (300, 0, 31), (0, 290, 17, 1), (32768, 32769, 500, 70000)),
    (70000, 512, (250, 0, 31, 257), (0, 240, 17, 255), (2048, 2049, 500, 70000)),
    (9000, 4096, (2048, 2049, 2500, 0), (1500, 0, 1590, 2100, 1), (9000, 2600)),
])
def test_add_rows(ncols, M, wide_a, wide_b, span, alpha, beta, thr, dtype):
    N = 48
    prec = "double_real" if dtype == np.float64 else "single_real"
    a = _random(N, M, ncols, wide_a, span, 1, dtype)
    b = _random(N, M, ncols, wide_b, span, 2, dtype)
    for i in range(N):  # no row of the sum is wider than M
        b[2][i] = min(b[2][i], M - a[2][i]) if ncols > M else b[2][i]
    if dtype == np.float32:
        b[0][:, ::3] = -b[0][:, ::3]
    if ncols > 2 ** 16:  # columns that are multiples of the table apart
        a[1][1, :8] = b[1][1, :8] = np.arange(8) * 8192
        a[2][1], b[2][1] = 8, 8
    # half of B's columns where A has them too
    for i in range(0, N, 2):
        n = min(a[2][i], b[2][i]) // 2
        free = [k for k in b[1][i, n:b[2][i]] if k not in set(a[1][i, :n])]
        b[1][i, :n] = a[1][i, :n]
        b[1][i, n:n + len(free)] = free
        b[2][i] = n + len(free)
    A = B.Ellpack.from_arrays(*a, N, M, prec)
    Bm = B.Ellpack.from_arrays(*b, N, M, prec)
    B.lib.bml_add(A.h, Bm.h, alpha, beta, thr)
    B.check()
    v, ix, nz = A.download()
    v, ix = v.reshape(N, M), ix.reshape(N, M)
    want = _sum(a, b, alpha, beta, thr, dtype)
    for i in range(N):
        assert int(nz[i]) == len(want[i])
        assert [int(k) for k in ix[i, :nz[i]]] == [k for k, _ in want[i]]
        assert np.array_equal(v[i, :nz[i]], np.array([x for _, x in want[i]], dtype))


def test_add_overflow_keeps_the_first_entries():
    N, M = 33, 64
    a = _random(N, M, 500, (60,), (500,), 3, np.float64)
    b = _random(N, M, 500, (50,), (500,), 4, np.float64)
    A, Bm = (B.Ellpack.from_arrays(*x, N, M) for x in (a, b))
    B.lib.bml_b200_set_verbose(0)
    B.lib.bml_add(A.h, Bm.h, 1.0, 1.0, 0.0)
    assert B.last_error() == B.ERR_ROW_OVERFLOW
    B.clear_error()
    B.lib.bml_b200_set_verbose(1)
    v, ix, nz = A.download()
    want = _sum(a, b, 1.0, 1.0, 0.0, np.float64)
    for i in range(N):
        n = min(len(want[i]), M)
        assert nz[i] == n
        assert [int(k) for k in ix[i * M:i * M + n]] == [k for k, _ in want[i][:n]]


@pytest.mark.parametrize("wa,wb", [(300, 20), (20, 300), (0, 5)])
def test_trace_mult_sized_by_rows(wa, wb):
    N, M, ncols = 5000, 512, 5000
    a = _random(N, M, ncols, (wa, wa // 2), (600,), 5, np.float64)
    b = _random(N, M, ncols, (wb,), (600,), 6, np.float64)
    A, Bm = (B.Ellpack.from_arrays(*x, N, M) for x in (a, b))
    want = size = 0.0
    for i in range(N):
        y = dict(zip(b[1][i, :b[2][i]].tolist(), b[0][i, :b[2][i]].tolist()))
        p = [x * y[k] for k, x in zip(a[1][i, :a[2][i]].tolist(), a[0][i, :a[2][i]].tolist()) if k in y]
        want += sum(p)
        size += sum(map(abs, p))
    assert abs(B.lib.bml_trace_mult(A.h, Bm.h) - want) <= 1e-12 * max(size, 1e-300)


def test_add_to_a_column_stored_twice():
    """Two entries of A in one column (bml_set_element appends to rows of at
    most two entries): B's entry joins the sum once."""
    import ctypes as C
    N, M = 40, 8
    A, Bm = B.Ellpack(N, M), B.Ellpack(N, M)
    x = C.c_double()
    for i in range(N):
        for y in (1.0, 2.0):
            x.value = y
            B.lib.bml_set_element(A.h, i, (i + 3) % N, C.byref(x))
        x.value = 10.0
        B.lib.bml_set_element(Bm.h, i, (i + 3) % N, C.byref(x))
    B.lib.bml_add(A.h, Bm.h, 1.0, 0.5, 0.0)
    B.check()
    v, ix, nz = A.download()
    for i in range(N):
        at = slice(i * M, i * M + nz[i])
        assert list(ix[at]) == [(i + 3) % N] * 2
        assert v[at].sum() == 8.0


@pytest.mark.parametrize("wa,wb", [(20, 300), (300, 20), (2, 300), (40, 40)])
@pytest.mark.parametrize("twice", ["a", "b"])
def test_trace_mult_of_columns_stored_twice(wa, wb, twice):
    """Every entry of A counts once, against the last of B's in its column."""
    N, M, ncols = 5000, 512, 5000
    a = _random(N, M, ncols, (wa,), (600,), 7, np.float64)
    b = _random(N, M, ncols, (wb,), (600,), 8, np.float64)
    for x in (a, b):
        for i in range(0, N, 2):  # columns that both store
            n = min(a[2][i], b[2][i]) // 2
            if x is b:
                free = [k for k in b[1][i, n:b[2][i]] if k not in set(a[1][i, :n])]
                b[1][i, :n], b[1][i, n:n + len(free)] = a[1][i, :n], free
                b[2][i] = n + len(free)
    d = a if twice == "a" else b
    for i in range(0, N, 3):
        if d[2][i] >= 2:
            d[1][i, d[2][i] - 1] = d[1][i, 0]
    A, Bm = (B.Ellpack.from_arrays(*x, N, M) for x in (a, b))
    want = size = 0.0
    for i in range(N):
        y = dict(zip(b[1][i, :b[2][i]].tolist(), b[0][i, :b[2][i]].tolist()))
        p = [x * y[k] for k, x in zip(a[1][i, :a[2][i]].tolist(), a[0][i, :a[2][i]].tolist()) if k in y]
        want += sum(p)
        size += sum(map(abs, p))
    assert abs(B.lib.bml_trace_mult(A.h, Bm.h) - want) <= 1e-12 * size
