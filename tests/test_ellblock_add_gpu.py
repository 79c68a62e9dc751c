"""ELLBLOCK add, copy and scale against their definitions, bit for bit, for
blocks of at most 32 x 32 (a warp per block of the sum) and larger ones (a CTA
per block): A's blocks in order, then B's new ones, alpha*a + beta*b rounded
step by step, kept when max |x| > threshold; rows of more blocks than a CTA
has threads, empty rows, rows too wide for MB."""
import ctypes as C

import numpy as np
import pytest

import bml_b200 as B
from test_ellblock_f64_gpu import _free, _lists

pytestmark = pytest.mark.gpu


def _partition(bs, mb):
    B.lib.bml_b200_reset_block_sizes()
    B.lib.bml_set_block_sizes((C.c_int * len(bs))(*bs), len(bs), mb)


def _import(D, bs, mb, dtype):
    _partition(bs, mb)
    a = np.ascontiguousarray(D, dtype)
    h = B.lib.bml_import_from_dense(3, 2 if dtype == np.float64 else 1, 0, D.shape[0], D.shape[0],
                                    a.ctypes.data_as(C.c_void_p), 0.0, 0)
    B.check()
    return h


def _dense(h, n, dtype):
    p = B.lib.bml_export_to_dense(h, 0)
    t = C.c_double if dtype == np.float64 else C.c_float
    d = np.ctypeslib.as_array(C.cast(p, C.POINTER(t)), shape=(n * n,)).copy().reshape(n, n)
    B.lib.bml_free_memory(C.c_void_p(p))
    return d


def _blocks(bs, share, seed, dtype, scale=1.0):
    rng = np.random.default_rng(seed)
    off = np.concatenate([[0], np.cumsum(bs)])
    D = np.zeros((off[-1], off[-1]), dtype)
    for i in range(len(bs)):
        for j in range(len(bs)):
            if i != 2 and (i == j or rng.random() < share):
                D[off[i]:off[i + 1], off[j]:off[j + 1]] = rng.standard_normal((bs[i], bs[j])) * (
                    scale if rng.random() < 0.3 else 1.0)
    return D, off


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("bs,share", [([4] * 300, 0.95), ([32] * 20, 0.4), ([1, 7, 32, 5, 16, 31] * 4, 0.5),
                                      ([40, 8, 64, 33] * 2, 0.6)], ids=["wide", "32", "mixed", "large"])
@pytest.mark.parametrize("alpha,beta,thr", [(2.0, -1.0, 1e-2), (0.0, 1.5, 0.0), (1.0, 0.0, 1e-2)])
def test_add_copy_scale(bs, share, alpha, beta, thr, dtype):
    nb = len(bs)
    Da, off = _blocks(bs, share, 1, dtype, 1e-4)
    Db, _ = _blocks(bs, share, 2, dtype, 1e-4)
    n = int(off[-1])
    a, b = _import(Da, bs, nb, dtype), _import(Db, bs, nb, dtype)
    la, lb = _lists(a), _lists(b)
    c = B.lib.bml_copy_new(a)
    assert _lists(c) == la and np.array_equal(_dense(c, n, dtype), Da)
    B.lib.bml_add(c, b, alpha, beta, thr)
    B.check()
    S = np.zeros_like(Da)
    if alpha:
        S = (0.0 + alpha * Da.astype(np.float64)).astype(dtype)
    if beta:
        S = (S.astype(np.float64) + beta * Db.astype(np.float64)).astype(dtype)
    want = np.zeros_like(S)
    lists = []
    for i in range(nb):
        row = (la[i] if alpha else []) + [k for k in (lb[i] if beta else []) if not alpha or k not in la[i]]
        keep = [k for k in row if np.abs(S[off[i]:off[i + 1], off[k]:off[k + 1]]).max() > dtype(thr)]
        lists.append(keep)
        for k in keep:
            want[off[i]:off[i + 1], off[k]:off[k + 1]] = S[off[i]:off[i + 1], off[k]:off[k + 1]]
    assert _lists(c) == lists
    assert np.array_equal(_dense(c, n, dtype), want)
    s = (C.c_double if dtype == np.float64 else C.c_float)(0.3)
    B.lib.bml_scale_inplace(C.byref(s), c)
    assert np.array_equal(_dense(c, n, dtype), dtype(s.value) * want)
    _free(a, b, c)


def test_add_overflow():
    bs, nb = [8] * 30, 30
    Da, _ = _blocks(bs, 0.2, 3, np.float64)
    Db, _ = _blocks(bs, 0.9, 4, np.float64)
    b = _import(Db, bs, nb, np.float64)
    a = _import(Da, bs, nb, np.float64)
    widest = max(len(r) for r in _lists(a))
    _partition(bs, widest)
    c = B.lib.bml_zero_matrix(3, 2, 240, 240, 0)
    B.lib.bml_copy(a, c)
    B.check()
    B.lib.bml_b200_set_verbose(0)
    B.lib.bml_add(c, b, 1.0, 1.0, 0.0)
    st = B.last_error()
    B.clear_error()
    B.lib.bml_b200_set_verbose(1)
    assert st == B.ERR_ROW_OVERFLOW
    assert max(len(r) for r in _lists(c)) == widest
    _free(a, b, c)
