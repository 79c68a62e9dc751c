"""The FP64 tensor-instruction form of the ELLBLOCK product (32 x 32 blocks,
unordered form) against the ordered block product, which other tests hold bit
for bit to the restatement: the same block lists (first-touch order) and
counts, values within 1e-12 of S = |A| |B|, traces likewise.  X symmetric and
not, A*B, blocks dropped from the middle of rows, more block columns touched
than MB holds, overflow, empty block rows."""
import ctypes as C

import numpy as np
import pytest

import bml_b200 as B
from test_ellblock_tc_gpu import block_lattice, from_dense, set_partition, to_dense

pytestmark = [pytest.mark.gpu, pytest.mark.unordered]
BS = 32


class _Lists(C.Structure):
    _fields_ = [("matrix_type", C.c_int), ("matrix_precision", C.c_int), ("distribution_mode", C.c_int),
                ("N", C.c_int), ("M", C.c_int), ("NB", C.c_int), ("MB", C.c_int), ("ptr_value", C.c_void_p),
                ("indexb", C.POINTER(C.c_int)), ("nnzb", C.POINTER(C.c_int))]


def _lists(h):
    assert B.lib.bml_get_bandwidth(h) >= 0  # brings the host mirror up to date
    s = _Lists.from_address(h)
    nz = np.ctypeslib.as_array(s.nnzb, shape=(s.NB,)).copy()
    ix = np.ctypeslib.as_array(s.indexb, shape=(s.NB * s.MB,)).copy()
    return [list(ix[i * s.MB:i * s.MB + nz[i]]) for i in range(s.NB)]


def _free(*hs):
    for h in hs:
        B.lib.bml_deallocate(C.byref(C.c_void_p(h)))


def _product(a, b, nb, MB, thr, exact):
    """(status, traces or None, dense C, block lists) of A*B, or X^2 for b None."""
    old = B.lib.bml_b200_set_x2_exact(exact)
    set_partition(nb, MB)
    N = nb * BS
    h = B.lib.bml_zero_matrix(3, 2, N, N, 0)
    B.lib.bml_b200_set_verbose(0)
    tr = (C.c_double * 2)()
    if b is None:
        st = B.lib.bml_b200_multiply_x2(a, h, thr, tr)
    else:
        B.lib.bml_multiply_AB(a, b, h, thr)
        st = B.last_error()
    B.clear_error()
    B.lib.bml_b200_set_verbose(1)
    B.lib.bml_b200_set_x2_exact(old)
    D = to_dense(h, N)
    out = (st, (tr[0], tr[1]) if b is None else None, D, _lists(h))
    _free(h)
    return out


def _compare(A, Bm, nb, MB, thr, status=B.OK):
    set_partition(nb, nb)
    a = from_dense(A)
    b = None if Bm is None else from_dense(Bm)
    got, want = (_product(a, b, nb, MB, thr, e) for e in (0, 1))
    S = np.abs(A) @ np.abs(A if Bm is None else Bm)
    _free(*([a] if b is None else [a, b]))
    assert got[0] == want[0] == status
    assert got[3] == want[3]
    assert (np.abs(got[2] - want[2]) <= 1e-12 * S + 1e-300).all()
    if Bm is None:
        for g, w in zip(got[1], want[1]):
            assert abs(g - w) <= 1e-12 * max(np.trace(S), np.abs(np.diag(A)).sum())
    return got[2]


def _random_blocks(nb, per_row, seed, symmetric, small=0.0):
    """Random block pattern; a share `small` of the blocks scaled to 1e-4."""
    rng = np.random.default_rng(seed)
    D = np.zeros((nb * BS, nb * BS))
    for i in range(nb):
        for j in set(rng.integers(0, nb, per_row)) | {i}:
            x = rng.standard_normal((BS, BS)) * (1e-4 if rng.random() < small else 1.0)
            D[i * BS:(i + 1) * BS, j * BS:(j + 1) * BS] = x
    return (D + D.T) / 2 if symmetric else D


@pytest.mark.parametrize("L,radius", [(1, 1.0), (2, 1.0), (3, 1.0), (3, 2.0), (4, 1.5)])
def test_x2_symmetric_lattice(L, radius):
    H = block_lattice(L, radius, seed=L)
    D = _compare(H, None, L ** 3, L ** 3, 1e-5)
    assert np.array_equal(D, D.T)


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("nb,per_row,thr", [(5, 2, 0.0), (17, 3, 1e-5), (40, 3, 20.0), (40, 4, 1e-3), (64, 40, 1e-5),
                                            # queued without the lists' lengths up to 128 block rows
                                            (128, 3, 1e-5), (129, 3, 1e-5)])
def test_x2_random_blocks(nb, per_row, thr, symmetric):
    X = _random_blocks(nb, per_row, nb, symmetric, small=0.4)
    _compare(X, None, nb, nb, thr)


def test_x2_symmetric_pattern_with_one_unequal_entry():
    X = _random_blocks(20, 3, 7, True)
    i, j = np.argwhere(X != 0)[100]
    X[i, j] += 1e-9
    _compare(X, None, 20, 20, 1e-5)


@pytest.mark.parametrize("nb,per_row", [(9, 2), (33, 4)])
def test_ab(nb, per_row):
    A, Bm = _random_blocks(nb, per_row, 1, False, 0.3), _random_blocks(nb, per_row, 2, False, 0.3)
    A[BS:2 * BS] = 0.0  # an empty block row of A, and of B
    Bm[2 * BS:3 * BS] = 0.0
    _compare(A, Bm, nb, nb, 1e-3)


def test_more_block_columns_touched_than_mb_holds():
    """Blocks past MB before thresholding that the threshold drops again, and
    rows that stay too wide."""
    nb = 40
    X = _random_blocks(nb, 3, 11, True, small=0.7)
    set_partition(nb, nb)
    x = from_dense(X)
    touched = max(len(r) for r in _product(x, None, nb, nb, -1.0, 1)[3])
    kept = max(len(r) for r in _product(x, None, nb, nb, 1.0, 1)[3])
    _free(x)
    assert kept < touched
    _compare(X, None, nb, kept, 1.0)
    _compare(X, None, nb, kept - 2, 1.0, status=B.ERR_ROW_OVERFLOW)
