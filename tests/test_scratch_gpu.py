"""The scratch arena gives way to matrices: as many fit the device after a
product that took a large workspace as before it."""
import ctypes as C

import numpy as np
import pytest

import bml_b200 as B

pytestmark = [pytest.mark.gpu, pytest.mark.unordered]


def _fill(N, M):
    """Matrices of N rows of M (12 bytes an entry) until none fits; how many."""
    held = []
    while len(held) < 400:
        h = B.lib.bml_noinit_matrix(B.TYPE["ellpack"], 2, N, M, B.SEQUENTIAL)
        if not h:
            assert B.last_error() == B.ERR_ALLOC
            B.clear_error()
            break
        held.append(h)
    for h in held:
        B.lib.bml_deallocate(C.byref(C.c_void_p(h)))
    B.lib.bml_b200_synchronize()
    return len(held)


def test_a_matrix_fits_after_the_arena_has_grown():
    N, M = 32768, 8192  # 3 GiB each
    B.lib.bml_b200_set_verbose(0)
    try:
        _fill(N, M)  # the arena of earlier calls goes
        before = _fill(N, M)
        assert before >= 1
        # X^2 of a diagonal matrix into wide rows: the workspace is sized by the rows' room, not by what they hold
        n = 2 * N  # 5 GiB of workspace
        v, ix = np.zeros((n, 32)), np.zeros((n, 32), np.int32)
        v[:, 0], ix[:, 0] = 1.0 + np.arange(n), np.arange(n)
        X = B.Ellpack.from_arrays(v, ix, np.ones(n, np.int32), n, 32)
        Y = B.Ellpack(n, 16384)
        st, _ = B.multiply_x2(X, Y, 0.0)
        assert st == B.OK
        X.free()
        Y.free()
        assert _fill(N, M) == before
    finally:
        B.lib.bml_b200_set_verbose(1)
        B.clear_error()
