"""X^2 and A*B on the dense tier at its smallest sizes (N from 1024, tiles of
128), symmetric (one triangle formed) and not, against the dense FP64 product:
values within 1e-12 of S = |A| |B| (FP32: 2 n 2^-24), the kept pattern, the
diagonal kept where a product touches it (a stored row of zeros included, and a
row of zeros whose column nothing stores), traces, rows in any order."""
import numpy as np
import pytest

import bml_b200 as B
import x2check

pytestmark = [pytest.mark.gpu, pytest.mark.unordered]


def _ell(P, D, shuffle):
    """ELLPACK arrays of the entries of pattern P with D's values."""
    N = D.shape[0]
    M = int(P.sum(1).max())
    rng = np.random.default_rng(0)
    v, ix, nz = np.zeros((N, M), D.dtype), np.zeros((N, M), np.int32), P.sum(1).astype(np.int32)
    for i in range(N):
        c = np.flatnonzero(P[i])
        if shuffle:
            rng.shuffle(c)
        v[i, :len(c)], ix[i, :len(c)] = D[i, c], c
    return (v.reshape(-1), ix.reshape(-1), nz), M


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("N", [1024, 1025, 1200])
@pytest.mark.parametrize("kind", ["symmetric", "one_entry_off", "ab"])
def test_dense_tier(N, kind, dtype):
    rng = np.random.default_rng(N)

    def matrix():
        P = rng.random((N, N)) < 0.6
        D = rng.standard_normal((N, N)) / np.sqrt(N)
        if kind != "ab":
            P, D = P | P.T, (D + D.T) / 2
            if kind == "one_entry_off":
                i, j = np.argwhere(P)[1234]
                D[i, j] += 0.5
        D[7], D[:, 7] = 0.0, 0.0  # stored zeros: touched through them
        P[7, 9] = P[9, 7] = True
        P[11, :], P[:, 11] = False, False  # an empty row and column
        if kind != "symmetric":
            D[13] = 0.0  # zeros, and nothing stored in that column but the diagonal's absence
            P[:, 13] = False
        return P, np.where(P, D, 0.0).astype(dtype)

    Pa, Da = matrix()
    Pb, Db = matrix() if kind == "ab" else (Pa, Da)
    want = Da.astype(np.float64) @ Db.astype(np.float64)
    S = abs(Da.astype(np.float64)) @ abs(Db.astype(np.float64))
    touched = (Pa.astype(np.float32) @ Pb.astype(np.float32)).diagonal() > 0
    thr = 0.02
    a, ma = _ell(Pa, Da, True)
    prec = "double_real" if dtype == np.float64 else "single_real"
    A = B.Ellpack.from_arrays(*a, N, ma, prec)
    Cm = B.Ellpack(N, N, prec)
    if kind == "ab":
        b, mb = _ell(Pb, Db, False)
        Bm = B.Ellpack.from_arrays(*b, N, mb, prec)
        B.lib.bml_multiply_AB(A.h, Bm.h, Cm.h, thr)
        B.check()
    else:
        st, tr = B.multiply_x2(A, Cm, thr)
        assert st == B.OK
        assert abs(tr[1] - np.trace(want)) <= (1e-12 if dtype == np.float64 else 1e-5) * np.trace(S)
    assert B.lib.bml_b200_last_x2_dense() == 1
    got = Cm.download()
    assert x2check.rows_sorted(got, N)
    v, ix, nz = got[0].reshape(N, N), got[1].reshape(N, N), got[2]
    G, K = np.zeros((N, N)), np.zeros((N, N), bool)
    for i in range(N):
        G[i, ix[i, :nz[i]]], K[i, ix[i, :nz[i]]] = v[i, :nz[i]], True
    tol = (1e-12 if dtype == np.float64 else 2.0 * N * 2.0 ** -24) * S
    keep = abs(want) > thr
    np.fill_diagonal(keep, touched)
    sure = (abs(abs(want) - thr) > tol) | np.eye(N, dtype=bool)
    assert np.array_equal(K[sure], keep[sure])
    assert (abs(G - want)[K] <= tol[K] + 1e-300).all()
    if kind == "symmetric":
        assert np.array_equal(G, G.T)


def test_entries_of_a_row_that_cancel():
    """A row whose two entries lie in one column and cancel, nothing stored in
    its own column: no product touches its diagonal."""
    N = 1024
    D = np.random.default_rng(1).standard_normal((N, N))
    D = D + D.T
    D[50] = D[:, 50] = 0.0
    (v, ix, nz), M = _ell(D != 0, D, False)
    v[50 * M:50 * M + 2], ix[50 * M:50 * M + 2], nz[50] = (1.0, -1.0), 49, 2
    Y = B.Ellpack(N, N)
    st, tr = B.multiply_x2(B.Ellpack.from_arrays(v, ix, nz, N, M), Y, 1e-9)
    assert st == B.OK and B.lib.bml_b200_last_x2_dense() == 1
    assert Y.download()[2][50] == 0
    assert abs(tr[1] - np.trace(D @ D)) <= 1e-12 * np.trace(abs(D) @ abs(D))
