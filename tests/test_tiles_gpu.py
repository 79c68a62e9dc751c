"""The tile form of the unordered symmetric X^2 (8 x 8 tiles, groups of 32
rows) against the C restatement, at the sizes where its tiles, groups and
bitmap words end: within 1e-12 of S = sum |x_ij x_jk| (FP32: 2 n 2^-24, n
products per entry), patterns equal except at the threshold, rows ascending,
the result exactly symmetric, the traces of the same bound."""
import numpy as np
import pytest
import torch

import bml_b200 as B
import x2check

pytestmark = [pytest.mark.gpu, pytest.mark.unordered]
SINGLE, DOUBLE = 1, 2


@pytest.fixture
def tiles():
    """The tile form wherever it applies, whatever the counts say."""
    old = B.lib.bml_b200_set_tiles(2)
    yield
    B.lib.bml_b200_set_tiles(old)


def _banded(N, band, density, seed, empty=(), dtype=np.float64):
    """Symmetric matrix of a band, each pair present with the given
    probability, rows and columns in `empty` without entries."""
    rng = np.random.default_rng(seed)
    D = np.zeros((N, N), dtype)
    for d in range(0, min(band, N - 1) + 1):
        x = rng.standard_normal(N - d).astype(dtype) * (rng.random(N - d) < (density if d else 1.0))
        i = np.arange(N - d)
        D[i, i + d] = x
        D[i + d, i] = x
    D[list(empty), :] = 0
    D[:, list(empty)] = 0
    return D


def _rows(D, M, shuffle, seed):
    N = D.shape[0]
    rng = np.random.default_rng(seed)
    v, ix, nz = np.zeros((N, M), D.dtype), np.zeros((N, M), np.int32), np.zeros(N, np.int32)
    for i in range(N):
        c = np.flatnonzero(D[i])
        if shuffle:
            rng.shuffle(c)
        v[i, :len(c)], ix[i, :len(c)], nz[i] = D[i, c], c, len(c)
    return v.reshape(-1), ix.reshape(-1), nz


def _x2(arrs, N, M, M2, thr, prec):
    X = B.Ellpack.from_arrays(*arrs, N, M, prec)
    Y = B.Ellpack(N, M2, prec)
    st, tr = B.multiply_x2(X, Y, thr)
    return st, tr, Y.download()


def _dense(arrs, N, M):
    v, ix, nz = arrs
    D = np.zeros((N, N))
    for i in range(N):
        D[i, ix[i * M:i * M + nz[i]]] = v[i * M:i * M + nz[i]]
    return D


def _check(O, D, shuffle, thr, prec, M2=None):
    N = D.shape[0]
    M = max(1, int((D != 0).sum(1).max()))
    M2 = M2 or N
    arrs = _rows(D, M, shuffle, 3)
    ref, tr_ref, _ = O.rest_x2(*arrs, N, M, thr, M2, prec)
    av = np.abs(arrs[0].astype(np.float64))
    S, _, _ = O.rest_x2(av, arrs[1], arrs[2], N, M, -1.0, M2, DOUBLE)
    st, tr, got = _x2(arrs, N, M, M2, thr, prec)
    assert st == B.OK
    n = int(arrs[2].max())
    eps = 1e-12 if prec == DOUBLE else 2.0 * n * 2.0 ** -24
    x2check.compare(got, ref, S, M2, M2, M2, thr, eps)
    assert x2check.rows_sorted(got, M2)
    G = _dense(got, N, M2)
    assert np.array_equal(G, G.T)
    Sd = np.trace(_dense(S, N, M2))
    assert abs(tr[0] - tr_ref[0]) <= eps * max(1.0, np.abs(np.diag(D)).sum())
    assert abs(tr[1] - tr_ref[1]) <= max(eps, 1e-5 if prec == SINGLE else 0.0) * max(Sd, 1e-300)


# N at the ends of tiles (8), groups (32) and words of the bitmaps (256 rows);
# bands inside one tile, across groups, and the whole matrix
CASES = [(1, 0, 1.0, ()), (7, 3, 0.6, ()), (8, 8, 0.9, ()), (9, 2, 1.0, ()), (31, 5, 0.7, (3, 4)),
         (32, 31, 0.5, ()), (33, 33, 0.4, (0, 32)), (65, 9, 0.5, tuple(range(24, 64))), (256, 40, 0.8, ()),
         (257, 40, 0.5, (256,)), (300, 299, 0.3, ()), (513, 300, 0.9, ()), (1000, 20, 1.0, ())]


@pytest.mark.parametrize("prec", [DOUBLE, SINGLE], ids=["fp64", "fp32"])
@pytest.mark.parametrize("shuffle", [False, True], ids=["ascending", "any_order"])
@pytest.mark.parametrize("N,band,density,empty", CASES)
def test_tiles_against_restatement(tiles, N, band, density, empty, shuffle, prec):
    from oracle import oracle as O
    D = _banded(N, band, density, N + band, empty, np.float64 if prec == DOUBLE else np.float32)
    for thr in (0.0, 1e-2):
        _check(O, D, shuffle, thr, prec)
        assert B.product_form() == "tiles_symmetric"
    assert B.lib.bml_b200_last_x2_symmetric() == 1


@pytest.mark.parametrize("N", [8 * 127, 8 * 128, 8 * 129, 8400])
def test_tiles_long_lists(N):
    """As many common tile columns as a warp lists at a time (128), one more
    and less, and many more."""
    M = N
    rng = np.random.default_rng(0)
    D = np.zeros((N, N))
    D[:8, :] = rng.standard_normal((8, N))
    D = D + D.T
    D[np.arange(N), np.arange(N)] = 1.0
    arrs = _rows(D, M, False, 0)
    st, tr, got = _x2(arrs, N, M, N, 1e-9, DOUBLE)
    assert st == B.OK
    assert B.product_form() == "tiles_symmetric"
    Dt = torch.from_numpy(D).cuda()  # the FP64 dense product as the oracle
    want, S = Dt @ Dt, Dt.abs() @ Dt.abs()
    G = torch.from_numpy(_dense(got, N, N)).cuda()
    tol = 1e-12 * S + torch.where(G == 0, 1e-9, 0.0)  # an entry at the threshold may be dropped
    assert bool(((G - want).abs() <= tol).all())
    assert abs(tr[1] - float(want.trace())) <= 1e-12 * float(S.trace())


def test_matrices_the_tile_form_leaves_to_the_sparse_one():
    """Infinite entries, a stored row of zeros and an asymmetric entry give
    the full form's result."""
    N = 200
    D = _banded(N, 20, 0.8, 1)
    M = int((D != 0).sum(1).max())
    base = _rows(D, M, False, 0)
    v, ix, nz = base
    inf = v.copy()
    inf[5 * M + int(np.flatnonzero(ix[5 * M:5 * M + nz[5]] == 5)[0])] = np.inf
    zero = v.copy()
    row = np.repeat(np.arange(N), M)
    zero[(row == 7) | (ix == 7)] = 0.0
    asym = v.copy()
    asym[9 * M] += 1.0
    for vals in (inf, zero, asym):
        st, tr, got = _x2((vals, ix, nz), N, M, N, 1e-5, DOUBLE)
        assert B.product_form() == ("sparse" if vals is asym else "sparse_symmetric")
        old = B.lib.bml_b200_set_x2_symmetric(0)
        st0, tr0, want = _x2((vals, ix, nz), N, M, N, 1e-5, DOUBLE)
        B.lib.bml_b200_set_x2_symmetric(old)
        assert st == st0 == B.OK
        assert np.array_equal(got[2], want[2])
        assert np.array_equal(got[1], want[1])
        np.testing.assert_allclose(got[0], want[0], rtol=1e-9, atol=1e-12)


def test_entries_of_a_row_that_cancel():
    """A row whose two entries lie in one column and cancel, nothing stored in
    its own column: no product touches its diagonal."""
    N, M = 200, 20
    D = _banded(N, 5, 1.0, 3, (50,))
    v, ix, nz = _rows(D, M, False, 0)
    v[50 * M:50 * M + 2], ix[50 * M:50 * M + 2], nz[50] = (1.0, -1.0), 49, 2
    st, tr, got = _x2((v, ix, nz), N, M, N, 1e-9, DOUBLE)
    assert st == B.OK
    assert got[2][50] == 0
    assert B.product_form() == "sparse"
    assert tr[1] == pytest.approx(np.trace(D @ D), rel=1e-12)


@pytest.mark.parametrize("i,j", [(180, 3), (3, 180), (20, 3), (97, 64), (199, 0)])
def test_an_entry_without_its_mirror(i, j):
    """An entry outside the band with no mirror, in a tile that has none
    either, on each side of the diagonal and within a group of 32 rows: X^2 is
    not formed as X X^T."""
    N = 200
    D = _banded(N, 2, 1.0, 3)
    D[i, j] = 0.5
    M = N
    st, tr, got = _x2(_rows(D, M, False, 0), N, M, N, 0.0, DOUBLE)
    assert st == B.OK
    S = np.abs(D) @ np.abs(D)
    assert (np.abs(_dense(got, N, N) - D @ D) <= 1e-12 * S).all()
    assert tr[1] == pytest.approx(np.trace(D @ D), rel=1e-12)
    assert B.lib.bml_b200_last_x2_symmetric() == 0
    assert B.product_form() == "sparse"


@pytest.mark.parametrize("M2", [40, 76], ids=["pool_runs_out", "rows_too_wide"])
def test_tiles_row_overflow(M2):
    """A result row wider than M (81 here) is reported, rows hold at most M
    entries of the product and the traces are whole.  With M2 = 40 the pool of
    packed blocks runs out and the sparse form completes the call."""
    N = 300
    D = _banded(N, 20, 1.0, 2)
    M = int((D != 0).sum(1).max())
    arrs = _rows(D, M, False, 0)
    B.lib.bml_b200_set_verbose(0)
    try:
        st, tr, got = _x2(arrs, N, M, M2, 0.0, DOUBLE)
    finally:
        B.lib.bml_b200_set_verbose(1)
        B.clear_error()
    assert st == B.ERR_ROW_OVERFLOW
    X2 = D @ D
    assert tr[1] == pytest.approx(np.trace(X2), rel=1e-12)
    for i in range(N):
        n = int(got[2][i])
        assert 0 < n <= M2
        k = got[1][i * M2:i * M2 + n]
        np.testing.assert_allclose(got[0][i * M2:i * M2 + n], X2[i, k], rtol=0, atol=1e-11)
    if M2 == 76:
        assert B.lib.bml_b200_last_required_M() == 81
    assert B.product_form() == ("tiles_symmetric" if M2 == 76 else "sparse_symmetric")


@pytest.mark.parametrize("L,radius", [(6, 2), (7, 3)])
def test_masked_tiles_unsymmetric_weights(tiles, L, radius):
    """The adjoint's masked products on tiles (the second operand through its
    transpose): weights that are not symmetric, so neither are the gradients
    that the products take; against the ordered form's gradient (whole
    products, restricted), as test_adjoint_gpu.py does, to 1e-10."""
    import ctypes as C
    N, MH = L ** 3, 128
    v, ix, nz = B.gen_lattice(L, radius, N, MH, 4)
    M = N
    pad = lambda a: np.pad(a.reshape(N, MH), ((0, 0), (0, M - MH)))[:, :M].reshape(-1)  # noqa: E731
    v, ix = pad(v), pad(ix)
    vv = np.random.default_rng(1).uniform(-0.01, 0.01, N * M)
    grads = []
    for exact in (0, 1):
        old = B.lib.bml_b200_set_x2_exact(exact)
        H = B.Ellpack.from_arrays(v, ix, nz, N, M)
        V = B.Ellpack.from_arrays(vv, ix, nz, N, M)
        dH = B.Ellpack(N, M)
        loss = C.c_double()
        B.check(B.lib.bml_b200_sp2_adjoint(H.h, V.h, 1e-5, N / 2.0, 6, 2, M, dH.h, C.byref(loss)))
        assert B.product_form() == ("ordered" if exact else "tiles_masked")
        grads.append((loss.value, dH.download()))
        B.lib.bml_b200_set_x2_exact(old)
    (l0, (g0, i0, n0)), (l1, (g1, i1, n1)) = grads
    assert l0 == pytest.approx(l1, rel=1e-10)
    mask = (np.arange(M)[None, :] < nz[:, None]).reshape(-1)
    assert np.array_equal(n0, n1) and np.array_equal(i0[mask], i1[mask])
    assert np.abs(g0[mask] - g1[mask]).max() <= 1e-10 * np.abs(g1[mask]).max()


def _random_band(N, band, density, seed, empty, dtype):
    rng = np.random.default_rng(seed)
    i, j = np.indices((N, N))
    D = np.where((abs(i - j) <= band) & (rng.random((N, N)) < density), rng.standard_normal((N, N)), 0.0).astype(dtype)
    D[list(empty), :] = 0
    return D


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("square", [False, True], ids=["ab", "x2_not_symmetric"])
@pytest.mark.parametrize("N,ba,bb,density,empty", [
    (1, 0, 0, 1.0, ()), (9, 2, 8, 0.9, (3,)), (32, 31, 5, 0.8, ()), (33, 4, 33, 0.7, (0, 32)),
    (257, 30, 60, 0.6, tuple(range(32, 64))), (400, 399, 20, 0.5, ()), (900, 12, 80, 0.9, ()),
    (4095, 4, 33, 0.7, ()), (4096, 12, 80, 0.9, ()), (4097, 399, 20, 0.5, (0, 4096)),
    (4129, 30, 60, 0.6, tuple(range(32, 64)))])
def test_general_tiles(tiles, N, ba, bb, density, empty, square, dtype):
    """A*B and X^2 of matrices that are not symmetric, rows in any order: the
    kept entries and the diagonal where some product touches it, against the
    dense FP64 product; and the refusal of a row that touches more than M
    columns although fewer are kept."""
    prec = "double_real" if dtype == np.float64 else "single_real"
    Da = _random_band(N, ba, density, 1, empty, dtype)
    Db = Da if square else _random_band(N, bb, density, 2, empty, dtype)
    if N > 8:  # a diagonal that nothing touches
        Da[5, :] = 0
        Db = Da if square else Db
    pa, pb = (Da != 0).astype(float), (Db != 0).astype(float)
    want, S = Da.astype(float) @ Db.astype(float), abs(Da.astype(float)) @ abs(Db.astype(float))
    touched = pa @ pb > 0
    thr = 0.5
    n = int((Da != 0).sum(1).max()) or 1
    tol = (1e-12 if dtype == np.float64 else 2.0 * n * 2.0 ** -24) * S
    keep = abs(want) > thr
    np.fill_diagonal(keep, touched.diagonal())
    ma, mb = (max(1, int((d != 0).sum(1).max())) for d in (Da, Db))
    A = B.Ellpack.from_arrays(*_rows(Da, ma, True, 3), N, ma, prec)
    Bm = A if square else B.Ellpack.from_arrays(*_rows(Db, mb, False, 4), N, mb, prec)
    wide = max(1, int(touched.sum(1).max()))
    for M, status in ((wide, B.OK), (wide - 1, B.ERR_ROW_OVERFLOW)):
        if M < 1 or (square and status != B.OK):
            continue
        Cm = B.Ellpack(N, M, prec)
        B.lib.bml_b200_set_verbose(0)
        if square:
            st, tr = B.multiply_x2(A, Cm, thr)
            assert abs(tr[0] - np.trace(Da.astype(float))) <= 1e-12 * max(1.0, abs(np.diag(Da)).sum())
            assert abs(tr[1] - np.trace(want)) <= (1e-12 if dtype == np.float64 else 1e-5) * max(np.trace(S), 1e-300)
        else:
            B.lib.bml_multiply_AB(A.h, Bm.h, Cm.h, thr)
            st = B.last_error()
        B.clear_error()
        B.lib.bml_b200_set_verbose(1)
        assert st == status
        # (a single row is symmetric)
        assert B.product_form() == ("tiles_symmetric" if square and N == 1 else "tiles")
        if status != B.OK:
            continue
        got = Cm.download()
        assert x2check.rows_sorted(got, M)
        v, ix, nz = got[0].reshape(N, M), got[1].reshape(N, M), got[2]
        G, K = np.zeros((N, N)), np.zeros((N, N), bool)
        for i in range(N):
            G[i, ix[i, :nz[i]]], K[i, ix[i, :nz[i]]] = v[i, :nz[i]], True
        sure = abs(abs(want) - thr) > tol + 1e-300
        sure |= np.eye(N, dtype=bool)
        assert np.array_equal(K[sure], keep[sure])
        assert (abs(G - want)[K] <= (tol + 1e-300)[K] + (abs(want)[K] * 2.0 ** -24 if dtype == np.float32 else 0)).all()


def _random_rows(N, w, seed, symmetric):
    """ELLPACK arrays of w random columns a row."""
    rng = np.random.default_rng(seed)
    D = np.zeros((N, N))
    for i in range(N):
        D[i, rng.choice(N, w, replace=False)] = rng.standard_normal(w)
    if symmetric:
        D = D + D.T
    M = int((D != 0).sum(1).max())
    return D, _rows(D, M, False, 0), M


def _check_dense(got, D, E, thr):
    N = D.shape[0]
    want, S = D @ E, abs(D) @ abs(E)
    G = _dense(got, N, len(got[0]) // N)
    assert (abs(G - want) <= 1e-12 * S + np.where(G == 0, thr, 0.0)).all()


@pytest.mark.parametrize("kind,N,w,form", [
    # few products per tile product: the sparse form, counted while packed and (4200 rows) before
    ("random", 700, 6, "sparse_symmetric"), ("random", 4200, 3, "sparse_symmetric"),
    # the same without symmetry: found by the sample of entries
    ("random_asym", 700, 6, "sparse"), ("random_asym", 4200, 3, "sparse"),
    # a band without symmetry, too little work for the tile form's launches, and enough of it
    ("band_asym", 700, 31, "sparse"), ("band_asym", 3000, 201, "tiles"), ("band_asym", 4200, 201, "tiles"),
    # symmetric but for one entry: found by the check of all
    ("band_one", 700, 31, "sparse"), ("band_one", 4200, 201, "tiles"),
    ("band", 700, 31, "tiles_symmetric"), ("band", 4200, 31, "tiles_symmetric"),
    # a few groups that pack badly among many that do not
    ("mixed", 2000, 61, "tiles_symmetric")])
def test_which_form(kind, N, w, form):
    if kind.startswith("random"):
        D, arrs, M = _random_rows(N, w, 1, kind == "random")
    else:
        D = _random_band(N, w // 2, 1.0, 1, (), np.float64)
        if kind != "band_asym":
            D = np.triu(D) + np.triu(D, 1).T
        if kind == "band_one":
            D[5, 6] += 1.0
        if kind == "mixed":
            far = np.random.default_rng(2).choice(np.arange(64, N), 40, replace=False)
            D[np.arange(40) % 32, far] = D[far, np.arange(40) % 32] = 0.25
        M = int((D != 0).sum(1).max())
        arrs = _rows(D, M, False, 0)
    st, tr, got = _x2(arrs, N, M, min(N, 1024), 1e-9, DOUBLE)
    assert st == B.OK
    assert B.product_form() == form
    _check_dense(got, D, D, 1e-9)


# rooms of 512: up to 4095 rows the lengths are asked first, and the counts where those speak for tiles
@pytest.mark.parametrize("wa,wb,N,form", [(3, 3, 600, "sparse"), (201, 201, 600, "sparse"), (201, 201, 3000, "tiles"),
                                          (1, 41, 2000, "sparse"), (41, 1, 3000, "sparse"), (201, 3, 4200, "tiles"),
                                          (201, 201, 4095, "tiles"), (3, 3, 4095, "sparse"), (3, 3, 4096, "sparse")])
def test_which_form_of_a_product(wa, wb, N, form):
    Da, Db = (_random_band(N, w // 2, 1.0, w, (), np.float64) for w in (wa, wb))
    A, Bm = (B.Ellpack.from_arrays(*_rows(D, 512, False, 0), N, 512) for D in (Da, Db))
    Cm = B.Ellpack(N, min(N, 512))
    B.lib.bml_multiply_AB(A.h, Bm.h, Cm.h, 1e-9)
    B.check()
    assert B.product_form() == form
    _check_dense(Cm.download(), Da, Db, 1e-9)


def test_lengths_for_tiles_and_counts_against():
    """Wide rows of scattered columns: the row lengths speak for tiles, the
    tile products against; the sparse form is begun twice."""
    N, w = 2500, 250
    (D, arrs, M), (E, brrs, _) = (_random_rows(N, w, s, False) for s in (1, 2))
    A, Bm, Cm = B.Ellpack.from_arrays(*arrs, N, M), B.Ellpack.from_arrays(*brrs, N, M), B.Ellpack(N, N)
    B.lib.bml_multiply_AB(A.h, Bm.h, Cm.h, 1e-9)
    B.check()
    assert B.product_form() == "sparse"
    _check_dense(Cm.download(), D, E, 1e-9)


def test_set_tiles():
    D = _banded(300, 20, 1.0, 2)
    arrs = _rows(D, 41, False, 0)
    forms = []
    for mode in (0, 1, 2, 1):
        old = B.lib.bml_b200_set_tiles(mode)
        st, tr, got = _x2(arrs, 300, 41, 128, 0.0, DOUBLE)
        B.lib.bml_b200_set_tiles(old)
        assert st == B.OK and old == 1
        forms.append(B.product_form())
    assert forms == ["sparse_symmetric", "tiles_symmetric", "tiles_symmetric", "tiles_symmetric"]
