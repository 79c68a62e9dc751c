"""Performance cases of the library's public entry points.

Each case is one call, or one short sequence of calls, that a program built on
the library makes: products of ELLPACK and ELLBLOCK matrices, the SP2
purification loop and its adjoint, and the update between two products.  Inputs
have the shapes of this repository's configurations (1-D chains, cubic
lattices, block lattices of 32 x 32 blocks), made on the GPU from a seed.

Interface: listed() and draw(rng) give cases (dicts of plain values);
prepare(case, seed) makes the state a program holds before the call;
run(state) is one pass and returns its outputs; exact(case, seed) is the same
result from plain FP64 torch; work(case) the bytes and operations of a pass;
tolerance(case) the difference another correct implementation may show.
"""
import ctypes as C
import math

import numpy as np
import torch

import bml_b200 as B

DEV = "cuda"
SEQ = 0
ELLPACK, ELLBLOCK = B.TYPE["ellpack"], B.TYPE["ellblock"]
THR = 1e-5  # the threshold of every configuration
BS = 32     # ELLBLOCK block size


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # first X^2 of a small chain: the smallest product a solve makes, launches and host time count
        {"name": "x2_chain_first", "kind": "x2", "shape": "chain", "N": 512, "R": 16.0, "prec": "f64", "M": 96},
        # X^2 in the middle of the chain configuration's solve (N = 4096): rows of about 340
        {"name": "x2_chain_wide", "kind": "x2", "shape": "chain", "N": 4096, "R": 170.0, "prec": "f64", "M": 512},
        # X^2 of a wide SP2 iterate on the 40^3 lattice (N = 64000, M = 2048): the product that bounds the solve
        {"name": "x2_lattice_wide", "kind": "x2", "shape": "lattice", "L": 40, "N": 64000, "R": 6.4, "prec": "f64",
         "M": 2048},
        # first X^2 in FP32 (the bulk phase of a mixed solve), a lattice cut at an odd number of rows
        {"name": "x2_lattice_f32", "kind": "x2", "shape": "lattice", "L": 30, "N": 26999, "R": 3.0, "prec": "f32",
         "M": 896},
        # the headline workload: the first 4 SP2 iterations on the 40^3 lattice, then the band energy
        {"name": "sp2_lattice", "kind": "sp2", "shape": "lattice", "L": 40, "N": 64000, "R": 3.0, "iters": 4,
         "M": 2048},
        # a whole chain solve (fixed count, so every run takes the same steps)
        {"name": "sp2_chain", "kind": "sp2", "shape": "chain", "N": 4096, "R": 16.0, "iters": 30, "M": 512},
        # a general product of two unlike, non-symmetric matrices
        {"name": "ab_lattice", "kind": "ab", "L": 28, "N": 21951, "R": 3.0, "R2": 4.5, "M": 2048},
        # the update X <- 2X - X^2 of an SP2 step written by the caller, with the old iterate kept
        {"name": "update_lattice", "kind": "update", "L": 40, "N": 64000, "R": 6.0, "R2": 6.6, "M": 2048},
        # late iterates of a metallic system fill in to dense rows
        {"name": "x2_filled", "kind": "filled", "N": 5001, "M": 5001},
        # ELLBLOCK X^2 in FP64 on a block lattice
        {"name": "eb_x2", "kind": "eb_x2", "L": 11, "R": 2.0, "MB": 264},
        # mixed ELLBLOCK SP2: tensor-core iterations closed by one in FP64
        {"name": "eb_sp2_mixed", "kind": "eb_sp2", "L": 7, "R": 2.0, "iters": 5, "split": 1, "nclose": 1},
        # the backward direction: dL/dH through 3 SP2 iterations
        {"name": "adjoint_lattice", "kind": "adjoint", "L": 16, "N": 4096, "R": 3.0, "iters": 3, "every": 2,
         "M": 1536},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lattice_rows(rng, L):
    """All sites, or a cut at an odd place."""
    full = L ** 3
    return full if rng.random() < 0.3 else full - rng.randrange(1, max(2, full // 8))


def draw(rng):
    kind = rng.choice(["x2c", "x2l", "x2l", "x2f32", "sp2l", "sp2c", "ab", "update", "filled", "eb_x2", "eb_tc",
                       "eb_sp2", "adjoint"])
    if kind == "x2c":
        N = _log_int(rng, 300, 40000)
        R = min(_log_int(rng, 16, 240), N // 4)
        return {"kind": "x2", "shape": "chain", "N": N, "R": float(R), "prec": "f64", "M": 3 * R + 64}
    if kind == "x2l":
        L = rng.randrange(15, 41)
        R = rng.choice([3.0, 4.0, 4.5, 5.0, 5.5, 6.0, 6.4])
        return {"kind": "x2", "shape": "lattice", "L": L, "N": _lattice_rows(rng, L), "R": R, "prec": "f64",
                "M": 2048}
    if kind == "x2f32":
        L = rng.randrange(12, 41)
        return {"kind": "x2", "shape": "lattice", "L": L, "N": _lattice_rows(rng, L),
                "R": rng.choice([2.0, 3.0, 3.5]), "prec": "f32", "M": 1536}
    if kind == "sp2l":
        L = rng.randrange(14, 37)
        return {"kind": "sp2", "shape": "lattice", "L": L, "N": L ** 3, "R": 3.0, "iters": rng.randrange(1, 4),
                "M": 2048}
    if kind == "sp2c":
        return {"kind": "sp2", "shape": "chain", "N": _log_int(rng, 600, 8000), "R": 16.0,
                "iters": rng.randrange(10, 31), "M": 512}
    if kind == "ab":
        L = rng.randrange(12, 31)
        return {"kind": "ab", "L": L, "N": _lattice_rows(rng, L), "R": rng.choice([2.0, 3.0]),
                "R2": rng.choice([2.5, 3.5, 4.5]), "M": 2048}
    if kind == "update":
        L = rng.randrange(15, 41)
        R = rng.choice([3.0, 4.0, 5.0, 6.0])
        return {"kind": "update", "L": L, "N": _lattice_rows(rng, L), "R": R, "R2": R + 0.6, "M": 2048}
    if kind == "filled":
        N = _log_int(rng, 1100, 5001)
        return {"kind": "filled", "N": N, "M": N}
    if kind == "eb_x2":
        return {"kind": "eb_x2", "L": rng.randrange(3, 12), "R": rng.choice([1.0, 1.5, 2.0]), "MB": 264}
    if kind == "eb_tc":
        return {"kind": "eb_tc", "L": rng.randrange(3, 14), "R": rng.choice([1.0, 1.5, 2.0]), "MB": 264,
                "split": rng.randrange(2)}
    if kind == "eb_sp2":
        return {"kind": "eb_sp2", "L": rng.randrange(3, 8), "R": rng.choice([1.5, 2.0]), "iters": rng.randrange(2, 5),
                "split": 1, "nclose": 1}
    L = rng.randrange(8, 16)
    iters = rng.randrange(1, 4)
    return {"kind": "adjoint", "L": L, "N": L ** 3, "R": rng.choice([2.0, 3.0]), "iters": iters,
            "every": rng.randrange(1, iters + 1), "M": min(1536, L ** 3)}


# ---------------------------------------------------------------------------
# inputs: cols, vals, present of shape (rows, offsets), columns ascending
# ---------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(1 + int(seed))
    return g


def _offsets(shape, L, R):
    """(shift, distance, displacement) of the sites within R, by ascending shift."""
    if shape == "chain":
        r = int(R)
        return [(d, float(abs(d)), (d, 0, 0)) for d in range(-r, r + 1)]
    r = int(R)
    out = []
    for z in range(-r, r + 1):
        for y in range(-r, r + 1):
            for x in range(-r, r + 1):
                if x * x + y * y + z * z <= R * R:
                    out.append((x + L * y + L * L * z, math.sqrt(x * x + y * y + z * z), (x, y, z)))
    return sorted(out)


def _sites(N, L, shape):
    i = torch.arange(N, device=DEV)
    if shape == "chain":
        return i, torch.zeros_like(i), torch.zeros_like(i)
    return i % L, (i // L) % L, i // (L * L)


def _stencil(shape, L, N, R, seed, amplitude, diagonal, noise, symmetric=True, cut=0.0):
    """Entries amplitude(d) * noise(draw) for every pair of sites within R, diagonal(draw) on the diagonal."""
    g = _generator(seed)
    offs = _offsets(shape, L, R)
    W, mid = len(offs), len(offs) // 2
    x, y, z = _sites(N, L, shape)
    rows = torch.arange(N, device=DEV)
    vals = torch.zeros(N, W, dtype=torch.float64, device=DEV)
    here = torch.zeros(N, W, dtype=torch.bool, device=DEV)
    vals[:, mid] = diagonal(torch.randn(N, generator=g, device=DEV, dtype=torch.float64))
    here[:, mid] = True
    side = N if shape == "chain" else L
    for p in range(mid + 1, W):
        s, d, (dx, dy, dz) = offs[p]
        ok = (x + dx >= 0) & (x + dx < side) & (rows + s < N)
        if shape != "chain":
            ok &= (y + dy >= 0) & (y + dy < L) & (z + dz >= 0) & (z + dz < L)
        v = amplitude(d) * noise(torch.randn(N, generator=g, device=DEV, dtype=torch.float64))
        u = v if symmetric else amplitude(d) * noise(torch.randn(N, generator=g, device=DEV, dtype=torch.float64))
        if cut > 0.0:
            keep = ok & (v.abs() > cut)
            ok_u = ok & (u.abs() > cut)
        else:
            keep = ok_u = ok
        vals[:, p] = torch.where(keep, v, 0.0)
        here[:, p] = keep
        q = W - 1 - p
        if s < N:
            vals[s:, q] = torch.where(ok_u, u, 0.0)[: N - s]
            here[s:, q] = ok_u[: N - s]
    cols = rows[:, None] + torch.tensor([o[0] for o in offs], device=DEV)[None, :]
    return cols, vals, here


def _hamiltonian(case, seed):
    """The chain and lattice Hamiltonians of the configurations."""
    if case["shape"] == "chain":
        return _stencil("chain", 0, case["N"], case["R"], seed, lambda d: math.exp(-d / 4.0),
                        lambda g: torch.erf(g / math.sqrt(2.0)), lambda g: torch.erf(g / math.sqrt(2.0)))
    return _stencil("lattice", case["L"], case["N"], case["R"], seed, lambda d: -math.exp(-d), lambda g: g,
                    lambda g: 1.0 + 0.1 * g)


def _iterate(shape, L, N, R, seed, symmetric=True):
    """A matrix like an SP2 iterate: half-filled diagonal, decaying oscillating entries, those below the threshold
    missing."""
    alpha = math.log(0.15 / (2.0 * THR)) / max(R - 1.0, 1.0)
    return _stencil(shape, L, N, R, seed, lambda d: 0.15 * math.exp(-alpha * (d - 1.0)) * math.cos(2.2 * d),
                    lambda g: 0.5 + 0.1 * g, lambda g: 1.0 + 0.2 * g, symmetric, THR)


def _positive(shape, L, N, R, seed):
    """Entries of one sign, so that every structural entry of the FP32 product stays far above the threshold and its
    pattern does not depend on rounding."""
    return _stencil(shape, L, N, R, seed, lambda d: math.exp(-d), lambda g: 1.0 + 0.1 * g.clamp(-3, 3),
                    lambda g: 1.0 + 0.1 * g.clamp(-3, 3))


def _input(case, seed):
    shape, L, N, R = case.get("shape", "lattice"), case.get("L", 0), case["N"], case["R"]
    if case["kind"] in ("sp2", "adjoint"):
        return _hamiltonian(dict(case, shape=shape), seed)
    if case.get("prec") == "f32":
        return _positive(shape, L, N, R, seed)
    if R <= 3.0 or (shape == "chain" and R <= 16.0):
        return _hamiltonian(dict(case, shape=shape), seed)
    return _iterate(shape, L, N, R, seed, case["kind"] != "ab")


def _filled(N, seed):
    g = _generator(seed)
    a = torch.randn(N, N, generator=g, device=DEV, dtype=torch.float64) * (0.1 / math.sqrt(N))
    a = a + a.T
    a.diagonal().add_(0.5)
    return a


# ---------------------------------------------------------------------------
# matrices and their device arrays
# ---------------------------------------------------------------------------
class _View:
    """A device array; `owner` keeps the matrix that holds it alive as long as a tensor of it is in use."""

    def __init__(self, ptr, shape, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "data": (ptr, False),
                                         "version": 3, "strides": None, "stream": None}


def _tensor(ptr, shape, typestr, owner):
    return torch.as_tensor(_View(ptr, shape, typestr, owner), device=DEV)


def _arrays(m):
    """The device arrays (value[N, ld], index[N, ld], nnz[N]) of an ELLPACK matrix, as tensors."""
    pv, pi, pn, ld = C.c_void_p(), C.POINTER(C.c_int)(), C.POINTER(C.c_int)(), C.c_int()
    B.check(B.lib.bml_b200_ellpack_device_arrays(m.h, C.byref(pv), C.byref(pi), C.byref(pn), C.byref(ld)))
    at = lambda p: C.cast(p, C.c_void_p).value  # noqa: E731
    return (_tensor(pv.value, (m.N, ld.value), "<f8" if m.prec == 2 else "<f4", m),
            _tensor(at(pi), (m.N, ld.value), "<i4", m), _tensor(at(pn), (m.N,), "<i4", m))


def _empty(N, M, prec="f64"):
    """A zero matrix with the arrays past its rows' ends zeroed too, so that an output compares whole."""
    m = B.Ellpack(N, M, "double_real" if prec == "f64" else "single_real")
    for t in _arrays(m):
        t.zero_()
    torch.cuda.synchronize()
    return m


def _load(cols, vals, here, M, prec="f64"):
    N, W = vals.shape
    m = _empty(N, M, prec)
    v, ix, nz = _arrays(m)
    for a in range(0, N, 16384):
        b = min(N, a + 16384)
        h = here[a:b]
        at = torch.cumsum(h, 1) - 1
        r, p = h.nonzero(as_tuple=True)
        q = at[r, p]
        v[a + r, q] = vals[a:b][r, p].to(v.dtype)
        ix[a + r, q] = cols[a:b][r, p].to(torch.int32)
        nz[a:b] = h.sum(1).to(torch.int32)
    torch.cuda.synchronize()
    return m


class _EllblockStruct(C.Structure):
    """The public leading fields of an ELLBLOCK matrix, and the device arrays after them."""
    _fields_ = [("matrix_type", C.c_int), ("matrix_precision", C.c_int), ("distribution_mode", C.c_int),
                ("N", C.c_int), ("M", C.c_int), ("NB", C.c_int), ("MB", C.c_int), ("ptr_value", C.c_void_p),
                ("indexb", C.c_void_p), ("nnzb", C.c_void_p), ("bsize", C.c_void_p), ("domain", C.c_void_p),
                ("domain2", C.c_void_p), ("h_pool", C.c_void_p), ("d_pool", C.c_void_p), ("d_indexb", C.c_void_p),
                ("d_nnzb", C.c_void_p)]


class _Handle:
    def __init__(self, h):
        B.check()
        self.h = h

    def __del__(self):
        try:
            h = C.c_void_p(self.h)
            B.lib.bml_deallocate(C.byref(h))
        except Exception:
            pass


class _Ellblock:
    def __init__(self, h):
        own = _Handle(h)
        self.h, self.own = h, own
        s = _EllblockStruct.from_address(h)
        self.arrays = (_tensor(s.d_pool, (s.NB, s.MB, BS, BS), "<f8", own),
                       _tensor(s.d_indexb, (s.NB, s.MB), "<i4", own), _tensor(s.d_nnzb, (s.NB,), "<i4", own))


def _partition(nb, mb):
    B.lib.bml_b200_reset_block_sizes()
    B.lib.bml_set_block_sizes((C.c_int * nb)(*([BS] * nb)), nb, mb)


def _eb_empty(nb, mb):
    _partition(nb, mb)
    return _Ellblock(B.lib.bml_zero_matrix(ELLBLOCK, 2, nb * BS, nb * BS, SEQ))


def _eb_input(L, R, seed):
    """Blocks (NB, W, 32, 32) of a symmetric block lattice, entries N(0,1) exp(-d): columns, values, present."""
    g = _generator(seed)
    nb = L ** 3
    offs = [o for o in _offsets("lattice", max(L, 2 * int(R) + 1), R)]
    x, y, z = _sites(nb, L, "lattice")
    out = []
    for _, d, (dx, dy, dz) in offs:
        s = dx + L * dy + L * L * dz
        ok = (x + dx >= 0) & (x + dx < L) & (y + dy >= 0) & (y + dy < L) & (z + dz >= 0) & (z + dz < L)
        out.append((s, d, ok))
    order = sorted(range(len(out)), key=lambda k: out[k][0])
    # blocks of a small lattice may share a shift; only one of them is present in a given row
    cols = torch.stack([torch.arange(nb, device=DEV) + out[k][0] for k in order], 1)
    here = torch.stack([out[k][2] for k in order], 1)
    W = len(order)
    blocks = torch.zeros(nb, W, BS, BS, dtype=torch.float64, device=DEV)
    place = {offs[k][2]: p for p, k in enumerate(order)}
    for p, k in enumerate(order):
        (dx, dy, dz), (s, d, ok) = offs[k][2], out[k]
        if (dz, dy, dx) < (0, 0, 0):
            continue
        blk = torch.randn(nb, BS, BS, generator=g, device=DEV, dtype=torch.float64) * math.exp(-d)
        if (dx, dy, dz) == (0, 0, 0):
            blocks[:, p] = 0.5 * (blk + blk.transpose(1, 2))
            continue
        rows = ok.nonzero()[:, 0]
        blocks[rows, p] = blk[rows]
        blocks[rows + s, place[(-dx, -dy, -dz)]] = blk[rows].transpose(1, 2)
    return cols, blocks, here


def _eb_load(cols, blocks, here, mb):
    """The block lattice as an ELLBLOCK matrix, through an ELLPACK one."""
    nb, W = here.shape
    order = torch.argsort(torch.where(here, cols, nb + cols.abs()), dim=1, stable=True)
    lines = torch.gather(here, 1, order)
    k = torch.gather(cols, 1, order)
    blk = torch.gather(blocks, 1, order[:, :, None, None].expand(-1, -1, BS, BS))
    e = _empty(nb * BS, W * BS)
    v, ix, nz = _arrays(e)
    v.view(nb, BS, -1)[:, :, : W * BS] = blk.permute(0, 2, 1, 3).reshape(nb, BS, W * BS)
    c = (k[:, None, :, None] * BS + torch.arange(BS, device=DEV)).expand(nb, BS, W, BS)
    ix.view(nb, BS, -1)[:, :, : W * BS] = torch.where(lines[:, None, :, None], c, 0).reshape(nb, BS, W * BS).to(torch.int32)
    nz.copy_((lines.sum(1) * BS).repeat_interleave(BS).to(torch.int32))
    torch.cuda.synchronize()
    _partition(nb, mb)
    return _Ellblock(B.lib.bml_convert(e.h, ELLBLOCK, 2, nb * BS, SEQ))


# ---------------------------------------------------------------------------
# states and passes
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "x2":
        s["X"] = _load(*_input(case, seed), case["M"], case["prec"])
        s["C"] = _empty(case["N"], case["M"], case["prec"])
    elif kind == "filled":
        N, M = case["N"], case["M"]
        s["X"] = _empty(N, M)
        v, ix, nz = _arrays(s["X"])
        v[:, :N] = _filled(N, seed)
        ix[:, :N] = torch.arange(N, device=DEV, dtype=torch.int32)
        nz.fill_(N)
        s["C"] = _empty(N, M)
    elif kind == "sp2":
        s["H"] = _load(*_input(case, seed), case["M"])
        s["D"] = B.Ellpack(case["N"], case["M"])
        s["C"] = _empty(case["N"], case["M"])
        s["iters"], s["occ"], s["info"] = case["iters"], case["N"] / 2.0, (C.c_double * 6)()
    elif kind == "ab":
        s["A"] = _load(*_input(case, seed), case["M"])
        s["B"] = _load(*_input(dict(case, R=case["R2"]), seed + 7919), case["M"])
        s["C"] = _empty(case["N"], case["M"])
    elif kind == "update":
        s["X"] = _load(*_input(case, seed), case["M"])
        s["X2"] = _load(*_input(dict(case, R=case["R2"]), seed + 7919), case["M"])
        s["W"] = B.Ellpack(case["N"], case["M"])
        s["C"] = _empty(case["N"], case["M"])
    elif kind in ("eb_x2", "eb_tc"):
        cols, blocks, here = _eb_input(case["L"], case["R"], seed)
        nb = case["L"] ** 3
        s["X"] = _eb_load(cols, blocks, here, here.shape[1])
        s["C"] = _eb_empty(nb, min(nb, case["MB"]))
        s["split"] = case.get("split", 0)
    elif kind == "eb_sp2":
        nb = case["L"] ** 3
        cols, blocks, here = _eb_input(case["L"], case["R"], seed)
        s["H"] = _eb_load(cols, blocks, here, nb)
        s["D"], s["C"] = _eb_empty(nb, nb), _eb_empty(nb, nb)
        s.update(iters=case["iters"], split=case["split"], nclose=case["nclose"], occ=nb * BS / 2.0,
                 info=(C.c_double * 8)())
    else:
        cols, vals, here = _input(case, seed)
        s["H"] = _load(cols, vals, here, case["M"])
        s["V"] = _load(cols, _weights(cols, here, seed), here, case["M"])
        s["dH"] = B.Ellpack(case["N"], case["M"])
        s["C"] = _empty(case["N"], case["M"])
        s.update(iters=case["iters"], every=case["every"], M=case["M"], occ=case["N"] / 2.0)
    s["out"] = s["C"].arrays if kind.startswith("eb_") else _arrays(s["C"])
    torch.cuda.synchronize()
    return s


def _weights(cols, here, seed):
    """Symmetric weights of the loss on H's pattern."""
    i = torch.arange(cols.shape[0], device=DEV)[:, None]
    lo, hi = torch.minimum(i, cols).double(), torch.maximum(i, cols).double()
    return torch.where(here, 0.01 * torch.sin(12.9898 * lo + 78.233 * hi + (seed % 1000)), 0.0)


def run(s):
    kind, lib = s["kind"], B.lib
    if kind in ("x2", "filled"):
        st, tr = B.multiply_x2(s["X"], s["C"], THR if kind == "x2" else 1e-9)
        B.check(st)
        return [*s["out"], tr[0], tr[1]]
    if kind == "sp2":
        B.check(lib.bml_b200_sp2(s["H"].h, s["D"].h, THR, s["occ"], s["iters"], -1.0, 0, s["info"]))
        energy = lib.bml_trace_mult(s["D"].h, s["H"].h)
        lib.bml_copy(s["D"].h, s["C"].h)
        return [*s["out"], energy, s["info"][2]]
    if kind == "ab":
        lib.bml_multiply_AB(s["A"].h, s["B"].h, s["C"].h, THR)
        B.check()
        return list(s["out"])
    if kind == "update":
        lib.bml_copy(s["X"].h, s["W"].h)
        lib.bml_add(s["W"].h, s["X2"].h, 2.0, -1.0, THR)
        lib.bml_copy(s["W"].h, s["C"].h)
        B.check()
        return list(s["out"])
    if kind == "eb_x2":
        tr = (C.c_double * 2)()
        B.check(lib.bml_b200_multiply_x2(s["X"].h, s["C"].h, THR, tr))
        return [*s["out"], tr[0], tr[1]]
    if kind == "eb_tc":
        tr = (C.c_double * 2)()
        lib.bml_b200_set_tc_split(s["split"])
        B.check(lib.bml_b200_ellblock_multiply_x2_tc(s["X"].h, s["C"].h, THR, tr))
        return [*s["out"], tr[0], tr[1]]
    if kind == "eb_sp2":
        lib.bml_b200_set_tc_split(s["split"])
        B.check(lib.bml_b200_ellblock_sp2_mixed(s["H"].h, s["D"].h, THR, s["occ"], s["iters"], -1.0, 0, s["nclose"],
                                                s["info"]))
        lib.bml_copy(s["D"].h, s["C"].h)
        return [*s["out"], s["info"][2]]
    loss = C.c_double()
    B.check(lib.bml_b200_sp2_adjoint(s["H"].h, s["V"].h, THR, s["occ"], s["iters"], s["every"], s["M"], s["dH"].h,
                                     C.byref(loss)))
    lib.bml_copy(s["dH"].h, s["C"].h)
    B.check()
    return [*s["out"], loss.value]


# ---------------------------------------------------------------------------
# the same results from dense FP64 torch
# ---------------------------------------------------------------------------
def _ld(M):
    return (M + 31) // 32 * 32


class _Rows:
    """ELLPACK arrays filled row block by row block."""

    def __init__(self, N, M, dtype=torch.float64):
        self.v = torch.zeros(N, _ld(M), dtype=dtype, device=DEV)
        self.ix = torch.zeros(N, _ld(M), dtype=torch.int32, device=DEV)
        self.nz = torch.zeros(N, dtype=torch.int32, device=DEV)

    def put(self, r0, dense, keep, c0=0, key=None):
        r, k = keep.nonzero(as_tuple=True)
        if key is not None:
            order = torch.argsort(r * (int(key.max()) + 1) + key[r, k])
            r, k = r[order], k[order]
        n = keep.sum(1)
        q = torch.arange(r.numel(), device=DEV) - torch.repeat_interleave(torch.cumsum(n, 0) - n, n)
        self.v[r0 + r, q] = dense[r, k].to(self.v.dtype)
        self.ix[r0 + r, q] = (c0 + k).to(torch.int32)
        self.nz[r0:r0 + keep.shape[0]] = n.to(torch.int32)

    def arrays(self):
        return [self.v, self.ix, self.nz]


def _dense(cols, vals, here, r0, r1, c0, c1):
    out = torch.zeros(r1 - r0, c1 - c0, dtype=torch.float64, device=DEV)
    r, p = here[r0:r1].nonzero(as_tuple=True)
    c = cols[r0:r1][r, p] - c0
    ok = (c >= 0) & (c < c1 - c0)
    out[r[ok], c[ok]] = vals[r0:r1][r[ok], p[ok]]
    return out


def _product(a, b, M, diagonal=True):
    """Rows of A B by dense products of the windows that hold the entries."""
    N = a[0].shape[0]
    out = _Rows(N, M)
    tr = 0.0
    reach = lambda m: int((m[0] - torch.arange(N, device=DEV)[:, None]).abs().where(m[2], 0).max())  # noqa: E731
    ha, hb = reach(a), reach(b)
    step = max(64, min(2048, N))
    for r0 in range(0, N, step):
        r1 = min(N, r0 + step)
        j0, j1 = max(0, r0 - ha), min(N, r1 + ha)
        k0, k1 = max(0, j0 - hb), min(N, j1 + hb)
        x = _dense(*a, r0, r1, j0, j1) @ _dense(*b, j0, j1, k0, k1)
        keep = x.abs() > THR
        rows = torch.arange(r0, r1, device=DEV)
        if diagonal:
            keep[rows - r0, rows - k0] = True
        tr += float(x[rows - r0, rows - k0].sum())
        out.put(r0, x, keep, k0)
    return out, tr


def _start(h, N):
    """X0 of SP2, dense, with its normalisation: (X0, emin, emax)."""
    H = _dense(*h, 0, N, 0, N)
    d = H.diagonal()
    radius = H.abs().sum(1) - d.abs()
    emax, emin = float((d + radius).max()), float((d - radius).min())
    X = H * (-1.0 / (emax - emin))
    X.diagonal().add_(emax / (emax - emin))
    return H, X, emin, emax


def _sp2_dense(X, here, iters, occ):
    """SP2 steps with the library's keep rules and row order: yields (X, here, key, X2 here, branch)."""
    N = X.shape[0]
    cols = torch.arange(N, device=DEV)[None, :]
    key = cols.expand(N, N).clone()
    eye = torch.eye(N, dtype=torch.bool, device=DEV)
    for n in range(iters):
        Y = X @ X
        t, t2 = float(X.trace()), float(Y.trace())
        keep = (Y.abs() > THR) | eye
        Y = torch.where(keep, Y, 0.0)
        if abs(t2 - occ) <= abs(2 * t - t2 - occ):
            branch, Z, now, nkey = 0, Y, keep, cols.expand(N, N).clone()
        else:
            branch, Z = 1, 2 * X - Y
            now = (here | keep) & (Z.abs() > THR)
            nkey = torch.where(here, key, cols + (n + 1) * N)
            Z = torch.where(now, Z, 0.0)
        yield X, here, Z, now, nkey, keep, branch
        X, here, key = Z, now, nkey


def _pairs(cols, blocks, here):
    """Every block product (ib, jb, kb) of the square of a block matrix, in the order of the rows."""
    nb = here.shape[0]
    row = [[(int(c), p) for p, c in enumerate(cs) if hs[p]] for cs, hs in zip(cols.tolist(), here.tolist())]
    for r in row:
        r.sort()
    for ib in range(nb):
        for jb, p in row[ib]:
            for kb, q in row[jb]:
                yield ib, jb, kb, p, q


def _eb_square(cols, blocks, here, mb, ascending):
    nb, W = here.shape
    arr = np.array([(ib, jb, kb, p, q) for ib, jb, kb, p, q in _pairs(cols, blocks, here)], dtype=np.int64)
    flat = arr[:, 0] * nb + arr[:, 2]
    uniq, first, inv = np.unique(flat, return_index=True, return_inverse=True)
    n = len(uniq)
    acc = torch.zeros(n, BS, BS, dtype=torch.float64, device=DEV)
    t = torch.from_numpy(arr).to(DEV)
    inv_t = torch.from_numpy(inv.reshape(-1)).to(DEV)
    for a in range(0, len(arr), 65536):
        s = t[a:a + 65536]
        acc.index_add_(0, inv_t[a:a + 65536], torch.bmm(blocks[s[:, 0], s[:, 3]], blocks[s[:, 1], s[:, 4]]))
    ib, kb = uniq // nb, uniq % nb
    keep = (acc.abs().amax((1, 2)) > THR).cpu().numpy() | (ib == kb)
    pool = torch.zeros(nb, mb, BS, BS, dtype=torch.float64, device=DEV)
    index = np.full((nb, mb), -1, dtype=np.int32)
    nnzb = np.zeros(nb, dtype=np.int32)
    order = np.lexsort((kb if ascending else first, ib))
    order = order[keep[order]]
    pos = np.arange(len(order)) - np.searchsorted(ib[order], ib[order])
    index[ib[order], pos] = kb[order]
    np.add.at(nnzb, ib[order], 1)
    o = torch.from_numpy(order).to(DEV)
    pool[torch.from_numpy(ib[order]).to(DEV), torch.from_numpy(pos).to(DEV)] = acc[o]
    d = torch.from_numpy(np.nonzero(ib == kb)[0]).to(DEV)
    dx = blocks[torch.arange(nb, device=DEV), torch.from_numpy(
        np.argmax((cols.cpu().numpy() == np.arange(nb)[:, None]) & here.cpu().numpy(), 1)).to(DEV)]
    return [pool, torch.from_numpy(index).to(DEV), torch.from_numpy(nnzb).to(DEV),
            float(dx.diagonal(dim1=1, dim2=2).sum()), float(acc[d].diagonal(dim1=1, dim2=2).sum())]


def exact(case, seed):
    kind = case["kind"]
    if kind == "x2":
        x = _input(case, seed)
        if case["prec"] == "f32":
            x = (x[0], x[1].float().double(), x[2])
        out, t2 = _product(x, x, case["M"])
        mid = x[1].shape[1] // 2
        return [*out.arrays(), float(x[1][:, mid].sum()), t2]
    if kind == "filled":
        N = case["N"]
        a = _filled(N, seed)
        x = a @ a
        out = _Rows(N, case["M"])
        out.put(0, x, (x.abs() > 1e-9) | torch.eye(N, dtype=torch.bool, device=DEV))
        return [*out.arrays(), float(a.trace()), float(x.trace())]
    if kind == "ab":
        return _product(_input(case, seed), _input(dict(case, R=case["R2"]), seed + 7919), case["M"])[0].arrays()
    if kind == "update":
        N = case["N"]
        a, b = _input(case, seed), _input(dict(case, R=case["R2"]), seed + 7919)
        pa, pb = (m[:2] + (m[2],) for m in (a, b))
        ones = lambda m: (m[0], m[2].double(), m[2])  # noqa: E731
        out = _Rows(N, case["M"])
        for r0 in range(0, N, 1000):
            r1 = min(N, r0 + 1000)
            ina = _dense(*ones(pa), r0, r1, 0, N) > 0
            x = 2.0 * _dense(*pa, r0, r1, 0, N) - _dense(*pb, r0, r1, 0, N)
            key = torch.arange(N, device=DEV)[None, :] + torch.where(ina, 0, N)
            out.put(r0, x, x.abs() > THR, 0, key)
        return out.arrays()
    if kind == "sp2":
        N = case["N"]
        if N > 16384:
            return None  # dense FP64 iterations take too long
        h = _input(case, seed)
        H, X, _, _ = _start(h, N)
        here = X != 0
        key = None
        for _, _, X, here, key, _, _ in _sp2_dense(X, here, case["iters"], N / 2.0):
            pass
        out = _Rows(N, case["M"])
        out.put(0, X, here, 0, key)
        return [*out.arrays(), float((X * H).sum()), float(X.trace())]
    if kind in ("eb_x2", "eb_tc"):
        cols, blocks, here = _eb_input(case["L"], case["R"], seed)
        return _eb_square(cols, blocks, here, min(here.shape[0], case["MB"]), kind == "eb_tc")
    if kind == "eb_sp2":
        return _eb_sp2_exact(case, seed)
    N = case["N"]
    cols, vals, here0 = h = _input(case, seed)
    H, X0, emin, emax = _start(h, N)
    V = _dense(cols, _weights(cols, here0, seed), here0, 0, N, 0, N)
    steps = list(_sp2_dense(X0, X0 != 0, case["iters"], N / 2.0))
    loss = float((steps[-1][2] * V).sum())
    G = torch.where(steps[-1][3], V, 0.0)
    for X, here, _, _, _, keep, branch in reversed(steps):
        Gh = G * keep if branch == 0 else -(G * keep)
        Gn = Gh @ X.T + X.T @ Gh
        if branch:
            Gn = Gn + 2.0 * G
        G = torch.where(here, Gn, 0.0)
    s = emax - emin
    gd, gh = float(G.trace()), float((G * H).sum())
    d_emax = gd / s - gd * emax / s ** 2 + gh / s ** 2
    d_emin = gd * emax / s ** 2 - gh / s ** 2
    dH = -G / s
    d = H.diagonal()
    radius = H.abs().sum(1) - d.abs()
    for w, r, sign in ((d_emax, int((d + radius).argmax()), 1.0), (d_emin, int((d - radius).argmin()), -1.0)):
        line = sign * torch.sign(H[r])
        line[r] = 1.0
        dH[r] += w * line
    out = _Rows(N, case["M"])
    out.put(0, dH, _dense(cols, here0.double(), here0, 0, N, 0, N) > 0)
    return [*out.arrays(), loss]


def _eb_sp2_exact(case, seed):
    """SP2 on the dense matrix with the block keep rules; blocks of a row in the library's order."""
    cols, blocks, here = _eb_input(case["L"], case["R"], seed)
    nb, W = here.shape
    N = nb * BS
    H = torch.zeros(nb, BS, nb, BS, dtype=torch.float64, device=DEV)
    r, p = here.nonzero(as_tuple=True)
    H[r, :, cols[r, p], :] = blocks[r, p]
    H = H.reshape(N, N)
    d = H.diagonal()
    radius = H.abs().sum(1) - d.abs()
    emax, emin = float((d + radius).max()), float((d - radius).min())
    X = H * (-1.0 / (emax - emin))
    X.diagonal().add_(emax / (emax - emin))
    del H
    norm = lambda m: m.reshape(nb, BS, nb, BS).abs().amax((1, 3))  # noqa: E731
    wide = lambda m: m.repeat_interleave(BS, 0).repeat_interleave(BS, 1)  # noqa: E731
    eye = torch.eye(nb, dtype=torch.bool, device=DEV)
    pat = norm(X) > 0
    index = torch.arange(nb, device=DEV)[None, :].expand(nb, nb)
    rows = [[int(k) for k in pat[i].nonzero()[:, 0]] for i in range(nb)]  # block columns in order
    occ = N / 2.0
    near = False  # some block so close to the threshold that the split's own error may decide it
    for n in range(case["iters"]):
        tensor_core = n < case["iters"] - case["nclose"]
        Y = X @ X
        t, t2 = float(X.trace()), float(Y.trace())
        keep = ((norm(Y) > THR) | eye) & ((pat.double() @ pat.double()) > 0)
        near |= bool(((norm(Y) / THR - 1.0).abs() < 1e-4).any())
        if tensor_core:
            yrows = [[int(k) for k in keep[i].nonzero()[:, 0]] for i in range(nb)]
        else:
            yrows = []
            for i in range(nb):
                order = dict.fromkeys(k for j in rows[i] for k in rows[j])
                ok = keep[i].tolist()
                yrows.append([k for k in order if ok[k]])
        Y = torch.where(wide(keep), Y, 0.0)
        if abs(t2 - occ) <= abs(2 * t - t2 - occ):
            X, pat, rows = Y, keep, yrows
        else:
            X = 2 * X - Y
            now = (pat | keep) & (norm(X) > THR)
            near |= bool(((norm(X) / THR - 1.0).abs() < 1e-4).any())
            merged = []
            for i in range(nb):
                ok = now[i].tolist()
                merged.append([k for k in dict.fromkeys(rows[i] + yrows[i]) if ok[k]])
            X, pat, rows = torch.where(wide(now), X, 0.0), now, merged
    del index
    pool = torch.zeros(nb, nb, BS, BS, dtype=torch.float64, device=DEV)
    ix = torch.full((nb, nb), -1, dtype=torch.int32, device=DEV)
    nz = torch.tensor([len(r) for r in rows], dtype=torch.int32, device=DEV)
    X4 = X.reshape(nb, BS, nb, BS)
    for i in range(nb):
        k = torch.tensor(rows[i], dtype=torch.int64, device=DEV)
        pool[i, : len(rows[i])] = X4[i][:, k].permute(1, 0, 2)
        ix[i, : len(rows[i])] = k.to(torch.int32)
    return [None, None, None, float(X.trace())] if near else [pool, ix, nz, float(X.trace())]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _row_counts(shape, L, N, R):
    """Sites within R of each site."""
    if shape == "chain":
        i = np.arange(N)
        return (np.minimum(i, int(R)) + np.minimum(N - 1 - i, int(R)) + 1).astype(np.float64)
    n = np.zeros((L, L, L))
    for _, _, (x, y, z) in _offsets("lattice", L, R):
        if max(abs(x), abs(y), abs(z)) < L:
            n[max(0, -z):L - max(0, z), max(0, -y):L - max(0, y), max(0, -x):L - max(0, x)] += 1
    return n.reshape(-1)[:N]


def work(case):
    """Bytes: every input read once, every output written once.  Flops: 2 per product term; a symmetric square
    needs the terms of one triangle."""
    kind = case["kind"]
    shape, L, N = case.get("shape", "lattice"), case.get("L", 0), case.get("N", 0)
    entry = 8 if case.get("prec") == "f32" else 12
    if kind == "x2":
        n = _row_counts(shape, L, N, case["R"])
        # kept width: the whole reach of a structural square, about a site more for a thresholded one
        grow = 2 * case["R"] if case["R"] <= 3.5 or (shape == "chain" and case["R"] <= 16) else (
            case["R"] * 1.25 if shape == "chain" else case["R"] + 0.8)
        m = _row_counts(shape, L, N, grow)
        return {"bytes": entry * (n.sum() + m.sum()) + 8 * N, "flops": float((n * n).sum())}
    if kind == "filled":
        return {"bytes": 24.0 * N * N, "flops": float(N) ** 3}
    if kind == "ab":
        a, b = _row_counts("lattice", L, N, case["R"]), _row_counts("lattice", L, N, case["R2"])
        m = _row_counts("lattice", L, N, case["R"] + case["R2"])
        return {"bytes": 12 * (a.sum() + b.sum() + m.sum()), "flops": 2.0 * float((a * b).sum())}
    if kind == "update":
        a, b = _row_counts("lattice", L, N, case["R"]), _row_counts("lattice", L, N, case["R2"])
        return {"bytes": 12 * (4 * a.sum() + b.sum() + 2 * b.sum()), "flops": 3.0 * float(b.sum())}
    if kind == "sp2":
        # the widths of the iterates: radii on the lattice, half-bandwidths on the chain
        grow = [3.0, 5.3, 5.7, 6.3, 6.9] if shape == "lattice" else [16, 32, 60, 100, 140] + [170] * 40
        n = [_row_counts(shape, L, N, r) for r in grow[: case["iters"] + 1]]
        return {"bytes": 12 * float(sum(a.sum() + b.sum() for a, b in zip(n, n[1:]))),
                "flops": float(sum((a * a).sum() for a in n[:-1]))}
    if kind == "adjoint":
        n = [_row_counts("lattice", L, N, r) for r in [3.0, 5.3, 5.7, 6.3, 6.9][: case["iters"] + 1]]
        return {"bytes": 12 * 4 * float(sum(a.sum() for a in n)),
                "flops": 5.0 * float(sum((a * a).sum() for a in n[:-1]))}
    nb = L ** 3
    n = _row_counts("lattice", L, nb, case["R"])
    if kind in ("eb_x2", "eb_tc"):
        m = _row_counts("lattice", L, nb, 2 * case["R"])
        return {"bytes": 8192.0 * float(n.sum() + m.sum()), "flops": 65536.0 * float((n * n).sum())}
    # the radii of the thresholded iterates, wider after 2X - X^2 than after X^2
    n = [_row_counts("lattice", L, nb, g * case["R"]) for g in (1.0, 1.5, 1.1, 1.8, 1.25, 2.0)[: case["iters"] + 1]]
    return {"bytes": 8192.0 * float(sum(a.sum() + b.sum() for a, b in zip(n, n[1:]))),
            "flops": 65536.0 * float(sum((a * a).sum() for a in n[:-1]))}


def tolerance(case):
    """About four times what two runs of the path, or the path and exact(), were seen to differ by."""
    kind = case["kind"]
    if kind == "x2" and case["prec"] == "f32":
        return {"rel": 5e-7}
    if kind == "eb_tc":
        return {"rel": 2e-5 if case["split"] == 0 else 4e-9}
    if kind == "eb_sp2":
        return {"rel": 1.5e-7}
    if kind in ("sp2", "adjoint"):
        return {"rel": 1e-13}
    return {"rel": 1e-14}
