"""The work that users of maxwell_gb300 have it do, as measurable cases.

A case is a call (or the short sequence of calls) that a program makes
through the C ABI of ``include/maxwell_gb300.h``:

* ``bands``          a whole band calculation, ``mxg_bloch_solve``;
* ``precondition``   the preconditioner of a block step: edge V-cycles on a defect;
* ``lift``           the gradient lifting of a block: M, G^H, node V-cycles, G;
* ``smooth``         the four-colour patch smoother, forward and backward;
* ``defect``         the eigenproblem's defect with one shift per vector;
* ``gram``           the Ritz products of a block;
* ``combine``        the Ritz combination of a block;
* ``orthonormalize`` the M-orthonormal basis of a block;
* ``pinvit``         one PINVIT step of the reference's driver flow;
* ``sensitivity``    the permittivity gradient (the adjoint) from host eigenvectors.

Sizes: ``n`` cells per side (``n0 << L`` where a grid hierarchy is needed), ``K``
k-points in a batch, ``m`` vectors per k-point.  ``prec`` is the storage of the
vectors: c64, c128 or cdd (float-float).
"""
import ctypes
import math
import random

import numpy as np
import torch

import maxwell_gb300 as mx

PREC = {"c64": mx.C64, "c128": mx.C128, "cdd": mx.CDD}
BYTES = {"c64": 8, "c128": 16, "cdd": 16}
DEV = "cuda"


# ----------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------
def listed():
    return [
        # a band diagram on a coarse mesh, as a parameter scan runs it by the
        # hundred: launches and the small dense problems count
        {"name": "bands_32", "kind": "bands", "n0": 8, "L": 2, "K": 8, "ieigs": 10, "m": 12, "precision": 1},
        # the benchmark's workload (512^2 cells, 12 pairs, block 16) with
        # eight k-points of the path in the batch
        {"name": "bands_512", "kind": "bands", "n0": 8, "L": 6, "K": 8, "ieigs": 12, "m": 16, "precision": 1},
        # the plain FP64 solver at the size of the reference's own runs
        {"name": "bands_fp64_64", "kind": "bands", "n0": 8, "L": 3, "K": 4, "ieigs": 10, "m": 12, "precision": 0},
        # the reference's preconditioner (row-order smoother, FP64) for a batch
        {"name": "precondition_128", "kind": "precondition", "n0": 8, "L": 4, "K": 8, "m": 12, "prec": "c128"},
        # the lifting of a search block on the benchmark's mesh
        {"name": "lift_512", "kind": "lift", "n0": 8, "L": 6, "K": 8, "m": 16, "prec": "c64"},
        # the solver's own smoother on the benchmark's mesh
        {"name": "smooth_512", "kind": "smooth", "n": 512, "K": 16, "m": 16, "prec": "c64"},
        # the defect of a float-float eigenvector block
        {"name": "defect_512", "kind": "defect", "n": 512, "K": 8, "m": 16, "prec": "cdd"},
        # Ritz products and combination of a float-float eigenvector block
        {"name": "gram_512", "kind": "gram", "n": 512, "K": 8, "m": 16, "prec": "cdd"},
        {"name": "combine_512", "kind": "combine", "n": 512, "K": 8, "m": 16, "prec": "cdd"},
        # an FP64 block of an odd number of vectors on a mesh that is no power of two
        {"name": "orthonormalize_120", "kind": "orthonormalize", "n": 120, "K": 5, "m": 11, "prec": "c128"},
        # the reference's single-vector step: one k-point, one vector, FP64
        {"name": "pinvit_64", "kind": "pinvit", "n0": 8, "L": 3, "K": 1, "m": 1, "prec": "c128"},
        # a band-gap gradient: nine bands at 24 k-points of a 128^2 mesh
        {"name": "sensitivity_128", "kind": "sensitivity", "n": 128, "K": 24, "m": 9},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _hierarchy(rng, lo, hi):
    """(n0, L) with n0 << L between lo and hi."""
    return rng.choice([(n0, L) for n0 in (6, 8, 10) for L in range(1, 7) if lo <= n0 << L <= hi])


def draw(rng):
    kind = rng.choice(["bands", "precondition", "lift", "smooth", "defect", "gram", "combine", "orthonormalize",
                       "pinvit", "sensitivity"])
    c = {"kind": kind}
    if kind == "bands":
        c["precision"] = rng.choice([1, 1, 1, 0])
        c["n0"], c["L"] = _hierarchy(rng, 24, 256 if c["precision"] else 64)
        c["m"] = rng.choice([8, 9, 12, 14, 16])
        c["ieigs"] = (3 * c["m"]) // 4
        n = c["n0"] << c["L"]
        c["K"] = _log(rng, 1, max(1, min(24, (8 << 18) // n ** 2 if c["precision"] else (4 << 12) // n ** 2)))
        return c
    if kind == "sensitivity":
        c["n"], c["m"] = 2 * _log(rng, 8, 80), rng.randint(1, 16)
        c["K"] = _log(rng, 1, max(1, min(32, 24 * 9 * 128 ** 2 // (c["n"] ** 2 * c["m"]))))
        return c
    # the largest listed block of the kind bounds n * n * K * m
    if kind in ("precondition", "lift", "pinvit"):
        # c64 V-cycles for A + M leave rounding of size 1e-7 n^2 in the gradients
        # (the lifting removes it): outside the solver these calls are FP64
        c["prec"] = rng.choice(["c64", "c64", "c64", "c128"]) if kind == "lift" else "c128"
        c["n0"], c["L"] = _hierarchy(rng, 12, {"precondition": 256, "lift": 512, "pinvit": 96}[kind])
        n, most = c["n0"] << c["L"], {"precondition": 1500000, "lift": 32 << 20, "pinvit": 1 << 16}[kind]
        if kind == "lift" and c["prec"] == "c128":
            most //= 16
    else:
        c["n"] = 2 * _log(rng, 8, 60 if kind == "orthonormalize" else 256)
        n, most = c["n"], {"smooth": 64 << 20, "defect": 32 << 20, "gram": 32 << 20, "combine": 32 << 20,
                           "orthonormalize": 800000}[kind]
        c["prec"] = rng.choice({"smooth": ["c64", "c64", "c64", "c128"], "defect": ["cdd", "cdd", "c64", "c128"],
                                "gram": ["cdd", "cdd", "c128"], "combine": ["cdd", "c64", "c128"],
                                "orthonormalize": ["c128", "cdd"]}[kind])
        if c["prec"] == "c128" and kind != "orthonormalize":
            most //= 16
    c["m"] = rng.randint(1, 16)
    while c["m"] > 1 and n * n * c["m"] > most:
        c["m"] -= 1
    c["K"] = _log(rng, 1, max(1, min(32, most // (n * n * c["m"]))))
    return c


def _n(c):
    return c["n"] if "n" in c else c["n0"] << c["L"]


# ----------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------
def _kappa(n, seed):
    """1/eps of a disc of seeded radius and permittivity, by the rule of
    setpattern_grid2d (a cell is inside when its lower left corner is)."""
    r = random.Random(seed)
    radius, eps = r.uniform(0.25, 0.35), r.uniform(8.9, 12.0)
    i = np.arange(n) / n
    X, Y = np.meshgrid(i, i)
    return np.ascontiguousarray(np.where((X - 0.5) ** 2 + (Y - 0.5) ** 2 <= radius ** 2, 1.0 / eps, 1.0).reshape(-1))


def _path(K):
    """K k-points evenly spaced in arc length on Gamma-X-M-Gamma."""
    pi, out = math.pi, []
    total = pi * (2.0 + math.sqrt(2.0))
    for q in range(K):
        t = total * q / max(1, K - 1)
        if t <= pi:
            out.append((t, 0.0))
        elif t <= 2 * pi:
            out.append((pi, t - pi))
        else:
            s = max(0.0, pi - (t - 2 * pi) / math.sqrt(2.0))
            out.append((s, s) if s > 1e-9 else (0.0, 0.0))
    return out


def _factors(case, seed):
    """(K, 2) complex factors e^{i kx}, e^{i ky}: the path for a band
    calculation, seeded points of the zone (away from Gamma) for the blocks."""
    if case["kind"] == "bands":
        k = np.array(_path(case["K"]))
    else:
        r = random.Random(seed + 1)
        k = np.array([[r.choice((-1, 1)) * r.uniform(0.3, math.pi) for _ in range(2)] for _ in range(case["K"])])
    return np.exp(1j * k)


def _normal(case, seed, planes=2):
    """A block of complex normal values, [K, planes, n, n, m] complex128 on
    the GPU; rounded to the storage's precision."""
    n = _n(case)
    g = torch.Generator(device=DEV).manual_seed(seed)
    z = torch.randn((case["K"], planes, n, n, case["m"], 2), generator=g, device=DEV, dtype=torch.float64)
    if case.get("prec") == "c64":
        z = z.float().double()
    elif case.get("prec") == "cdd":
        hi = z.float().double()
        z = hi + (z - hi).float().double()
    return torch.view_as_complex(z)


def _shifts(case, seed):
    r = random.Random(seed + 2)
    return np.array([[1.0 - r.uniform(1.0, 60.0) for _ in range(case["m"])] for _ in range(case["K"])])


def _coefficients(case, seed):
    """(K, m, m) complex: well conditioned, coef[k][i, j] of u_i in output j."""
    g = np.random.default_rng(seed + 3)
    m = case["m"]
    return (g.standard_normal((case["K"], m, m)) + 1j * g.standard_normal((case["K"], m, m))) / math.sqrt(2.0 * m)


class _View:
    """A device buffer of the library presented to torch without a copy; it
    keeps the block that owns the buffer alive."""

    def __init__(self, block, ptr, shape, kind):
        self.block = block
        self.__cuda_array_interface__ = {"shape": shape, "typestr": kind, "data": (ptr, False), "version": 2}


def _view(edge):
    """The storage [K][2][n][n][m][components] of an edge block."""
    f = mx.lib().mxg__edge_data
    f.restype, f.argtypes = ctypes.c_void_p, [ctypes.c_void_p]
    g = edge.g
    parts, kind = {mx.C64: (2, "<f4"), mx.C128: (2, "<f8"), mx.CDD: (4, "<f4")}[edge.prec]
    out = torch.as_tensor(_View(edge, f(edge.h), (g.K, 2, g.n, g.n, edge.m, parts), kind), device=DEV)
    out.block = edge   # the buffer must not go before the tensor
    return out


def _fill(edge, z):
    """Writes complex128 values into an edge block."""
    v, r = _view(edge), torch.view_as_real(z)
    if edge.prec == mx.CDD:
        hi = r.float()
        v.copy_(torch.stack([hi, (r - hi.double()).float()], -1).flatten(-2))
    else:
        v.copy_(r)


def _grids(case, seed):
    """The grid hierarchy, coarsest first, with the seeded permittivity and k-points."""
    n, L = _n(case), case.get("L", 0)
    grids = [mx.Grid(n, case["K"], _kappa(n, seed), _factors(case, seed))]
    for _ in range(L):
        grids.append(grids[-1].coarsen())
    return grids[::-1]


def _handles(objs):
    return (ctypes.c_void_p * len(objs))(*[o.h for o in objs])


def _inverse(grid, node):
    """The factored coarse matrix of A + M (or of the nodal Laplace)."""
    n, K = grid.n, grid.K
    a, info = mx.Matrix((1 if node else 2) * n * n, K), np.zeros(K, np.int32)
    if node:
        mx.check(mx.lib().densematrix_node2d_gpu(1, grid.h, a.h))
    else:
        mx.check(mx.lib().densematrix_edge2d_gpu(mx.fz(1.0), mx.fz(1.0), grid.h, a.h))
    mx.check(mx.lib().potrf_matrix_gpu(a.h, mx._ptr(info)))
    return a


class _Edges:
    """b, x, d work vectors of every level."""

    def __init__(self, grids, m, prec):
        self.b, self.x, self.d = ([mx.Edge(g, m, prec) for g in grids] for _ in range(3))
        self.hb, self.hx, self.hd = _handles(self.b), _handles(self.x), _handles(self.d)


class _Nodes:
    def __init__(self, grids, m, prec):
        self.b, self.x, self.d = ([mx.Node(g, m, prec) for g in grids] for _ in range(3))
        self.hb, self.hx, self.hd = _handles(self.b), _handles(self.x), _handles(self.d)


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    if kind == "bands":
        s["factors"] = _factors(case, seed)
        s["solver"] = mx.Solver(_kappa(_n(case), seed), n0=case["n0"], L=case["L"], ieigs=case["ieigs"], m=case["m"],
                                method=1, precision=case["precision"], max_nested=20, nested_tol=1e-2, max_steps=60,
                                wave=case["K"], relative=1, tol=1e-8)
        return s
    if kind == "sensitivity":
        s["kappa"], s["factors"] = _kappa(case["n"], seed), _factors(case, seed)
        z = _normal(case, seed).permute(0, 4, 1, 2, 3).reshape(case["K"], case["m"], -1)
        s["vectors"] = np.ascontiguousarray(z.cpu().numpy())
        s["weights"] = np.random.default_rng(seed + 4).standard_normal((case["K"], case["m"]))
        return s
    grids = s["grids"] = _grids(case, seed)
    fine, m, prec = grids[-1], case["m"], PREC[case["prec"]]
    if kind == "precondition":
        s["edges"], s["Ae"] = _Edges(grids, m, prec), _inverse(grids[0], False)
        _fill(s["edges"].b[-1], _normal(case, seed))
        s["out"] = _view(s["edges"].x[-1])
    elif kind in ("lift", "pinvit"):
        s["source"], s["e"], s["nodes"] = mx.Edge(fine, m, prec), mx.Edge(fine, m, prec), _Nodes(grids, m, prec)
        s["An"] = _inverse(grids[0], True)
        _fill(s["source"], _normal(case, seed))
        if kind == "pinvit":
            s["edges"], s["Ae"] = _Edges(grids, m, prec), _inverse(grids[0], False)
            s["lambda"] = np.ascontiguousarray(1.0 - _shifts(case, seed))
        else:
            s["d"] = mx.Edge(fine, m, prec)
        s["out"] = _view(s["e"])
    elif kind == "smooth":
        s["b"], s["x"] = mx.Edge(fine, m, prec), mx.Edge(fine, m, prec)
        _fill(s["b"], _normal(case, seed))
        s["out"] = _view(s["x"])
    elif kind == "defect":
        s["e"], s["r"] = mx.Edge(fine, m, prec), mx.Edge(fine, m, mx.C128 if prec == mx.C128 else mx.C64)
        _fill(s["e"], _normal(case, seed))
        s["shifts"] = _shifts(case, seed)
        s["out"] = _view(s["r"])
    elif kind == "gram":
        s["x"] = mx.Edge(fine, m, prec)
        _fill(s["x"], _normal(case, seed))
    elif kind == "combine":
        s["x"], s["y"] = mx.Edge(fine, m, prec), mx.Edge(fine, m, prec)
        _fill(s["x"], _normal(case, seed))
        s["coef"] = np.ascontiguousarray(_coefficients(case, seed).transpose(0, 2, 1))   # column-major per k
        s["out"] = _view(s["y"])
    else:
        s["source"], s["x"] = mx.Edge(fine, m, prec), mx.Edge(fine, m, prec)
        _fill(s["source"], _normal(case, seed))
        s["info"] = np.zeros(case["K"], np.int32)
    return s


def run(s):
    case, lib, one = s["case"], mx.lib(), mx.fz(1.0)
    kind = case["kind"]
    if kind == "bands":
        # the eigenvalues of the wanted pairs: the block's remaining columns
        # are guard vectors that the stopping rule leaves where they are
        lam, _, _ = s["solver"].solve(s["factors"])
        return lam[:, :case["ieigs"]]
    if kind == "precondition":
        w, L = s["edges"], case["L"]
        mx.check(lib.zero_edge2d_gpu(w.x[-1].h))
        for _ in range(2):
            mx.check(lib.vcycle_edge2d_gpu(L, 2, s["Ae"].h, w.hb, w.hx, w.hd))
        return s["out"]
    if kind == "lift":
        w, L = s["nodes"], case["L"]
        mx.check(lib.copy_edge2d_gpu(s["source"].h, s["e"].h))
        mx.check(lib.zero_edge2d_gpu(s["d"].h))
        mx.check(lib.addeval_edge2d_gpu(mx.fz(0.0), one, s["e"].h, s["d"].h))
        mx.check(lib.zero_node2d_gpu(w.b[-1].h))
        mx.check(lib.adjgradient_node2d_gpu(one, s["d"].h, w.b[-1].h))
        mx.check(lib.zero_node2d_gpu(w.x[-1].h))
        for _ in range(5):
            mx.check(lib.vcycle_node2d_gpu(L, 2, s["An"].h, w.hb, w.hx, w.hd))
        mx.check(lib.gradient_node2d_gpu(mx.fz(-1.0), w.x[-1].h, s["e"].h))
        return s["out"]
    if kind == "pinvit":
        w, v = s["edges"], s["nodes"]
        mx.check(lib.copy_edge2d_gpu(s["source"].h, s["e"].h))
        mx.check(lib.pinvit_edge2d_gpu(case["L"], 2, 2, 5, mx._ptr(s["lambda"]), s["e"].h, s["Ae"].h, w.hb, w.hx, w.hd,
                                       s["An"].h, v.hb, v.hx, v.hd))
        return s["out"]
    if kind == "smooth":
        mx.check(lib.zero_edge2d_gpu(s["x"].h))
        mx.check(lib.gscolour_edge2d_gpu(one, one, s["b"].h, s["x"].h, 2))
        return s["out"]
    if kind == "defect":
        mx.check(lib.zero_edge2d_gpu(s["r"].h))
        mx.check(lib.addeval_shifted_edge2d_gpu(1.0, mx._ptr(s["shifts"]), s["e"].h, s["r"].h))
        return s["out"]
    if kind == "gram":
        a, g = (np.empty((case["K"], case["m"], case["m"]), np.complex128) for _ in range(2))
        mx.check(lib.gram_edge2d_gpu(s["x"].h, mx._ptr(a), mx._ptr(g)))
        return a, g
    if kind == "combine":
        mx.check(lib.lincomb_edge2d_gpu(mx._ptr(s["coef"]), s["x"].h, s["y"].h))
        return s["out"]
    if kind == "orthonormalize":
        mx.check(lib.copy_edge2d_gpu(s["source"].h, s["x"].h))
        mx.check(lib.orthonormalize_edge2d_gpu(s["x"].h, mx._ptr(s["info"])))
        return _view(s["x"])   # its storage may have changed hands
    return mx.eps_sensitivity(case["n"], s["kappa"], s["factors"], s["vectors"], s["weights"])


# ----------------------------------------------------------------------
# the work of one pass: blocks read and written once, arithmetic of the method
# ----------------------------------------------------------------------
def work(case):
    n, K, m, kind = _n(case), case["K"], case["m"], case["kind"]
    e = 2.0 * n * n * K * m                     # entries of an edge block
    if kind == "bands":
        # per finest-level step the eigenvectors, the preconditioned defect
        # and the search directions are read and the new ones written; about
        # 12 steps, and two V-cycles, two liftings of five V-cycles, a Gram
        # matrix of three blocks and the combinations each
        big, low = (16, 8) if case["precision"] else (16, 16)
        flops = e * (2 * 4 * 60 * 1.33 + 2 * 5 * 2 * 30 * 1.33 + 3 * 3 * m * 8 + 2 * 3 * m * 8)
        return {"bytes": 12 * e * (2 * big + 4 * low), "flops": 12 * flops}
    if kind == "sensitivity":
        return {"bytes": 16 * e + 16.0 * n * n, "flops": 6 * e}
    b = BYTES[case["prec"]]
    if kind == "precondition":
        return {"bytes": 2 * b * e, "flops": e * 2 * (4 * 60 + 40) * 1.33}
    if kind == "lift":
        return {"bytes": 2 * b * e, "flops": e * (5 * (4 * 15 + 20) * 1.33 + 30)}
    if kind == "pinvit":
        return {"bytes": 2 * b * e, "flops": e * (2 * (4 * 60 + 40) * 1.33 + 5 * (4 * 15 + 20) * 1.33 + 60)}
    if kind == "smooth":
        return {"bytes": 2 * b * e, "flops": e * 2 * 120}
    if kind == "defect":
        return {"bytes": (b + (16 if b == 16 and case["prec"] == "c128" else 8)) * e, "flops": e * 40}
    if kind == "gram":
        return {"bytes": b * e, "flops": e * (m + 1) / 2 * 8 * 1.5}
    if kind == "combine":
        return {"bytes": 2 * b * e, "flops": e * m * 8}
    return {"bytes": 2 * b * e, "flops": e * ((m + 1) / 2 * 8 + m * 8)}


# ----------------------------------------------------------------------
# the same in 64 bits with torch alone.  Edge fields are pairs (x, y) of
# [K, j, i, m] complex128 tensors, node fields one such tensor.
# ----------------------------------------------------------------------
class _Cell:
    """One level: n, Bloch factors and 1/eps."""

    def __init__(self, n, f, kap):
        self.n, self.kap = n, kap
        self.xf = torch.as_tensor(f[:, 0], device=DEV)
        self.yf = torch.as_tensor(f[:, 1], device=DEV)

    def coarser(self):
        k = self.kap.reshape(self.n // 2, 2, self.n // 2, 2).mean((1, 3))
        return _Cell(self.n // 2, torch.stack([self.xf, self.yf], 1), k)

    def at(self, u, di, dj):
        """u at (i + di, j + dj), di and dj in -1, 0, 1, across the seams."""
        if di:
            u = torch.roll(u, -di, 2)
            u[:, :, -1 if di > 0 else 0] *= (self.xf if di > 0 else self.xf.conj())[:, None, None]
        if dj:
            u = torch.roll(u, -dj, 1)
            u[:, -1 if dj > 0 else 0] *= (self.yf if dj > 0 else self.yf.conj())[:, None, None]
        return u


def _levels(case, seed):
    """All levels, coarsest first."""
    n = _n(case)
    out = [_Cell(n, _factors(case, seed), torch.as_tensor(_kappa(n, seed).reshape(n, n), device=DEV))]
    for _ in range(case.get("L", 0)):
        out.append(out[-1].coarser())
    return out[::-1]


def _curl(c, x, y):
    return x - c.at(x, 0, 1) - y + c.at(y, 1, 0)


def _apply(c, alpha, beta, x, y):
    """(alpha A + beta M) (x, y); beta a number or broadcastable."""
    ox = beta / 6.0 * (4.0 * x + c.at(x, 0, 1) + c.at(x, 0, -1))
    oy = beta / 6.0 * (4.0 * y + c.at(y, 1, 0) + c.at(y, -1, 0))
    if alpha:
        w = alpha * c.n ** 2 * c.kap[None, :, :, None] * _curl(c, x, y)
        ox += w - c.at(w, 0, -1)
        oy += c.at(w, -1, 0) - w
    return ox, oy


def _patch(k, r0, r1, r2, r3, n):
    """The corrections of the vertex patches' edges x(i-1,j), x(i,j), y(i,j-1),
    y(i,j) from their residuals; k = kappa of the cells LL, UL, LR, UR."""
    ll, ul, lr, ur = (float(n) * n * q for q in k)
    s = 8.0 / 6.0
    d0, d1 = ul + lr + s, ll + ur
    l20, l21 = (ul - lr) / d0, (ll - ur) / d1
    d2 = ll + ul + lr + ur + s - l21 * l21 * d1
    c0, c1, c2, c3 = r0 + r1 + r2 + r3, r0 + r1 - r2 - r3, r0 - r1 - r2 + r3, r0 - r1 + r2 - r3
    c2 = (c2 - l20 * c0 - l21 * c1) / d2
    c0, c1, c3 = c0 / d0 - l20 * c2, c1 / d1 - l21 * c2, c3 / s
    return ((c0 + c1 + c2 + c3) / 4, (c0 + c1 - c2 - c3) / 4, (c0 - c1 - c2 + c3) / 4, (c0 - c1 + c2 - c3) / 4)


def _kappas(c):
    """kappa of the four cells around each vertex, [1, j, i, 1]."""
    k = c.kap
    return [torch.roll(k, s, (0, 1))[None, :, :, None] for s in ((1, 1), (0, 1), (1, 0), (0, 0))]


def _smooth_colours(c, b, x, back):
    """Vertex patches in four colours, one after the other."""
    x, y = x
    kap = _kappas(c)
    i = torch.arange(c.n, device=DEV)
    for ci, cj in ((0, 0), (1, 0), (0, 1), (1, 1))[:: -1 if back else 1]:
        ax, ay = _apply(c, 1.0, 1.0, x, y)
        rx, ry = b[0] - ax, b[1] - ay
        del ax, ay
        mask = ((i % 2 == cj)[:, None] & (i % 2 == ci)[None, :])[None, :, :, None]
        d = [q * mask for q in _patch(kap, c.at(rx, -1, 0), rx, c.at(ry, 0, -1), ry, c.n)]
        x = x + c.at(d[0], 1, 0) + d[1]
        y = y + c.at(d[2], 0, 1) + d[3]
    return x, y


def _smooth_rows(c, b, x, back):
    """Vertex patches along the rows, the even rows at once, then the odd
    ones (backward the reverse); updates x in place."""
    n, (x, y), (bx, by) = c.n, x, b
    mm, axy = 1.0 / 6.0, float(n) * n
    yf = c.yf[:, None]

    def col(u, i):   # column i of u, one period outside included: [K, j, m]
        v = u[:, :, i % n]
        return v * c.xf[:, None, None] if i >= n else v * c.xf.conj()[:, None, None] if i < 0 else v

    for par in ((1, 0) if back else (0, 1)):
        jc = torch.arange(par, n, 2, device=DEV)

        def row(v, dj):   # the rows jc + dj of a column
            r = v[:, (jc + dj) % n]
            if dj < 0 and par == 0:
                r = torch.cat([r[:, :1] * yf.conj()[..., None], r[:, 1:]], 1)
            if dj > 0 and par == 1:
                r = torch.cat([r[:, :-1], r[:, -1:] * yf[..., None]], 1)
            return r

        for i in (range(n - 1, -1, -1) if back else range(n)):
            xa, xb, ya, yb, yc = col(x, i - 1), col(x, i), col(y, i - 1), col(y, i), col(y, i + 1)
            xa0, xa1, xa2 = (row(xa, q) for q in (-1, 0, 1))
            xb0, xb1, xb2 = (row(xb, q) for q in (-1, 0, 1))
            ya0, ya1, yb0, yb1, yc0, yc1 = (row(u, q) for u in (ya, yb, yc) for q in (-1, 0))
            k = [c.kap[(jc + q) % n, (i + p) % n][None, :, None] for p, q in ((-1, -1), (-1, 0), (0, -1), (0, 0))]
            ll, ul = k[0] * (xa0 - xa1 - ya0 + yb0), k[1] * (xa1 - xa2 - ya1 + yb1)
            lr, ur = k[2] * (xb0 - xb1 - yb0 + yc0), k[3] * (xb1 - xb2 - yb1 + yc1)
            r0 = row(col(bx, i - 1), 0) - axy * (ul - ll) - mm * (4 * xa1 + xa2 + xa0)
            r1 = row(col(bx, i), 0) - axy * (ur - lr) - mm * (4 * xb1 + xb2 + xb0)
            r2 = row(col(by, i), -1) - axy * (ll - lr) - mm * (4 * yb0 + yc0 + ya0)
            r3 = row(col(by, i), 0) - axy * (ul - ur) - mm * (4 * yb1 + yc1 + ya1)
            d0, d1, d2, d3 = _patch(k, r0, r1, r2, r3, n)
            if i == 0:
                d0 = d0 * c.xf[:, None, None]
            x[:, jc, (i - 1) % n] += d0
            x[:, jc, i] += d1
            y[:, jc, i] += d3
            if par == 0:
                d2 = torch.cat([d2[:, :1] * yf[..., None], d2[:, 1:]], 1)
            y[:, (jc - 1) % n, i] += d2
    return x, y


def _restrict(c, u):
    """Edge restriction from level c."""
    x, y = u
    x = 0.25 * (c.at(x, 0, -1) + c.at(x, 0, 1)) + 0.5 * x
    y = 0.25 * (c.at(y, -1, 0) + c.at(y, 1, 0)) + 0.5 * y
    return x[:, ::2, ::2] + x[:, ::2, 1::2], y[:, ::2, ::2] + y[:, 1::2, ::2]


def _prolong(c, u):
    """Edge prolongation from level c to the next finer one."""
    x, y = u
    fx = torch.stack([0.5 * x, 0.25 * (x + c.at(x, 0, 1))], 2).flatten(1, 2)
    fy = torch.stack([0.5 * y, 0.25 * (y + c.at(y, 1, 0))], 3).flatten(2, 3)
    return fx.repeat_interleave(2, 2), fy.repeat_interleave(2, 1)


def _dense_solve(c, op, b):
    """op^-1 b on the coarsest level, the matrix from op on the unit vectors."""
    N = b.shape[1]
    unit = torch.eye(N, dtype=torch.complex128, device=DEV).expand(b.shape[0], N, N)
    return torch.linalg.solve(op(unit), b)


def _vcycle_edge(levels, b, x, nu=2):
    c = levels[-1]
    if len(levels) == 1:
        def op(v):
            u = v.reshape(v.shape[0], 2, c.n, c.n, -1)
            return torch.stack(_apply(c, 1.0, 1.0, u[:, 0], u[:, 1]), 1).reshape(v.shape)
        z = torch.stack(b, 1)
        z = _dense_solve(c, op, z.reshape(z.shape[0], 2 * c.n ** 2, -1)).reshape(z.shape)
        return z[:, 0].clone(), z[:, 1].clone()
    for _ in range(nu):
        x = _smooth_rows(c, b, x, False)
    a = _apply(c, 1.0, 1.0, *x)
    r = _restrict(c, (b[0] - a[0], b[1] - a[1]))
    p = _prolong(levels[-2], _vcycle_edge(levels[:-1], r, tuple(torch.zeros_like(q) for q in r), nu))
    x = (x[0] + p[0], x[1] + p[1])
    for _ in range(nu):
        x = _smooth_rows(c, b, x, True)
    return x


def _laplace(c, u):
    w = c.at(u, -1, 0) + u + c.at(u, 1, 0)
    return 3.0 * u - (w + c.at(w, 0, 1) + c.at(w, 0, -1)) / 3.0


def _smooth_node(c, b, x, back):
    """Point Gauss-Seidel: row 0, the odd rows below n-1, the even rows, row
    n-1, each row from left to right; backward the exact reverse.  Along a
    row x_i = x_{i-1} / 8 + beta_i, summed by doubling the span."""
    n = c.n
    if back:   # the same sweep in the mirrored coordinate
        c = _Cell(n, torch.stack([c.xf.conj(), c.yf], 1), c.kap.flip(1))
        b, x = b.flip(2), x.flip(2)
    x = x.clone()
    rows = [range(0, 1), range(1, n - 1, 2), range(2, n, 2), range(n - 1, n)]
    for g in rows[:: -1 if back else 1]:
        j = torch.as_tensor(list(g), device=DEV)
        old = x[:, j]
        s = torch.zeros_like(old)
        for dj in (-1, 1):
            r = x[:, (j + dj) % n]
            edge = j + dj
            f = torch.where((edge < 0)[None, :], c.yf.conj()[:, None],
                            torch.where((edge >= n)[None, :], c.yf[:, None], torch.ones_like(c.yf)[:, None]))
            r = r * f[:, :, None, None]
            s += c.at(r, -1, 0) + r + c.at(r, 1, 0)
        nxt = c.at(old, 1, 0)
        first = 0.375 * (b[:, j, 0] + (s[:, :, 0] + nxt[:, :, 0]) / 3.0) + c.at(old, -1, 0)[:, :, 0] / 8.0
        nxt[:, :, n - 1] = first * c.xf[:, None, None]
        v = 0.375 * (b[:, j] + (s + nxt) / 3.0)
        v[:, :, 0] = first
        d = 1
        while d < min(n, 32):
            w = v.clone()
            w[:, :, d:] += v[:, :, :-d] / 8.0 ** d
            v, d = w, 2 * d
        x[:, j] = v
    return x.flip(2) if back else x


def _restrict_node(c, u):
    w = u + 0.5 * (c.at(u, -1, 0) + c.at(u, 1, 0))
    return (w + 0.5 * (c.at(w, 0, -1) + c.at(w, 0, 1)))[:, ::2, ::2]


def _prolong_node(c, u):
    w = torch.stack([u, 0.5 * (u + c.at(u, 1, 0))], 3).flatten(2, 3)
    up = c.at(u, 0, 1)
    up = torch.stack([up, 0.5 * (up + c.at(up, 1, 0))], 3).flatten(2, 3)
    return torch.stack([w, 0.5 * (w + up)], 2).flatten(1, 2)


def _vcycle_node(levels, b, x, nu=2):
    c = levels[-1]
    if len(levels) == 1:
        def op(v):
            return _laplace(c, v.reshape(v.shape[0], c.n, c.n, -1)).reshape(v.shape)
        return _dense_solve(c, op, b.reshape(b.shape[0], c.n ** 2, -1)).reshape(b.shape)
    for _ in range(nu):
        x = _smooth_node(c, b, x, False)
    r = _restrict_node(c, b - _laplace(c, x))
    x = x + _prolong_node(levels[-2], _vcycle_node(levels[:-1], r, torch.zeros_like(r), nu))
    for _ in range(nu):
        x = _smooth_node(c, b, x, True)
    return x


def _lift(levels, e):
    c = levels[-1]
    mx_, my = _apply(c, 0.0, 1.0, *e)
    rhs = c.at(mx_, -1, 0) - mx_ + c.at(my, 0, -1) - my
    v = torch.zeros_like(rhs)
    for _ in range(5):
        v = _vcycle_node(levels, rhs, v)
    return e[0] - (c.at(v, 1, 0) - v), e[1] - (c.at(v, 0, 1) - v)


def _grams(c, z):
    """z^H (A+M) z and z^H M z per k-point, element (i, j) at [i, j]."""
    x, y = z[:, 0], z[:, 1]
    kx, ky = _apply(c, 1.0, 1.0, x, y)
    gx, gy = _apply(c, 0.0, 1.0, x, y)
    K, m = x.shape[0], x.shape[-1]

    def prod(u, v):
        return u.reshape(K, -1, m).conj().transpose(1, 2) @ v.reshape(K, -1, m)

    return prod(x, kx) + prod(y, ky), prod(x, gx) + prod(y, gy)


def _eigenvalues(case, seed):
    c = _levels(dict(case, L=0, n=_n(case)), seed)[0]
    N, out = 2 * c.n ** 2, []
    unit = torch.eye(N, dtype=torch.complex128, device=DEV).reshape(1, 2, c.n, c.n, N)
    f = torch.stack([c.xf, c.yf], 1)
    for k in range(case["K"]):
        ck = _Cell(c.n, f[k:k + 1], c.kap)
        a, g = (torch.stack(_apply(ck, al, be, unit[:, 0], unit[:, 1]), 1).reshape(N, N) for al, be in ((1.0, 0.0), (0.0, 1.0)))
        low = torch.linalg.cholesky(g)
        a = torch.linalg.solve_triangular(low, a, upper=False)
        a = torch.linalg.solve_triangular(low, a.conj().T, upper=False)
        w = torch.linalg.eigvalsh(0.5 * (a + a.conj().T)).cpu().numpy()
        out.append(w[w > 1e-6][:case["ieigs"]])   # the rest are gradients (and constants at Gamma)
    return np.array(out)


def _stored(z, prec):
    """An edge block as run() returns it."""
    r = torch.view_as_real(z.contiguous())
    if prec != "cdd":
        return r
    hi = r.float().double()
    return torch.stack([hi, r - hi], -1).flatten(-2)


def exact(case, seed):
    kind = case["kind"]
    if kind == "bands":
        # dense matrices of all edges: meshes up to 32 x 32 only
        return _eigenvalues(case, seed) if _n(case) <= 32 else None
    if kind == "sensitivity":
        c, z = _levels(case, seed)[0], _normal(case, seed)
        w = torch.as_tensor(np.random.default_rng(seed + 4).standard_normal((case["K"], case["m"])), device=DEV)
        s = (_curl(c, z[:, 0], z[:, 1]).abs() ** 2 * w[:, None, None, :]).sum((0, 3))
        return (-float(c.n) ** 2 * c.kap ** 2 * s).reshape(-1).cpu().numpy()
    levels, z, prec = _levels(case, seed), _normal(case, seed), case["prec"]
    c, e = levels[-1], (z[:, 0], z[:, 1])
    if kind == "precondition":
        x = (torch.zeros_like(e[0]), torch.zeros_like(e[1]))
        for _ in range(2):
            x = _vcycle_edge(levels, e, x)
    elif kind == "lift":
        x = _lift(levels, e)
    elif kind == "pinvit":
        shift = torch.as_tensor(_shifts(case, seed), device=DEV)[:, None, None, :]
        b = _apply(c, 1.0, shift, *e)
        x = (torch.zeros_like(e[0]), torch.zeros_like(e[1]))
        for _ in range(2):
            x = _vcycle_edge(levels, b, x)
        x = _lift(levels, (e[0] - x[0], e[1] - x[1]))
    elif kind == "smooth":
        x = (torch.zeros_like(e[0]), torch.zeros_like(e[1]))
        for back in (False, True):
            x = _smooth_colours(c, e, x, back)
    elif kind == "defect":
        x = _apply(c, 1.0, torch.as_tensor(_shifts(case, seed), device=DEV)[:, None, None, :], *e)
        prec = "c128"
    elif kind == "gram":
        return tuple(q.transpose(1, 2).cpu().numpy() for q in _grams(c, z))   # column-major per k
    elif kind == "combine":
        z = z.reshape(case["K"], -1, case["m"]) @ torch.as_tensor(_coefficients(case, seed), device=DEV)
        return _stored(z.reshape(case["K"], 2, c.n, c.n, case["m"]), prec)
    else:
        low = torch.linalg.cholesky(_grams(c, z)[1])
        q = torch.linalg.solve_triangular(low.conj().transpose(1, 2), z.reshape(case["K"], -1, case["m"]), upper=True,
                                          left=False)
        return _stored(q.reshape(z.shape), prec)
    return _stored(torch.stack(x, 1), prec)
