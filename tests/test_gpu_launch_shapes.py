"""Kernels whose launch shape depends on the size, at the sizes where the
shape changes, against the oracle.  Tolerances are those of the operators'
own tests (the storage's arithmetic)."""
import numpy as np
import pytest

import maxwell_gb300 as mx

pytestmark = pytest.mark.gpu

TOL = {mx.C128: 1e-12, mx.CDD: 1e-12, mx.C64: 2e-5}
FACTORS = np.array([[np.exp(0.7j), np.exp(-1.3j)], [1.0, 1.0], [np.exp(2.9j), np.exp(0.4j)]])


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def cv(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


@pytest.mark.parametrize("n, m, K", [(250, 16, 3), (446, 15, 2), (18, 32, 1), (64, 1, 1)])
@pytest.mark.parametrize("prec", [mx.C128, mx.CDD, mx.C64])
def test_edge_operator_strips(oracle, n, m, K, prec):
    """The edge operator in strips of 4 and 8 rows that do not divide the
    grid (250, 446) and of one row; 7, 15, 16 and 255 columns per tile."""
    rng = np.random.default_rng(n)
    kap = 1.0 / (1.0 + 11.0 * rng.random(n * n))
    g = mx.Grid(n, K, kap, FACTORS[:K])
    x, y = cv(rng, K, m, 2 * n * n), cv(rng, K, m, 2 * n * n)
    ex, ey = mx.Edge(g, m, prec, x), mx.Edge(g, m, prec, y)
    mx.check(mx.lib().addeval_edge2d_gpu(mx.fz(1.3), mx.fz(0.7), ex.h, ey.h))
    got = ey.get()
    for k in range(K):
        for v in {0, m - 1}:
            assert rel(got[k, v], oracle.addeval_edge(n, kap, *FACTORS[k], 1.3, 0.7, x[k, v], y[k, v])) < TOL[prec]


@pytest.mark.parametrize("n, m, K", [(2, 1, 1), (6, 32, 2), (64, 16, 1), (130, 7, 2), (96, 5, 3)])
@pytest.mark.parametrize("prec", [mx.C128, mx.CDD, mx.C64])
@pytest.mark.parametrize("direction", [0, 1])
def test_row_smoother_chunks(oracle, n, m, K, prec, direction):
    """The patch smoother in row order: chunks of one patch (n = 2), vectors
    split over CTAs (one k-point of 16, groups that do not divide 7 or 5),
    chunks that do not divide the row (130), 32 vectors."""
    rng = np.random.default_rng(n)
    kap = 1.0 / (1.0 + 11.0 * rng.random(n * n))
    g = mx.Grid(n, K, kap, FACTORS[:K])
    b, x = cv(rng, K, m, 2 * n * n), cv(rng, K, m, 2 * n * n)
    eb, ex = mx.Edge(g, m, prec, b), mx.Edge(g, m, prec, x)
    fn = [mx.lib().gsforward_edge2d_gpu, mx.lib().gsbackward_edge2d_gpu][direction]
    mx.check(fn(mx.fz(1.0), mx.fz(0.8), eb.h, ex.h))
    got = ex.get()
    for k in range(K):
        for v in {0, m // 2, m - 1}:
            want = oracle.gs_edge(n, kap, *FACTORS[k], 1.0, 0.8, direction, b[k, v], x[k, v])
            assert rel(got[k, v], want) < (1e-4 if prec == mx.C64 else 1e-11)


@pytest.mark.parametrize("n, m, K", [(2, 3, 1), (6, 16, 2), (8, 1, 1), (10, 24, 1), (74, 7, 2), (130, 32, 1),
                                     (64, 12, 3)])
@pytest.mark.parametrize("prec", [mx.C128, mx.CDD])
@pytest.mark.parametrize("direction", [0, 1])
def test_colour_smoother_parts(oracle, n, m, K, prec, direction):
    """The patch smoother in four colours, rows cut in four: rows too short
    to cut (2, 6), parts of one patch (8), parts that differ by one (10, 74,
    130), parts of one chunk and of several (130 with 8 patch lanes)."""
    rng = np.random.default_rng(n)
    kap = 1.0 / (1.0 + 11.0 * rng.random(n * n))
    g = mx.Grid(n, K, kap, FACTORS[:K])
    b, x = cv(rng, K, m, 2 * n * n), cv(rng, K, m, 2 * n * n)
    eb, ex = mx.Edge(g, m, prec, b), mx.Edge(g, m, prec, x)
    mx.check(mx.lib().gscolour_edge2d_gpu(mx.fz(1.0), mx.fz(0.8), eb.h, ex.h, direction))
    got = ex.get()
    for k in range(K):
        for v in {0, m // 2, m - 1}:
            want = oracle.gs_edge_colour(n, kap, *FACTORS[k], 1.0, 0.8, direction, b[k, v], x[k, v])
            assert rel(got[k, v], want) < 1e-11


@pytest.mark.parametrize("prec", [mx.C128, mx.CDD])
def test_colour_smoother_table_refill(prec):
    """Parts of more patches than their table holds (257 against 255): one
    vector alone and the same vector among four, whose chunks and tables are
    cut at other patches, agree to the bit."""
    rng = np.random.default_rng(29)
    n = 2052
    g = mx.Grid(n, 1, 1.0 / (1.0 + 11.0 * rng.random(n * n)), FACTORS[:1])
    b, x = cv(rng, 1, 1, 2 * n * n), cv(rng, 1, 1, 2 * n * n)
    got = []
    for m in (1, 4):
        eb, ex = [mx.Edge(g, m, prec, np.repeat(a, m, axis=1)) for a in (b, x)]
        mx.check(mx.lib().gscolour_edge2d_gpu(mx.fz(1.0), mx.fz(0.8), eb.h, ex.h, 0))
        got.append(ex.get()[0, m - 1])
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("n0, L, m", [(4, 2, 6), (6, 2, 9), (10, 1, 12), (12, 1, 8)])
@pytest.mark.parametrize("precision", [0, 1])
def test_coarse_grid_sizes(oracle, n0, L, m, precision):
    """Solves that start from coarse grids of 16, 36 (matrices in shared
    memory), 100 and 144 cells (in global memory), Gamma among the k-points."""
    rng = np.random.default_rng(n0)
    n = n0 << L
    kap = 1.0 / (1.0 + 11.0 * rng.random(n * n))
    fac, ie = FACTORS, (2 * m) // 3
    s = mx.Solver(kap, n0=n0, L=L, ieigs=ie, m=m, method=1, precision=precision, max_nested=40, max_steps=60,
                  wave=len(fac), relative=0, tol=1e-8)
    lam, _, res = s.solve(fac)
    st, lam_o, _, _, _ = oracle.bloch_solve(kap, fac, n0=n0, L=L, ieigs=ie, m=m, method=1, max_nested=40,
                                            max_steps=60, tol=1e-8, relative=0, extrapolation="n", wave=len(fac))
    assert st == 0 and res[:, :ie].max() <= 1e-8
    assert np.abs(lam[:, :ie] - lam_o[:, :ie]).max() / lam_o[:, :ie].max() < 1e-8


@pytest.mark.parametrize("n0, L, m, K", [(4, 1, 1, 1), (8, 3, 3, 2), (10, 2, 2, 1), (6, 4, 1, 2), (8, 4, 2, 1),
                                         (8, 3, 20, 1), (8, 2, 32, 3)])
@pytest.mark.parametrize("prec", [mx.C128, mx.CDD, mx.C64])
def test_node_vcycle_levels(oracle, n0, L, m, K, prec):
    """Node V-cycles from a given start on grids that run in one launch down
    to the coarse solve (8, 64, 40 and 96 nodes a side: one, two and three
    positions per lane, rows shorter than the warp; in FP64 96 and 128 keep
    upper levels of their own; four, two or one CTA for each FP64 vector)
    against the cycle put together from the oracle's sweeps, residual and
    transfers."""
    rng = np.random.default_rng(n0 + L)
    n = n0 << L
    fac = FACTORS[[0, 2, 0]][:K]
    grids = [mx.Grid(n, K, None, fac)]
    for _ in range(L):
        grids.append(grids[-1].coarsen())
    grids = grids[::-1]
    import ctypes as C
    b, x, d = ([mx.Node(g, m, prec) for g in grids] for _ in range(3))
    rhs, start = cv(rng, K, m, n * n), cv(rng, K, m, n * n)
    b[L].put(rhs)
    x[L].put(start)
    rhs, start = b[L].get(), x[L].get()   # as stored
    A, info = mx.Matrix(n0 * n0, K), np.zeros(K, np.int32)
    mx.check(mx.lib().densematrix_node2d_gpu(1, grids[0].h, A.h))
    mx.check(mx.lib().potrf_matrix_gpu(A.h, mx._ptr(info)))
    arr = [(C.c_void_p * (L + 1))(*[o.h for o in objs]) for objs in (b, x, d)]
    mx.check(mx.lib().vcycle_node2d_gpu(L, 2, A.h, *arr))
    got = x[L].get()

    def cycle(l, f, bl, xl):
        nl = n0 << l
        if l == 0:
            return np.linalg.solve(oracle.dense_node(n0, *f, 1), bl)
        for _ in range(2):
            xl = oracle.gs_node(nl, *f, 1.0, 0, bl, xl)
        r = oracle.addeval_node(nl, *f, -1.0, xl, bl)
        c = oracle.restrict_node(nl // 2, *f, 1.0, r, np.zeros(nl * nl // 4, complex))
        xl = oracle.prolong_node(nl // 2, *f, 1.0, cycle(l - 1, f, c, np.zeros_like(c)), xl)
        for _ in range(2):
            xl = oracle.gs_node(nl, *f, 1.0, 1, bl, xl)
        return xl

    # the sweeps' tolerances (2e-5 and 1e-11) over the cycle's coarse solve
    for k in range(K):
        for v in range(m):
            assert rel(got[k, v], cycle(L, fac[k], rhs[k, v], start[k, v])) < (1e-4 if prec == mx.C64 else 1e-10)


@pytest.mark.parametrize("n, K, m", [(2, 1, 1), (30, 40, 3), (126, 5, 32)])
def test_sensitivity_shares(oracle, n, K, m):
    """The permittivity gradient with one, several and all k-points per
    share of the reduction, zero weights among them."""
    rng = np.random.default_rng(n)
    kap = 1.0 / (1.0 + 11.0 * rng.random(n * n))
    fac = np.exp(1j * rng.uniform(-3, 3, (K, 2)))
    vec, w = cv(rng, K, m, 2 * n * n), rng.standard_normal((K, m))
    w[0, 0] = 0.0
    got = mx.eps_sensitivity(n, kap, fac, vec, w)
    want = sum(oracle.eps_sensitivity(n, kap, *fac[k], vec[k], w[k]) for k in range(K))
    assert rel(got, want) < 1e-12


@pytest.mark.parametrize("n, m, K", [(6, 1, 2), (10, 4, 1), (22, 11, 2), (16, 21, 1), (12, 32, 1)])
@pytest.mark.parametrize("prec", [mx.C128, mx.CDD, mx.C64])
def test_gram_and_combination_block_sizes(n, m, K, prec):
    """Ritz products and combinations of one block, whose entries leave the
    products' threads in 16, several or one group(s) and several entries a
    thread, against matrices put together from the dense operator."""
    rng = np.random.default_rng(m)
    kap = 1.0 / (1.0 + 11.0 * rng.random(n * n))
    g = mx.Grid(n, K, kap, FACTORS[:K])
    x = mx.Edge(g, m, prec, cv(rng, K, m, 2 * n * n))
    u = x.get()
    Kd, Md = mx.Matrix(2 * n * n, K), mx.Matrix(2 * n * n, K)
    mx.check(mx.lib().densematrix_edge2d_gpu(mx.fz(1.0), mx.fz(1.0), g.h, Kd.h))
    mx.check(mx.lib().densematrix_edge2d_gpu(mx.fz(0.0), mx.fz(1.0), g.h, Md.h))
    Kd, Md = Kd.get(), Md.get()
    a, b = np.zeros((K, m, m), complex), np.zeros((K, m, m), complex)
    mx.check(mx.lib().gram_edge2d_gpu(x.h, mx._ptr(a), mx._ptr(b)))
    tol = {mx.C128: 1e-13, mx.CDD: 1e-12, mx.C64: 2e-6}[prec]
    for k in range(K):
        assert rel(a[k].T, u[k].conj() @ Kd[k] @ u[k].T) < tol
        assert rel(b[k].T, u[k].conj() @ Md[k] @ u[k].T) < tol
    coef, y = cv(rng, K, m, m), mx.Edge(g, m, prec)
    ct = np.ascontiguousarray(coef.transpose(0, 2, 1))
    mx.check(mx.lib().lincomb_edge2d_gpu(mx._ptr(ct), x.h, y.h))
    got = y.get()
    for k in range(K):
        assert rel(got[k], coef[k].T @ u[k]) < {mx.C128: 1e-14, mx.CDD: 1e-13, mx.C64: 2e-6}[prec] * m


@pytest.mark.parametrize("n0, L, m, K, nu", [(8, 4, 2, 2, 2), (10, 4, 3, 1, 1), (8, 5, 1, 2, 2), (6, 5, 2, 1, 2),
                                             (8, 6, 1, 1, 2), (14, 3, 5, 1, 2)])
def test_node_vcycle_bands(oracle, n0, L, m, K, nu):
    """c64 node V-cycles whose fine levels run in bands of rows (112 to 512
    nodes a side; one and two sweeps each way, bands of 8 rows and more, the
    bands at the seam in both directions, a last segment of a row that is not
    full) against the cycle put together from the oracle's sweeps."""
    rng = np.random.default_rng(n0 + L)
    n = n0 << L
    fac = FACTORS[[0, 2]][:K]
    grids = [mx.Grid(n, K, None, fac)]
    for _ in range(L):
        grids.append(grids[-1].coarsen())
    grids = grids[::-1]
    import ctypes as C
    b, x, d = ([mx.Node(g, m, mx.C64) for g in grids] for _ in range(3))
    b[L].put(cv(rng, K, m, n * n))
    x[L].put(cv(rng, K, m, n * n))
    rhs, start = b[L].get(), x[L].get()
    A, info = mx.Matrix(n0 * n0, K), np.zeros(K, np.int32)
    mx.check(mx.lib().densematrix_node2d_gpu(1, grids[0].h, A.h))
    mx.check(mx.lib().potrf_matrix_gpu(A.h, mx._ptr(info)))
    arr = [(C.c_void_p * (L + 1))(*[o.h for o in objs]) for objs in (b, x, d)]
    mx.check(mx.lib().vcycle_node2d_gpu(L, nu, A.h, *arr))
    got = x[L].get()
    assert np.array_equal(b[L].get(), rhs)

    def cycle(l, f, bl, xl):
        nl = n0 << l
        if l == 0:
            return np.linalg.solve(oracle.dense_node(n0, *f, 1), bl)
        for _ in range(nu):
            xl = oracle.gs_node(nl, *f, 1.0, 0, bl, xl)
        r = oracle.addeval_node(nl, *f, -1.0, xl, bl)
        c = oracle.restrict_node(nl // 2, *f, 1.0, r, np.zeros(nl * nl // 4, complex))
        xl = oracle.prolong_node(nl // 2, *f, 1.0, cycle(l - 1, f, c, np.zeros_like(c)), xl)
        for _ in range(nu):
            xl = oracle.gs_node(nl, *f, 1.0, 1, bl, xl)
        return xl

    for k in range(K):
        for v in {0, m - 1}:
            assert rel(got[k, v], cycle(L, fac[k], rhs[k, v], start[k, v])) < 1e-4


@pytest.mark.parametrize("n", [1, 2, 31, 64, 97, 160, 161])
def test_hermitian_inverse_orders(n):
    """The explicit inverse behind potrf_matrix_gpu: orders below, at and
    above a warp, the largest whose triangle is held in shared memory and the
    first beyond it; and the report of pivots that are not positive.
    Condition numbers of 10 leave n times the rounding unit and a factor."""
    rng = np.random.default_rng(n)
    K = 2
    A, info = mx.Matrix(n, K), np.zeros(K, np.int32)
    q = [np.linalg.qr(cv(rng, n, n))[0] for _ in range(K)]
    a = np.array([(u * np.linspace(1.0, 10.0, n)) @ u.conj().T for u in q])
    a = (a + np.conj(np.transpose(a, (0, 2, 1)))) / 2
    A.put(a)
    mx.check(mx.lib().potrf_matrix_gpu(A.h, mx._ptr(info)))
    assert not info.any()
    assert rel(A.get(), np.linalg.inv(a)) < 100 * n * 2.2e-16
    a[1] -= 20.0 * np.eye(n)
    A.put(a)
    mx.check(mx.lib().potrf_matrix_gpu(A.h, mx._ptr(info)))
    assert info[0] == 0 and info[1] != 0


def node_levels(n0, L, K, m, prec, fac):
    """Grids, b, x, d of a node hierarchy (coarsest first), the factored
    coarse matrix and the handles' arrays."""
    import ctypes as C
    grids = [mx.Grid(n0 << L, K, None, fac)]
    for _ in range(L):
        grids.append(grids[-1].coarsen())
    grids = grids[::-1]
    b, x, d = ([mx.Node(g, m, prec) for g in grids] for _ in range(3))
    A, info = mx.Matrix(n0 * n0, K), np.zeros(K, np.int32)
    mx.check(mx.lib().densematrix_node2d_gpu(1, grids[0].h, A.h))
    mx.check(mx.lib().potrf_matrix_gpu(A.h, mx._ptr(info)))
    return b, x, d, A, [(C.c_void_p * (L + 1))(*[o.h for o in objs]) for objs in (b, x, d)]


def node_cycle(oracle, n0, l, f, b, x, nu=2):
    """A V-cycle of one vector put together from the oracle's sweeps,
    residual and transfers."""
    n = n0 << l
    if l == 0:
        return np.linalg.solve(oracle.dense_node(n0, *f, 1), b)
    for _ in range(nu):
        x = oracle.gs_node(n, *f, 1.0, 0, b, x)
    r = oracle.addeval_node(n, *f, -1.0, x, b)
    c = oracle.restrict_node(n // 2, *f, 1.0, r, np.zeros(n * n // 4, complex))
    x = oracle.prolong_node(n // 2, *f, 1.0, node_cycle(oracle, n0, l - 1, f, c, np.zeros_like(c), nu), x)
    for _ in range(nu):
        x = oracle.gs_node(n, *f, 1.0, 1, b, x)
    return x


@pytest.mark.parametrize("prec, K", [(mx.C64, 65), (mx.C128, 33), (mx.CDD, 15)])
def test_node_vcycle_large_batch(oracle, prec, K):
    """Coarse node levels of batches of more vectors than the one-launch form
    takes, which run level by level."""
    n0, L, m = 4, 2, 32
    n = n0 << L
    rng = np.random.default_rng(K)
    fac = np.exp(1j * rng.uniform(0.3, 3.0, (K, 2)))
    b, x, d, A, arr = node_levels(n0, L, K, m, prec, fac)
    b[L].put(cv(rng, K, m, n * n))
    x[L].put(cv(rng, K, m, n * n))
    rhs, start = b[L].get(), x[L].get()
    mx.check(mx.lib().vcycle_node2d_gpu(L, 2, A.h, *arr))
    got = x[L].get()
    for k, v in [(0, 0), (K // 2, m // 2), (K - 1, m - 1)]:
        want = node_cycle(oracle, n0, L, fac[k], rhs[k, v], start[k, v])
        assert rel(got[k, v], want) < (1e-4 if prec == mx.C64 else 1e-10)


@pytest.mark.parametrize("prec, n0, L, K, m", [(mx.C64, 8, 1, 512, 32), (mx.C128, 8, 1, 512, 32), (mx.CDD, 8, 2, 256, 32)])
def test_node_vcycle_large_batch_costs_its_sweeps(prec, n0, L, K, m):
    """A V-cycle of a large batch takes no longer than the sweeps, residuals,
    transfers and coarse solve it stands for, called one by one (with half as much again
    for the timing; one CTA per vector took 2.3 to 4.5 times as long)."""
    import time
    lib, one = mx.lib(), mx.fz(1.0)
    b, x, d, A, arr = node_levels(n0, L, K, m, prec, np.exp(1j * np.random.default_rng(1).uniform(0.3, 3.0, (K, 2))))
    mx.check(lib.random_node2d_gpu(b[L].h, 3))
    mx.check(lib.zero_node2d_gpu(x[L].h))

    def whole():
        mx.check(lib.vcycle_node2d_gpu(L, 2, A.h, *arr))

    def parts():
        for l in range(L, 0, -1):
            for _ in range(2):
                mx.check(lib.gsforward_node2d_gpu(one, b[l].h, x[l].h))
            mx.check(lib.copy_node2d_gpu(b[l].h, d[l].h))
            mx.check(lib.addeval_node2d_gpu(mx.fz(-1.0), x[l].h, d[l].h))
            mx.check(lib.zero_node2d_gpu(b[l - 1].h))
            mx.check(lib.restriction_node2d_gpu(one, d[l].h, b[l - 1].h))
            mx.check(lib.zero_node2d_gpu(x[l - 1].h))
        mx.check(lib.vcycle_node2d_gpu(0, 2, A.h, *arr))   # the coarse solve
        for l in range(1, L + 1):
            mx.check(lib.prolongation_node2d_gpu(one, x[l - 1].h, x[l].h))
            for _ in range(2):
                mx.check(lib.gsbackward_node2d_gpu(one, b[l].h, x[l].h))

    def seconds(f):
        f()
        times = []
        for _ in range(5):
            t = time.perf_counter()
            f()
            times.append(time.perf_counter() - t)
        return min(times)

    assert seconds(whole) < 1.5 * seconds(parts)


@pytest.mark.parametrize("prec, n, m, K", [(mx.C64, 16, 1, 200), (mx.C64, 64, 2, 150), (mx.C64, 2, 32, 1800),
                                           (mx.C128, 8, 1, 1100), (mx.C128, 64, 2, 20), (mx.C128, 4, 16, 520),
                                           (mx.C128, 130, 1, 21), (mx.C128, 2, 1, 2500), (mx.CDD, 8, 5, 1030),
                                           (mx.CDD, 32, 1, 1100), (mx.CDD, 64, 3, 130)])
@pytest.mark.parametrize("direction", [0, 1])
def test_row_smoother_pairs(oracle, prec, n, m, K, direction):
    """The patch smoother in row order where a CTA takes vectors of several
    k-points (few vectors of many k-points, small grids), groups that the
    batch does not fill, and the smallest grid in a c64 batch that would be
    large enough for a thread per chain."""
    rng = np.random.default_rng(n)
    kap = 1.0 / (1.0 + 11.0 * rng.random(n * n))
    fac = np.exp(1j * rng.uniform(0.3, 3.0, (K, 2)))
    g = mx.Grid(n, K, kap, fac)
    b, x = cv(rng, K, m, 2 * n * n), cv(rng, K, m, 2 * n * n)
    eb, ex = mx.Edge(g, m, prec, b), mx.Edge(g, m, prec, x)
    fn = [mx.lib().gsforward_edge2d_gpu, mx.lib().gsbackward_edge2d_gpu][direction]
    mx.check(fn(mx.fz(1.0), mx.fz(0.8), eb.h, ex.h))
    got = ex.get()
    for k in {0, 1, K // 2, K - 2, K - 1}:
        for v in {0, m - 1}:
            want = oracle.gs_edge(n, kap, *fac[k], 1.0, 0.8, direction, b[k, v], x[k, v])
            assert rel(got[k, v], want) < (1e-4 if prec == mx.C64 else 1e-11)


@pytest.mark.parametrize("beta", [1.0, 0.8])
@pytest.mark.parametrize("direction", [0, 1])
def test_row_smoother_chains(oracle, beta, direction):
    """The c64 patch smoother in row order with a thread per row and vector
    (57344 chains and more), with the scalars that the tabulated factors were
    made for and with others.  Its residuals are differences of curls of size
    n^2 rounded to 2^-24, four to an edge, which the local solve does not
    divide by n^2 again in the direction of the vertex' gradient."""
    n, m, K = 128, 32, 28
    rng = np.random.default_rng(n)
    kap = 1.0 / (1.0 + 11.0 * rng.random(n * n))
    fac = np.exp(1j * rng.uniform(0.3, 3.0, (K, 2)))
    g = mx.Grid(n, K, kap, fac)
    b, x = cv(rng, 1, m, 2 * n * n), cv(rng, 1, m, 2 * n * n)   # the same block at every k-point
    eb, ex = mx.Edge(g, m, mx.C64, b), mx.Edge(g, m, mx.C64, x)
    fn = [mx.lib().gsforward_edge2d_gpu, mx.lib().gsbackward_edge2d_gpu][direction]
    mx.check(fn(mx.fz(1.0), mx.fz(beta), eb.h, ex.h))
    got = ex.get()
    for k, v in {(0, 0), (K // 2, m // 2), (K - 1, m - 1)}:
        want = oracle.gs_edge(n, kap, *fac[k], 1.0, beta, direction, b[0, v], x[0, v])
        assert rel(got[k, v], want) < 4 * n * n * 2.0 ** -24


@pytest.mark.parametrize("prec, n", [(mx.C128, 16), (mx.CDD, 32)])
def test_row_smoother_batch_shape(prec, n):
    """The row-order smoother costs about as much for a vector at each of
    2048 k-points as for 32 at 64 (2.4 to 4.3 times as much where a CTA held
    vectors of one k-point only)."""
    import time
    lib, one, dot = mx.lib(), mx.fz(1.0), np.zeros(2048)
    times = []
    for K, m in ((2048, 1), (64, 32)):
        g = mx.Grid(n, K, np.full(n * n, 0.5), np.exp(1j * np.random.default_rng(1).uniform(0.3, 3.0, (K, 2))))
        b, x = mx.Edge(g, m, prec), mx.Edge(g, m, prec)
        mx.check(lib.random_edge2d_gpu(b.h, 3))
        mx.check(lib.zero_edge2d_gpu(x.h))
        runs = []
        for _ in range(6):
            mx.check(lib.norm2_edge2d_gpu(x.h, mx._ptr(dot)))   # waits
            t = time.perf_counter()
            for _ in range(10):
                mx.check(lib.gsforward_edge2d_gpu(one, one, b.h, x.h))
            mx.check(lib.norm2_edge2d_gpu(x.h, mx._ptr(dot)))
            runs.append(time.perf_counter() - t)
        times.append(min(runs[1:]))
    assert times[0] < 1.7 * times[1]


@pytest.mark.parametrize("n, m, K", [(8, 16, 100), (32, 5, 40), (64, 1, 20), (32, 17, 70), (66, 16, 60)])
@pytest.mark.parametrize("prec", [mx.C128, mx.CDD])
@pytest.mark.parametrize("direction", [0, 1])
def test_colour_smoother_whole_rows(oracle, n, m, K, prec, direction):
    """The patch smoother in four colours in batches of so many rows that a
    CTA takes a whole one: one chunk and several, several tables."""
    rng = np.random.default_rng(n)
    kap = 1.0 / (1.0 + 11.0 * rng.random(n * n))
    fac = np.exp(1j * rng.uniform(0.3, 3.0, (K, 2)))
    g = mx.Grid(n, K, kap, fac)
    b, x = cv(rng, K, m, 2 * n * n), cv(rng, K, m, 2 * n * n)
    eb, ex = mx.Edge(g, m, prec, b), mx.Edge(g, m, prec, x)
    mx.check(mx.lib().gscolour_edge2d_gpu(mx.fz(1.0), mx.fz(0.8), eb.h, ex.h, direction))
    got = ex.get()
    for k in {0, K // 2, K - 1}:
        for v in {0, m // 2, m - 1}:
            want = oracle.gs_edge_colour(n, kap, *fac[k], 1.0, 0.8, direction, b[k, v], x[k, v])
            assert rel(got[k, v], want) < 1e-11


@pytest.mark.parametrize("n, m, K", [(64, 6, 512), (8, 16, 512)])
def test_colour_smoother_batch_shape(n, m, K):
    """The four-colour smoother of float-float blocks costs about as much for
    vectors spread over many k-points as for the same number at 32 per
    k-point (1.7 to 5 times as much with every row cut in four)."""
    import time
    lib, one, dot = mx.lib(), mx.fz(1.0), np.zeros(K * m)
    times = []
    for kk, mm in ((K, m), (K * m // 32, 32)):
        g = mx.Grid(n, kk, np.full(n * n, 0.5), np.exp(1j * np.random.default_rng(1).uniform(0.3, 3.0, (kk, 2))))
        b, x = mx.Edge(g, mm, mx.CDD), mx.Edge(g, mm, mx.CDD)
        mx.check(lib.random_edge2d_gpu(b.h, 3))
        mx.check(lib.zero_edge2d_gpu(x.h))
        runs = []
        for _ in range(6):
            mx.check(lib.norm2_edge2d_gpu(x.h, mx._ptr(dot)))   # waits
            t = time.perf_counter()
            for _ in range(4):
                mx.check(lib.gscolour_edge2d_gpu(one, one, b.h, x.h, 0))
            mx.check(lib.norm2_edge2d_gpu(x.h, mx._ptr(dot)))
            runs.append(time.perf_counter() - t)
        times.append(min(runs[1:]))
    assert times[0] < 2.0 * times[1]


@pytest.mark.parametrize("K, m", [(32, 32), (41, 25), (3000, 1)])
@pytest.mark.parametrize("prec", [mx.C128, mx.CDD, mx.C64])
def test_shifts_of_many_pairs(oracle, K, m, prec):
    """The operator with a shift per (k-point, vector): the most pairs whose
    shifts are converted on the host (1024), one more and many."""
    n = 6
    rng = np.random.default_rng(K)
    kap = 1.0 / (1.0 + 11.0 * rng.random(n * n))
    fac = np.exp(1j * rng.uniform(-3.0, 3.0, (K, 2)))
    g = mx.Grid(n, K, kap, fac)
    x, y, shift = cv(rng, K, m, 2 * n * n), cv(rng, K, m, 2 * n * n), rng.uniform(-60.0, 0.0, (K, m))
    ex, ey = mx.Edge(g, m, prec, x), mx.Edge(g, m, prec, y)
    mx.check(mx.lib().addeval_shifted_edge2d_gpu(1.3, mx._ptr(shift), ex.h, ey.h))
    got = ey.get()
    for k in {0, K // 3, K - 1}:
        for v in range(m):
            want = oracle.addeval_edge(n, kap, *fac[k], 1.3, shift[k, v], x[k, v], y[k, v])
            assert rel(got[k, v], want) < TOL[prec]


@pytest.mark.parametrize("n", [1, 8, 31, 32, 33])
def test_hermitian_inverses_of_many(n):
    """Inverses of more small matrices than there are SMs (orders up to 32
    take a form of their own) and of an order beyond; one of them indefinite.
    Bound as in test_hermitian_inverse_orders."""
    rng = np.random.default_rng(n)
    K = 200
    A, info = mx.Matrix(n, K), np.zeros(K, np.int32)
    q = [np.linalg.qr(cv(rng, n, n))[0] for _ in range(K)]
    a = np.array([(u * np.linspace(1.0, 10.0, n)) @ u.conj().T for u in q])
    a = (a + np.conj(np.transpose(a, (0, 2, 1)))) / 2
    A.put(a)
    mx.check(mx.lib().potrf_matrix_gpu(A.h, mx._ptr(info)))
    assert not info.any()
    assert rel(A.get(), np.linalg.inv(a)) < 100 * n * 2.2e-16
    a[7] -= 20.0 * np.eye(n)
    A.put(a)
    mx.check(mx.lib().potrf_matrix_gpu(A.h, mx._ptr(info)))
    assert info[7] != 0 and info.astype(bool).sum() == 1


@pytest.mark.parametrize("n", [4, 33, 70])
def test_eigenvalues_with_nan(n):
    """A NaN on the diagonal stays there and the other eigenvalues ascend
    around it, each with its eigenvector; a pencil that turns NaN as a whole
    reports that or NaN eigenvalues."""
    K = 2
    d = np.arange(1.0, n + 1.0)[::-1]
    a = np.array([np.diag(d), np.diag(d)]).astype(complex)
    a[1, 2, 2] = np.nan
    A, info, lam = mx.Matrix(n, K), np.zeros(K, np.int32), np.zeros((K, n))
    A.put(a)
    mx.check(mx.lib().syev_matrix_gpu(A.h, mx._ptr(lam), mx._ptr(info)))
    assert np.array_equal(lam[0], np.sort(d))
    assert np.array_equal(np.delete(lam[1], 2), np.sort(np.delete(d, 2))) and np.isnan(lam[1, 2])
    z = np.abs(A.get())
    assert np.array_equal(z[0], np.eye(n)[:, ::-1])
    assert np.array_equal(np.sort(z[1].argmax(0)), np.arange(n)) and np.array_equal(z[1].sum(0), np.ones(n))
    A.put(a)
    B = mx.Matrix(n, K)
    B.put(np.array([np.eye(n)] * K))
    mx.check(mx.lib().sygv_matrix_gpu(A.h, B.h, mx._ptr(lam), mx._ptr(info)))
    assert info[0] == 0 and np.abs(lam[0] - np.sort(d)).max() < 1e-12 * n
    assert info[1] != 0 or np.isnan(lam[1]).all()


def test_pencils_of_large_order():
    """Generalised eigenvalues of orders whose rotation data alone takes more
    than 48 KB of shared memory (diagonal matrices: nothing to rotate)."""
    n = 940
    d = np.linspace(1.0, 2.0, n)
    A, B, info, lam = mx.Matrix(n, 1), mx.Matrix(n, 1), np.zeros(1, np.int32), np.zeros(n)
    A.put(np.diag(d))
    B.put(np.eye(n))
    mx.check(mx.lib().sygv_matrix_gpu(A.h, B.h, mx._ptr(lam), mx._ptr(info)))
    assert info[0] == 0 and np.abs(lam - d).max() < 1e-12


@pytest.mark.parametrize("level", [1, 2])
def test_node_vcycle_refuses_other_precisions(level):
    """d of another precision than b and x is refused on every level, those
    that run in one launch among them."""
    n0, L = 8, 2
    b, x, d, A, arr = node_levels(n0, L, 1, 2, mx.C128, FACTORS[:1])
    b[L].put(np.zeros(b[L].shape))
    x[L].put(np.zeros(x[L].shape))
    other = mx.Node(d[level].g, 2, mx.C64)
    arr[2][level] = other.h
    assert mx.lib().vcycle_node2d_gpu(L, 2, A.h, *arr) == -1
    arr[2][level] = d[level].h
    assert mx.lib().vcycle_node2d_gpu(L, 2, A.h, *arr) == 0


@pytest.mark.parametrize("n0, m", [(4, 5), (8, 12)])
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_solver_without_refinement(oracle, n0, m, precision):
    """A hierarchy of one grid: the dense eigenpairs with their residuals.
    Bound: order times rounding unit times the largest eigenvalue (1e3), and a
    factor."""
    rng = np.random.default_rng(n0)
    kap = rng.uniform(0.3, 1.0, n0 * n0)
    fac = FACTORS[[0, 2]]
    s = mx.Solver(kap, n0=n0, L=0, ieigs=m - 2, m=m, method=1, precision=precision, max_nested=20, max_steps=20, wave=2,
                  relative=1, tol=1e-8)
    lam, steps, res = s.solve(fac)
    assert res[:, :m - 2].max() <= 1e-8 and not steps.any()
    for k, f in enumerate(fac):
        R = np.linalg.inv(np.linalg.cholesky(oracle.dense_edge(n0, kap, *f, 0.0, 1.0)))
        want = np.linalg.eigvalsh(R @ oracle.dense_edge(n0, kap, *f, 1.0, 0.0) @ R.conj().T)
        want = want[np.abs(want) > 1e-8]
        assert np.abs(lam[k] - want[:m]).max() < 1e-9


@pytest.mark.parametrize("n0, L, K, m, nu", [(10, 4, 4, 32, 2), (8, 5, 4, 32, 2), (8, 6, 2, 20, 2), (8, 6, 2, 20, 1),
                                             (10, 5, 4, 32, 2), (14, 3, 4, 32, 1)])
def test_node_vcycle_tall_bands(oracle, n0, L, K, m, nu):
    """c64 node V-cycles of batches whose bands are higher than the 8 rows
    that few vectors get: 16 to 46 rows, other heights on the way down than up
    (512^2: 16 and 18, 256^2: 44 and 46, 320^2: 24 and 28), last bands of 8 to
    36 rows."""
    rng = np.random.default_rng(n0 + L)
    n = n0 << L
    fac = FACTORS[[0, 2, 1, 0]][:K]
    b, x, d, A, arr = node_levels(n0, L, K, m, mx.C64, fac)
    b[L].put(cv(rng, K, m, n * n))
    x[L].put(cv(rng, K, m, n * n))
    rhs, start = b[L].get(), x[L].get()
    mx.check(mx.lib().vcycle_node2d_gpu(L, nu, A.h, *arr))
    got = x[L].get()
    for k, v in [(0, 0), (1, m // 2), (K - 1, m - 1)]:
        want = node_cycle(oracle, n0, L, fac[k], rhs[k, v], start[k, v], nu)
        assert rel(got[k, v], want) < 1e-4


@pytest.mark.parametrize("n, m, K", [(260, 3, 1), (514, 1, 2), (514, 1, 4)])
@pytest.mark.parametrize("prec", [mx.C128, mx.CDD, mx.C64])
@pytest.mark.parametrize("direction", [0, 1])
def test_row_smoother_table_refill(oracle, n, m, K, prec, direction):
    """The row-order smoother on rows of more columns than its table of
    matrices holds (256).  In 64 bits the oracle's residuals are differences
    of curls of size n^2: its rounding is the bound."""
    rng = np.random.default_rng(n)
    kap = 1.0 / (1.0 + 11.0 * rng.random(n * n))
    fac = np.exp(1j * rng.uniform(0.3, 3.0, (K, 2)))
    g = mx.Grid(n, K, kap, fac)
    b, x = cv(rng, K, m, 2 * n * n), cv(rng, K, m, 2 * n * n)
    eb, ex = mx.Edge(g, m, prec, b), mx.Edge(g, m, prec, x)
    fn = [mx.lib().gsforward_edge2d_gpu, mx.lib().gsbackward_edge2d_gpu][direction]
    mx.check(fn(mx.fz(1.0), mx.fz(0.8), eb.h, ex.h))
    got = ex.get()
    for k in {0, K - 1}:
        for v in {0, m - 1}:
            want = oracle.gs_edge(n, kap, *fac[k], 1.0, 0.8, direction, b[k, v], x[k, v])
            assert rel(got[k, v], want) < (1e-4 if prec == mx.C64 else 8 * n * n * 2.0 ** -53)


@pytest.mark.parametrize("n0, negative", [(4, 3), (8, 5)])
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_negative_coarse_kappa(oracle, n0, negative, precision):
    """A coarsest grid with negative kappa starts from the pencil of the edge
    matrices (orders 32, in shared memory, and 128): as many negative
    eigenvalues as cells, here the wanted ones, against the dense pencil.
    kappa is so small there that A + M stays definite.  Bound: order times
    rounding unit times the largest eigenvalue (1e3), and a factor."""
    rng = np.random.default_rng(n0)
    kap = rng.uniform(0.3, 1.0, n0 * n0)
    kap[rng.choice(n0 * n0, negative, replace=False)] = -1e-4
    m = negative - 1
    s = mx.Solver(kap, n0=n0, L=0, ieigs=m, m=m, method=1, precision=precision, max_nested=20, max_steps=20, wave=2,
                  relative=1, tol=1e-8)
    lam, _, res = s.solve(FACTORS[[0, 2]])
    assert res.max() <= 1e-8
    for k, f in enumerate(FACTORS[[0, 2]]):
        R = np.linalg.inv(np.linalg.cholesky(oracle.dense_edge(n0, kap, *f, 0.0, 1.0)))
        want = np.linalg.eigvalsh(R @ oracle.dense_edge(n0, kap, *f, 1.0, 0.0) @ R.conj().T)
        assert (want[:negative] < -1e-8).all() and abs(want[negative]) < 1e-8
        assert np.abs(lam[k] - want[:m]).max() < 1e-9
