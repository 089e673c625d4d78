"""Calls of several host threads at once, each on objects of its own."""
import ctypes as C
import threading

import numpy as np
import pytest

import maxwell_gb300 as mx

pytestmark = pytest.mark.gpu


def _potrf(n, status, times):
    """Inverses of order n, into which a thread's matrix is turned back and forth."""
    A, info = mx.Matrix(n, 1), np.zeros(1, np.int32)
    A.put(2.0 * np.eye(n))

    def work():
        for _ in range(times):
            status.append(mx.lib().potrf_matrix_gpu(A.h, mx._ptr(info)))

    return work, lambda: np.array_equal(A.get()[0], (2.0 if times % 2 == 0 else 0.5) * np.eye(n))


def _vcycle(n0, L, status, times):
    """Node V-cycles with b = 0 from x = 0."""
    n = n0 << L
    grids = [mx.Grid(n, 1, None, np.exp(1j * np.array([[0.7, -1.3]])))]
    for _ in range(L):
        grids.append(grids[-1].coarsen())
    grids = grids[::-1]
    b, x, d = ([mx.Node(g, 1, mx.C128) for g in grids] for _ in range(3))
    b[L].put(np.zeros(b[L].shape))
    x[L].put(np.zeros(x[L].shape))
    A, info = mx.Matrix(n0 * n0, 1), np.zeros(1, np.int32)
    mx.check(mx.lib().densematrix_node2d_gpu(1, grids[0].h, A.h))
    mx.check(mx.lib().potrf_matrix_gpu(A.h, mx._ptr(info)))
    arr = [(C.c_void_p * (L + 1))(*[o.h for o in objs]) for objs in (b, x, d)]

    def work(keep=(grids, b, x, d)):
        for _ in range(times):
            status.append(mx.lib().vcycle_node2d_gpu(L, 2, A.h, *arr))

    return work, lambda: not x[L].get().any()


@pytest.mark.parametrize("small, large", [(lambda s: _potrf(8, s, 6000), lambda s: _potrf(160, s, 400)),
                                          (lambda s: _vcycle(4, 1, s, 6000), lambda s: _vcycle(8, 3, s, 2000))])
def test_sizes_of_one_kernel_in_two_threads(small, large):
    """The same kernels with little and with much dynamic shared memory, each
    size in a thread of its own: no call fails."""
    status = []
    jobs = [small(status), large(status)]
    threads = [threading.Thread(target=work) for work, _ in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not any(status)
    assert all(right() for _, right in jobs)
