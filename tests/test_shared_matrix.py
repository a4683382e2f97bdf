"""One matrix under several Lanczos objects: each keeps what it derives from the matrix to itself."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SECTORS = [(8, 8, 4, 0, 1), (12, 12, 6, 3, 5), (12, 12, 6, 0, 0)]  # complex, complex, real


def create(ctx, H, steps, prec_opts):
    from blqh_gb300._lib import LanczosOpts, lib

    h = ctypes.c_void_p()
    o = LanczosOpts(steps, 1, 0.0, 10, 5, 0, prec_opts)
    ctx.check(lib().blqh_lanczos_create(ctx.h, H.h, ctypes.byref(o), ctypes.byref(h)))
    return h


def coefficients(ctx, H, steps=60):
    from blqh_gb300._lib import lib

    h = create(ctx, H, steps, 0)
    n = ctypes.c_int()
    ctx.check(lib().blqh_lanczos_iterate(h, ctypes.byref(n)))
    a, b = np.zeros(n.value), np.zeros(n.value + 1)
    ctx.check(lib().blqh_lanczos_coeffs(h, a.ctypes.data_as(ctypes.c_void_p), b.ctypes.data_as(ctypes.c_void_p)))
    lib().blqh_lanczos_destroy(h)
    return np.concatenate([a, b])


@pytest.mark.parametrize("sec", SECTORS, ids=str)
def test_objects_leave_nothing_on_the_matrix(sec):
    """A second object on the same matrix allocates as much as the first: no storage of the first one is left on the
    matrix, to outlive it or to be read before another stream has filled it."""
    import blqh_gb300 as B
    from blqh_gb300._lib import lib

    ctx = B.Context(0)
    b = B.Basis(*sec, ctx=ctx)
    H = B.Hamiltonian(b, 0.9)
    count = []
    for _ in range(2):
        lib().blqh_debug_fail_alloc(ctx.h, 100000)
        lib().blqh_lanczos_destroy(create(ctx, H, 60, 0))
        count.append(100000 - lib().blqh_debug_fail_alloc(ctx.h, 0))
    assert count[0] == count[1] > 0
    for x in (H, b, ctx):
        x.close()


@pytest.mark.parametrize("sec", SECTORS, ids=str)
def test_contexts_and_threads_share_a_matrix(sec):
    """Runs on the same matrix from four contexts, one after the other and from a thread each, return the same bits."""
    import blqh_gb300 as B

    ctx = [B.Context(0) for _ in range(4)]
    b = B.Basis(*sec, ctx=ctx[0])
    H = B.Hamiltonian(b, 0.9)
    ref = coefficients(ctx[0], H)
    for c in ctx[1:]:
        assert np.array_equal(coefficients(c, H), ref)
    got = [None] * len(ctx)

    def work(i):
        got[i] = [coefficients(ctx[i], H) for _ in range(3)]

    th = [threading.Thread(target=work, args=(i,)) for i in range(len(ctx))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert all(np.array_equal(r, ref) for g in got for r in g)
    for x in (H, b, *ctx):
        x.close()
