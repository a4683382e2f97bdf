"""The Gram-Schmidt dots of complex sectors in their fixed-point forms (tiles of 1024 and 256 doubles; one exponent per
vector in batched instances) against extended precision and against the FP64 pass."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = {1: "1024", 2: "256", 3: "batch"}


def dots(V, w, form):
    import blqh_gb300 as B
    from blqh_gb300._lib import lib

    ctx = B.Context.default()
    V, w = np.ascontiguousarray(V, np.complex128), np.ascontiguousarray(w, np.complex128)
    h = np.zeros(len(V), np.complex128)
    ptr = [a.ctypes.data_as(ctypes.c_void_p) for a in (V, w, h)]
    ctx.check(lib().blqh_debug_dots(ctx.h, 2 * w.size, len(V), ptr[0], ptr[1], form, ptr[2]))
    return h


def exact(V, w):
    wl = w.astype(np.clongdouble)
    return np.array([np.sum(v.astype(np.clongdouble).conj() * wl) for v in V])


def rms(a, b):
    return float(np.sqrt(np.mean(abs(a - b) ** 2)))


SIZES = [11, 79, 1430, 5940, 26176, 60096, 100141]  # complex entries


@pytest.mark.parametrize("form", FORMS, ids=FORMS.get)
@pytest.mark.parametrize("dim", SIZES)
def test_entries_keep_53_bits_down_to_a_sixteenth_of_the_largest(dim, form):
    """Vectors with one entry of 1.5 and one of 2^-4 times a number of 53 bits, against unit vectors: the dots are
    those entries, exactly, whatever the length."""
    rng = np.random.default_rng(dim)
    at = rng.choice(np.arange(1, dim), 5, replace=False)
    at[0] = dim - 1
    V = np.zeros((5, dim), np.complex128)
    w = np.zeros(dim, np.complex128)
    odd = 1.0 + (2 * rng.integers(0, 2 ** 51, 5) + 1) * 2.0 ** -52  # last bit set
    for k in range(5):
        V[k, 0] = 1.5
        V[k, at[k]] = odd[k] * 2.0 ** -4 * (1 if k % 2 else 1j)
        w[at[k]] = 1.0
    V[:, at] = np.where(np.eye(5) > 0, V[:, at], 0)
    h = dots(V, w, form)
    assert np.array_equal(h, np.array([V[k, at[k]].conj() for k in range(5)]))


@pytest.mark.parametrize("dim", SIZES)
def test_random_vectors(dim):
    """Normalized random vectors: no further off than the FP64 dots (root mean square over 24 vectors)."""
    rng = np.random.default_rng(dim + 1)
    V = rng.standard_normal((24, 2 * dim)).view(np.complex128)
    w = rng.standard_normal(2 * dim).view(np.complex128)
    V /= np.linalg.norm(V, axis=1, keepdims=True)
    w /= np.linalg.norm(w)
    ref = exact(V, w)
    err = {f: rms(dots(V, w, f), ref) for f in range(4)}
    assert all(err[f] <= err[0] for f in FORMS), err


@pytest.mark.parametrize("sec,d", [((8, 8, 4, 0, 1), 0.9), ((12, 12, 6, 0, 5), 0.3), ((12, 12, 6, 0, 5), 2.7),
                                   ((14, 14, 7, 0, 3), 0.9)], ids=str)
def test_krylov_vectors(sec, d):
    """The vectors of a run against what its step leaves of H v after the three-term update, as the pass meets them
    (dots that are rounding noise themselves): no further off than the FP64 dots."""
    import blqh_gb300 as B
    from blqh_gb300._lib import lib

    b = B.Basis(*sec)
    H = B.Hamiltonian(b, d)
    V = []
    for m in (1, 2, 3, 5, 8, 12, 16, 20, 30, 39, 40):
        L = B.Lanczos(H, max_steps=m, tol=0.0, seed=3, accumulate=1)
        L.iterate()
        x, y = np.zeros(H.dim, np.complex128), np.zeros(H.dim, np.complex128)
        L.ctx.check(lib().blqh_debug_lanczos_product(L.h, x.ctypes.data_as(ctypes.c_void_p),
                                                     y.ctypes.data_as(ctypes.c_void_p)))
        L.close()
        V.append(x)
    V = np.array(V)
    w = y - V[-1] * np.vdot(V[-1], y) - V[-2] * np.vdot(V[-2], y)
    ref = exact(V, w)
    err = {f: rms(dots(V, w, f), ref) for f in range(4)}
    assert all(err[f] <= err[0] for f in FORMS), err
    H.close()
    b.close()


@pytest.mark.parametrize("size", [2.0 ** -29, 2.0 ** -31, 2.0 ** -33, 2.0 ** -35, 2.0 ** -38, 2.0 ** -46])
@pytest.mark.parametrize("dim", [79, 5940, 60096])
def test_batched_correction(dim, size):
    """w - sum_k h_k V_k of 64 random vectors, coefficients of about `size` of |w|: no further off than the plain FP64
    sum, which subtracts vector by vector (restated here), whichever form the instances take."""
    import blqh_gb300 as B
    from blqh_gb300._lib import lib

    rng = np.random.default_rng(dim)
    V = rng.standard_normal((64, 2 * dim)).view(np.complex128)
    V /= np.linalg.norm(V, axis=1, keepdims=True)
    w = rng.standard_normal(2 * dim).view(np.complex128)
    w /= np.linalg.norm(w)
    h = rng.choice([-1, 1], 128).view() * size * rng.uniform(0.5, 1.0, 128)
    h = h.view(np.complex128)
    ref = w.astype(np.clongdouble) - np.sum(h.astype(np.clongdouble)[:, None] * V.astype(np.clongdouble), axis=0)
    plain = w.copy()
    for k in range(64):
        plain -= h[k] * V[k]
    ctx = B.Context.default()
    out = w.copy()
    ctx.check(lib().blqh_debug_batch_update(ctx.h, 2 * dim, 64, *(a.ctypes.data_as(ctypes.c_void_p) for a in (V, out, h))))
    err, native = rms(out, ref), rms(plain, ref)
    print("update", dim, size, "%.3f" % (err / native))
    assert err <= native * (1 + 1e-3), (err, native)  # (the FP64 form is the same sum up to fused operations)
