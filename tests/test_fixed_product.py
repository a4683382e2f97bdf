"""The fixed-point product of complex FP64 matrices, as the Lanczos recurrence takes it, against the same matrix in
extended precision: the vector's scale comes from the kernel before it (256- and 1024-double tiles, with and without
the full Gram-Schmidt pass, the pass's FP64 branch) or from the start vector."""
import ctypes
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def B():
    import blqh_gb300

    return blqh_gb300


def build(B, kind, sec):
    if kind == "spin":
        b = B.basis_spin(*sec)
        return b, B.hamiltonian_spin(b, 0.9)
    if kind == "mono":
        b = B.basis_mono(*sec)
        return b, B.hamiltonian_mono(b, 1.0)
    b = B.Basis(*sec)
    return b, B.Hamiltonian(b, 0.9)


def product(L, dim):
    from blqh_gb300._lib import lib

    x, y = np.zeros(dim, np.complex128), np.zeros(dim, np.complex128)
    L.ctx.check(lib().blqh_debug_lanczos_product(L.h, x.ctypes.data_as(ctypes.c_void_p),
                                                 y.ctypes.data_as(ctypes.c_void_p)))
    return x, y


def errors(H, csr, x, y, rows):
    """y - H x of the sampled rows in extended precision, and each row's bound from the operands' rounding: the
    vector's to 2^-58 of its largest entry, the row's to 2^-57 of its largest off-diagonal one, and six FP64
    roundings of the row's sum and its diagonal term."""
    rp, col, val = csr
    n = rp[rows + 1] - rp[rows]
    first = np.cumsum(n) - n
    idx = np.repeat(rp[rows] - first, n) + np.arange(n.sum())
    r = np.repeat(rows, n)
    a, xc = val[idx], x[col[idx]]
    exact = np.add.reduceat(a.astype(np.clongdouble) * xc.astype(np.clongdouble), first)
    off = np.where(col[idx] == r, 0, a)
    dg = np.add.reduceat(np.where(col[idx] == r, a, 0), first)
    big = np.maximum.reduceat(np.maximum(abs(off.real), abs(off.imag)), first)
    l1 = np.add.reduceat(abs(off.real) + abs(off.imag), first)
    x1 = np.add.reduceat(np.where(off != 0, abs(xc.real) + abs(xc.imag), 0), first)
    top = max(np.max(abs(x.real)), np.max(abs(x.imag)))
    part = abs(exact - dg * x[rows]) + abs(dg * x[rows])
    bound = l1 * top * 2.0 ** -58 + x1 * big * 2.0 ** -57 + 6 * 2.0 ** -53 * part.astype(float)
    e = y[rows] - exact
    return np.maximum(abs(e.real), abs(e.imag)).astype(float), bound


CASES = [  # kind, sector, rows: 79 .. 100,141 states, short and long tiles
    ("ground", (8, 8, 4, 0, 1)), ("ground", (8, 7, -1, 3, 1)), ("ground", (12, 12, 6, 3, 5)), ("spin", (8, 8, 4, 4, 1, 3)),
    ("ground", (14, 14, 7, 0, 3)), ("mono", (30, 10, 0, 3)),
]


@pytest.mark.parametrize("kind,sec", CASES, ids=str)
@pytest.mark.parametrize("reorth", [True, False], ids=["full", "local"])
def test_no_further_off_than_native_fp64(B, kind, sec, reorth):
    """Krylov vectors after 0, 1, 2, 12 and 70 steps: every sampled row within its bound, and the error's root mean
    square over them no larger than that of the native FP64 product of the same vector."""
    b, H = build(B, kind, sec)
    assert H.is_complex
    csr = H.csr()
    rng = np.random.default_rng(zlib.crc32(repr(sec).encode()))
    rows = np.sort(rng.choice(H.dim, min(H.dim, 3000), replace=False))
    for m in (0, 1, 2, 12, 70):
        r = rng.standard_normal(2 * H.dim).view(np.complex128)
        L = B.Lanczos(H, max_steps=max(1, m), tol=0.0, start=r, reorth=reorth)
        if m:
            assert L.iterate() == m
        x, y = product(L, H.dim)
        L.close()
        e, bound = errors(H, csr, x, y, rows)
        assert np.all(e <= bound), float(np.max(e / bound))
        L = B.Lanczos(H, max_steps=1, tol=0.0, start=x, accumulate=1)
        en, _ = errors(H, csr, *product(L, H.dim), rows)
        L.close()
        rms, native = float(np.sqrt(np.mean(e ** 2))), float(np.sqrt(np.mean(en ** 2)))
        assert rms <= native, (m, rms, native)
    H.close()
    b.close()


@pytest.mark.parametrize("kind,sec", CASES[2:], ids=str)
def test_rows_without_their_diagonal_term(B, kind, sec):
    """A start vector that is zero on every other state: the rows of those states sum off-diagonal terms alone, where
    the vector's rounding is not hidden by that of the FP64 diagonal term (which both products share). Errors as
    above: bounded, and no larger than native FP64's."""
    b, H = build(B, kind, sec)
    csr = H.csr()
    rng = np.random.default_rng(3)
    r = rng.standard_normal(2 * H.dim).view(np.complex128)
    r[1::2] = 0
    rows = np.arange(1, H.dim, 2)[:3000]
    err = {}
    for accumulate in (0, 1):
        L = B.Lanczos(H, max_steps=1, tol=0.0, start=r, accumulate=accumulate)
        x, y = product(L, H.dim)
        L.close()
        assert not x[1::2].any()
        e, bound = errors(H, csr, x, y, rows)
        assert accumulate or np.all(e <= bound)
        err[accumulate] = float(np.sqrt(np.mean(e ** 2)))
    print("half", kind, sec, err)
    assert err[0] <= err[1], err
    H.close()
    b.close()


@pytest.mark.parametrize("kind,sec", [("mono", (24, 12, 0, 1)), ("spin", (8, 8, 4, 4, 1, 3)), ("ground", (14, 14, 7, 0, 3))],
                         ids=str)
def test_even_vectors_and_long_rows(B, kind, sec):
    """Every entry of the vector as large as the largest one, each with the sign that makes one row's terms add up:
    the largest sums that the row's 128 bits can meet."""
    b, H = build(B, kind, sec)
    csr = H.csr()
    rp, col, val = csr
    long = int(np.argmax(np.diff(rp)))
    r = np.full(H.dim, 1 + 1j)
    k = slice(rp[long], rp[long + 1])
    r.real[col[k]] = np.where(val[k].real < 0, -1, 1)
    r.imag[col[k]] = np.where(val[k].imag > 0, -1, 1)
    L = B.Lanczos(H, max_steps=1, tol=0.0, start=r)
    x, y = product(L, H.dim)
    rows = np.unique(np.append(np.linspace(0, H.dim - 1, 2000).astype(int), long))
    e, bound = errors(H, csr, x, y, rows)
    assert np.all(e <= bound), float(np.max(e / bound))
    for o in (L, H, b):
        o.close()


@pytest.mark.parametrize("sec", [(8, 8, 4, 0, 1), (12, 12, 6, 3, 5), (14, 14, 7, 0, 3)], ids=str)
def test_full_pass_near_an_invariant_subspace(B, monkeypatch, sec):
    """From a nearly converged state the first step's coefficients are not small and the full pass subtracts in FP64,
    one block then scaling the vector and its planes (256- and 1024-double tiles): the next product is as good as any,
    and ten steps give the FP64 pass's coefficients (beta_1 ~ 1e-6 known to 1e-15: what follows to 1e-7)."""
    b, H = build(B, "ground", sec)
    csr = H.csr()
    for steps in range(20, 200, 4):
        L = B.Lanczos(H, max_steps=steps, tol=0.0, seed=2)
        L.iterate()
        psi, E = L.ritz_vector(), L.rayleigh()
        L.close()
        res = np.linalg.norm(H.spmv(psi) - E * psi)
        if res < 3e-6:
            break
    assert res > 1e-8
    L = B.Lanczos(H, max_steps=1, tol=0.0, start=psi)
    L.iterate()
    x, y = product(L, H.dim)
    L.close()
    assert abs(np.linalg.norm(x) - 1) < 1e-13 and abs(np.vdot(psi, x)) < 1e-8
    e, bound = errors(H, csr, x, y, np.linspace(0, H.dim - 1, 2000).astype(int))
    assert np.all(e <= bound), float(np.max(e / bound))
    out = []
    for env in ("0", "1"):
        monkeypatch.setenv("BLQH_GS_FP64", env)
        L = B.Lanczos(H, max_steps=10, tol=0.0, start=psi)
        L.iterate()
        out.append(np.concatenate(L.coeffs()))
        L.close()
    assert np.max(np.abs(out[0] - out[1])) < 1e-7
    H.close()
    b.close()


def test_infinite_elements_stay_visible(B):
    """A tunnelling amplitude at the end of FP64's range, which short orbits multiply beyond it: a row with an infinite
    element has no finite product, and the recurrence no finite coefficient."""
    b = B.basis_spin(4, 4, -1, -1, 0, 1)
    H = B.hamiltonian_spin(b, 0.9, delta_sas=1.79e308)
    assert H.is_complex
    rp, col, val = H.csr()
    row = np.repeat(np.arange(H.dim), np.diff(rp))
    rows = np.unique(row[~(np.isfinite(val.real) & np.isfinite(val.imag)) & (col != row)])
    assert len(rows)
    for accumulate in (0, 1):
        L = B.Lanczos(H, max_steps=1, tol=0.0, start=np.ones(H.dim), accumulate=accumulate)
        y = product(L, H.dim)[1][rows]
        assert not np.any(np.isfinite(y.real) & np.isfinite(y.imag))
        L.iterate()
        assert not np.isfinite(L.coeffs()[0][0])
        L.close()
    H.close()
    b.close()
