"""The Lanczos step's Gram-Schmidt passes: fixed-point planes (complex sectors) and the ordered FP64 / FP32-plane
passes (real sectors), against the FP64 pass on the stored vectors and a dense diagonalization of the same matrix.

Sizes sit at the edges of the tiles: vectors shorter than one 256-double tile, one entry short of and past tile
borders, and beyond the 65,536 doubles where 1024-double tiles take over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SECTORS = [  # (nphi, nel, nel_up, J, K): dimension 11 .. 60,096, complex and real
    (6, 6, 3, 1, 2), (8, 8, 4, 0, 1), (8, 7, -1, 3, 1), (10, 10, 5, 0, 3), (10, 9, 4, 3, 2), (12, 12, 6, 3, 5),
    (14, 14, 7, 0, 3), (8, 8, 4, 2, 0), (10, 10, 5, 5, 0), (12, 12, 6, 3, 0), (14, 14, 7, 3, 7),
]


@pytest.fixture(scope="module")
def B():
    import blqh_gb300

    return blqh_gb300


def _run(B, sec, prec, steps, d=0.9):
    b = B.Basis(*sec)
    H = B.Hamiltonian(b, d, precision=prec)
    L = B.Lanczos(H, max_steps=steps, tol=0.0, seed=3)
    m = L.iterate()
    e, _ = L.eig()
    psi = L.ritz_vector()
    E = L.rayleigh()
    a, be = L.coeffs()
    res = np.linalg.norm(H.spmv(psi) - E * psi)
    out = dict(m=m, e=e, psi=psi, E=E, a=a, b=be, res=res, dim=H.dim)
    if H.dim <= 700:
        rp, col, val = H.csr()
        D = np.zeros((H.dim, H.dim), val.dtype)
        D[np.repeat(np.arange(H.dim), np.diff(rp)), col] = val
        out["dense"] = np.linalg.eigvalsh((D + D.conj().T) / 2)
    for x in (L, H, b):
        x.close()
    return out


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("sec", SECTORS, ids=str)
def test_against_fp64_pass(B, monkeypatch, sec, prec):
    """Same recurrence as the FP64 pass: the first coefficients to 1e-11 (rounding times the growth of 15 steps),
    the lowest Ritz value of 120 steps to 1e-12 of its size (FP32 values: the pass's own 2^-46), residual of the
    ground state as small as the FP64 pass's."""
    p = B.VAL_FP64 if prec == "f64" else B.VAL_FP32
    r = _run(B, sec, p, 120)
    monkeypatch.setenv("BLQH_GS_FP64", "1")
    f = _run(B, sec, p, 120)
    k = min(15, r["m"], f["m"], r["dim"] // 2)
    assert np.max(np.abs(r["a"][:k] - f["a"][:k])) < 1e-11
    assert np.max(np.abs(r["b"][:k] - f["b"][:k])) < 1e-11
    assert abs(r["e"][0] - f["e"][0]) < 1e-12 * max(1.0, abs(f["e"][0]))
    assert r["res"] <= 2 * f["res"] + 1e-11
    if "dense" in r:
        assert abs(r["e"][0] - r["dense"][0]) < 1e-11


@pytest.mark.parametrize("sec", [s for s in SECTORS if s[:2] in ((6, 6), (8, 8))], ids=str)
def test_exhausted_krylov_space(B, sec):
    """As many steps as the sector has states: the run ends at an invariant subspace (the coefficients of the full
    pass are then not small and it subtracts in FP64), without copies of the ground level."""
    r = _run(B, sec, B.VAL_FP64, 400)
    assert r["m"] <= r["dim"]
    assert abs(r["e"][0] - r["dense"][0]) < 1e-11
    assert np.sum(np.abs(r["e"] - r["dense"][0]) < 1e-9) == np.sum(np.abs(r["dense"] - r["dense"][0]) < 1e-9) or \
        np.sum(np.abs(r["e"] - r["dense"][0]) < 1e-9) == 1


COMPLEX = [(6, 6, 3, 1, 2), (8, 8, 4, 0, 1), (8, 7, -1, 3, 1), (10, 10, 5, 0, 3), (12, 12, 6, 3, 5)]


@pytest.mark.parametrize("sharp", [False, True], ids=["spread", "concentrated"])
@pytest.mark.parametrize("sec", COMPLEX, ids=str)
def test_fixed_point_product(B, monkeypatch, sec, sharp):
    """The fixed-point SpMV of complex FP64 matrices against an extended-precision product of the same matrix: alpha_0
    and beta_1 of a start vector (spread, or nearly one basis state) are no further off than the FP64 kernel's, or
    below 4 ulp of the matrix's size where both are at rounding."""
    b = B.Basis(*sec)
    H = B.Hamiltonian(b, 0.9)
    assert H.is_complex
    r = np.random.RandomState(5)
    x = r.standard_normal(H.dim) + 1j * r.standard_normal(H.dim)
    if sharp:
        x *= 1e-7
        x[H.dim // 3] = 1.0
    rp, col, val = H.csr()
    x = x / np.linalg.norm(x)
    xl = x.astype(np.clongdouble) / np.sqrt(np.sum(np.abs(x.astype(np.clongdouble)) ** 2))
    y = np.add.reduceat(val.astype(np.clongdouble) * xl[col], rp[:-1])
    a0 = np.sum(xl.conj() * y).real
    b1 = np.sqrt(np.sum(np.abs(y - a0 * xl) ** 2))

    def off():
        L = B.Lanczos(H, max_steps=2, tol=0.0, start=x)
        L.iterate()
        a, be = L.coeffs()
        L.close()
        return max(abs(float(a[0] - a0)), abs(float(be[1] - b1)))

    fixed = off()
    monkeypatch.setenv("BLQH_SPMV_FIXED", "0")
    H2 = B.Hamiltonian(b, 0.9)
    H.close()
    H = H2
    native = off()
    assert fixed <= max(native, 4 * np.finfo(float).eps * float(abs(a0) + b1)), (fixed, native)
    H.close()
    b.close()


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_batched_complex_instances(B, prec):
    """Complex instances of a batch (fixed-point pass, one exponent per vector): vectors of 2 x 11 .. 2 x 636 doubles,
    some not a multiple of four, up to the whole Krylov space; energies as the dense matrix's (FP32 values finish
    with the FP64 quotient of a 1e-7 vector: 1e-9)."""
    secs = [s for s in SECTORS if s[4] not in (0, s[0] // 2) and s[0] <= 10 and s[1] == s[0]]
    b = B.Batch([B.instance(*s, d) for s in secs for d in (0.6, 1.4)], lam=100,
                precision=B.VAL_FP64 if prec == "f64" else B.VAL_FP32)
    b.solve()
    res = b.results()
    for i, r in enumerate(res):
        sec, d = secs[i // 2], (0.6, 1.4)[i % 2]
        ref = _run(B, sec, B.VAL_FP64, 100, d)
        assert r["dim"] == ref["dim"]
        assert abs(r["energy"] - ref["dense"][0]) < (1e-10 if prec == "f64" else 1e-9)
        psi = b.ground_state(i)
        assert abs(np.linalg.norm(psi) - 1) < 1e-12
        assert 1 - abs(np.vdot(psi, ref["psi"])) < 1e-10
    b.close()


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_batched_vectors_larger_than_shared_memory(B, prec):
    """Batches whose largest vector is beyond (418 kB), within (174 kB) and far below a block's shared memory: the
    area for it stops at what the kernel's own variables leave. 150 steps converge to 1e-10; FP32 values to 1e-9."""
    secs = [(12, 10, 5, 9, 3), (12, 9, 4, 5, 3), (12, 8, 4, 5, 3)]
    ref = []
    for s in secs:
        bas = B.Basis(*s)
        H = B.Hamiltonian(bas, 0.9)
        L = B.Lanczos(H, max_steps=200, tol=0.0)
        L.iterate()
        ref.append(L.eig()[0][0])
        for x in (L, H, bas):
            x.close()
    for pick in ([0], [1], [0, 2], [0, 1, 2]):
        b = B.Batch([B.instance(*secs[i], 0.9) for i in pick], lam=150,
                    precision=B.VAL_FP64 if prec == "f64" else B.VAL_FP32)
        b.solve()
        for i, r in zip(pick, b.results()):
            assert abs(r["energy"] - ref[i]) < (1e-10 if prec == "f64" else 1e-9)
        b.close()
