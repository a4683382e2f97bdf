"""The Lanczos step on both sides of the sizes where its kernels change: 256- and 1024-double tiles and one or four
slices of vectors in complex sectors, sums in the dots' last block or in a kernel of their own in real ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 20
CASES = [  # kind, sector, tiles: complex 1024-double tiles (256-double ones up to 24 of them), real 1024-row tiles
    ("mono", (24, 12, 0, 1), 19), ("spin", (8, 8, 4, 4, 1, 3), 32), ("mono", (30, 10, 0, 3), 196),
    ("ground", (14, 14, -1, 0, 1), 400), ("ground", (14, 8, 4, 0, 0), 35), ("mono", (30, 10, 0, 0), 98),
    ("ground", (14, 10, 5, 0, 0), 140),
]


@pytest.mark.parametrize("kind,sec,tiles", CASES, ids=str)
def test_coefficients_against_numpy(kind, sec, tiles):
    """The first coefficients equal those of the plain recurrence with full reorthogonalization in FP64 on the host.
    Rounding of 2^-52 |H| a step, |H| < 30, amplified by the recurrence at most a thousandfold over 20 steps: 1e-10."""
    import scipy.sparse as sp

    import blqh_gb300 as B

    b = {"mono": B.basis_mono, "spin": B.basis_spin, "ground": B.Basis}[kind](*sec)
    H = B.hamiltonian_mono(b, 1.0) if kind == "mono" else (B.hamiltonian_spin if kind == "spin" else B.Hamiltonian)(b, 0.9)
    assert -(-H.dim * (2 if H.is_complex else 1) // 1024) == tiles
    rng = np.random.default_rng(tiles)
    v = rng.standard_normal(H.dim) + (1j * rng.standard_normal(H.dim) if H.is_complex else 0)
    v /= np.linalg.norm(v)
    L = B.Lanczos(H, max_steps=STEPS, tol=0.0, start=v)
    assert L.iterate() == STEPS
    a, be = L.coeffs()
    L.close()
    rp, col, val = H.csr()
    M = sp.csr_matrix((val, col, rp), shape=(H.dim, H.dim))
    V, ra, rb = [v], [], []
    for j in range(STEPS):
        w = M @ V[j]
        ra.append(np.vdot(V[j], w).real)
        for _ in range(2):
            w = w - np.array(V).T @ (np.array(V).conj() @ w)
        rb.append(np.linalg.norm(w))
        V.append(w / rb[-1])
    assert np.max(np.abs(a - ra)) < 1e-10 and np.max(np.abs(be[1:] - rb)) < 1e-10
    H.close()
    b.close()
