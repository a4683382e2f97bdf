"""The tridiagonal eigen-solve of a Lanczos run: all eigenvalues at the ends of its shared-memory ranges, and its fast
route (everything in shared memory, counting rounds played in FP32 pairs) against the plain recurrences, which runs of
thousands of allowed steps take, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 3, 32, 33, 150, 767, 768, 1536])
def test_all_ritz_values(m):
    """Against LAPACK's; both are good to a few ulp of the spectrum's size (below 100) per eigenvalue: 1e-12."""
    import blqh_gb300 as B

    b = B.Basis(12, 8, 4, 5, 3)
    H = B.Hamiltonian(b, 0.9)
    L = B.Lanczos(H, max_steps=m, tol=0.0, seed=2)
    L.iterate()
    e, _ = L.eig()
    a, be = L.coeffs()
    m = L.steps
    ref = np.linalg.eigvalsh(np.diag(a[:m]) + np.diag(be[1:m], 1) + np.diag(be[1:m], -1))
    assert np.max(np.abs(e[:m] - ref)) < 1e-12
    for x in (L, H, b):
        x.close()


@pytest.mark.parametrize("sec", [(12, 8, 4, 0, 0), (12, 8, 4, 5, 3)], ids=str)
@pytest.mark.parametrize("d", [0.4, 0.9, 1.7])
def test_lowest_pair_is_the_plain_one(sec, d):
    import blqh_gb300 as B

    b = B.Basis(*sec)
    H = B.Hamiltonian(b, d)
    out = []
    for steps in (500, 2000, 4000):  # both in shared memory; the vector's solve plain; all of it plain
        L = B.Lanczos(H, max_steps=steps, tol=1e-11, check_every=10, seed=7)
        L.iterate()
        a, be = L.coeffs()
        psi = np.array(L.ritz_vector())
        out.append((L.steps, a[: L.steps], be[: L.steps], psi))
        L.close()
    for o in out[1:]:
        assert o[0] == out[0][0]
        assert all(np.array_equal(x, y) for x, y in zip(o[1:], out[0][1:]))
    H.close()
    b.close()
