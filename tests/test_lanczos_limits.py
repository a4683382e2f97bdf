"""Lanczos options at the ends of their ranges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [767, 768, 1534, 1535, 1536, 3070, 3071, 3072, 4096])
def test_convergence_check_at_every_allowed_length(steps):
    """The convergence check's shared memory at the step limits where its staging level changes (4 doubles a step fit
    48 KB up to 1,534 steps, 2 up to 3,070): every run stops at the same step with the same coefficients."""
    import blqh_gb300 as B

    b = B.Basis(12, 10, 5, 3, 1)
    H = B.Hamiltonian(b, 0.9)
    assert H.dim > 1000
    out = []
    for m in (200, steps):
        L = B.Lanczos(H, max_steps=m, tol=1e-10, check_every=10, seed=4)
        n = L.iterate()
        out.append((n, *L.coeffs()))
        L.close()
    assert 10 < out[0][0] < 200 and out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
    H.close()
    b.close()
