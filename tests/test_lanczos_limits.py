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


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("sec", [(12, 10, 5, 3, 1), (14, 14, 7, 0, 3)], ids=str)
def test_accumulate_selects_native_fp64_in_complex_sectors(monkeypatch, sec, prec):
    """accumulate = 1 runs products and Gram-Schmidt sums in native FP64: the bits of the run whose integer and plane
    forms are all switched off; accumulate = 0 agrees to rounding (FP32 values: products good to 2^-48 of 500 terms)."""
    import blqh_gb300 as B

    b = B.Basis(*sec)
    H = B.Hamiltonian(b, 0.9, precision=B.VAL_FP64 if prec == "f64" else B.VAL_FP32)
    assert H.is_complex

    def run(accumulate):
        L = B.Lanczos(H, max_steps=25, tol=0.0, seed=4, accumulate=accumulate)
        L.iterate()
        r = np.concatenate(L.coeffs())
        L.close()
        return r

    native, fast = run(1), run(0)
    monkeypatch.setenv("BLQH_SPMV_FIXED", "0")
    monkeypatch.setenv("BLQH_GS_FP64", "1")
    assert np.array_equal(native, run(1))
    assert not np.array_equal(native, fast)
    assert np.max(np.abs(native - fast)) < 1e-9
    H.close()
    b.close()
