"""Calls whose fast route needs more device memory than their plain one take the plain one where the memory is not
there. Every allocation of a call is made to fail in turn: the call then either reports BLQH_ERR_NOMEM or returns what
it returns otherwise, and the context stays usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NOMEM = -3


@pytest.fixture()
def ctx():
    import blqh_gb300 as B

    c = B.Context(0)
    yield c
    c.close()


def sweep(ctx, call, limit=400):
    """Results of `call` with its 1st, 2nd, ... allocation failing (None: NOMEM), until none is left to fail."""
    from blqh_gb300._lib import BlqhError, lib

    out = []
    for n in range(1, limit):
        lib().blqh_debug_fail_alloc(ctx.h, n)
        try:
            r = call()
        except BlqhError as e:
            assert e.code == NOMEM, e
            r = None
        if lib().blqh_debug_fail_alloc(ctx.h, 0):
            assert r is not None
            return out
        out.append(r)
    raise AssertionError("more allocations than expected")


SPIN = [  # even and odd nphi, with and without translation symmetry, real and complex, every route of the generator
    ((4, 4, 2, 2, 0, 0), dict(delta_v=0.01, delta_z=0.02)), ((4, 4, -1, -1, 0, 1), dict(delta_sas=0.2)),
    ((6, 6, 3, 3, 1, 2), {}), ((5, 3, 1, 1, 2, 1), {}), ((4, 3, 1, 1, 2, -1), dict(delta_v=0.01)),
]


@pytest.mark.parametrize("sec,kw", SPIN, ids=str)
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_spinful_build(ctx, sec, kw, prec):
    """The row generator's staging (two buffers) and its orbit-member table each fail over: rows counted, then written,
    and targets searched. Same columns; values are sums of at most ~60 terms of size <= 2 in another order, 2e-14
    (FP32 values: one rounding of entries below 16 apart, 1e-6)."""
    import blqh_gb300 as B

    p = B.VAL_FP64 if prec == "f64" else B.VAL_FP32
    b = B.basis_spin(*sec, ctx=ctx)

    def build():
        H = B.hamiltonian_spin(b, 0.8, precision=p, **kw)
        r = H.csr()
        H.close()
        return r

    rp, col, val = build()
    got = sweep(ctx, build)
    assert sum(r is not None for r in got) >= 5  # table, two staging buffers, the CSR's two arrays
    for r in got:
        if r is not None:
            assert np.array_equal(r[0], rp) and np.array_equal(r[1], col)
            assert np.max(np.abs(r[2] - val)) < (2e-14 if prec == "f64" else 1e-6)
    b.close()


@pytest.mark.parametrize("sec,kw", SPIN, ids=str)
def test_spinful_observables_and_regenerated_energy(ctx, sec, kw):
    import blqh_gb300 as B

    b = B.basis_spin(*sec, ctx=ctx)
    H = B.hamiltonian_spin(b, 0.8, **kw)
    L = B.Lanczos(H, max_steps=60)
    L.iterate()
    L.ritz_vector(copy=False)

    def values():
        o = L.observables_spin(b)
        return np.concatenate([[v for k, v in sorted(o.items()) if k != "occupation"], o["occupation"].ravel()])

    for call in (values, lambda: np.array([L.rayleigh_fp64()])):
        ref = call()
        got = sweep(ctx, call)
        assert any(r is not None for r in got)  # the table
        for r in got:
            if r is not None:
                assert np.max(np.abs(r - ref)) < 1e-12  # sums of a few thousand terms below 10 in another order
    for x in (L, H, b):
        x.close()


RUNS = [  # sector, values, allocations that a run can do without
    ((8, 8, 4, 0, 1), "f64", 7),   # complex FP64: split matrix (3), split vector, planes (3)
    ((12, 10, 5, 3, 1), "f64", 7),
    ((12, 10, 5, 3, 1), "f32", 3),  # complex FP32: planes
    ((12, 10, 5, 5, 0), "f64", 1),  # real FP64: FP32 plane
    ((12, 10, 5, 5, 0), "f32", 2),  # real FP32: two FP32 planes
]


@pytest.mark.parametrize("sec,prec,spare", RUNS, ids=str)
def test_lanczos(ctx, monkeypatch, sec, prec, spare):
    """A run that lacks one of its spare buffers returns the bits of the run that does without what it belongs to."""
    import blqh_gb300 as B

    b = B.Basis(*sec, ctx=ctx)
    H = B.Hamiltonian(b, 0.9, precision=B.VAL_FP64 if prec == "f64" else B.VAL_FP32)

    def run():
        L = B.Lanczos(H, max_steps=40, tol=0.0, seed=3)
        L.iterate()
        r = np.concatenate([*L.coeffs(), L.ritz_vector().view(np.float64)])
        L.close()
        return r

    modes = [run()]
    for var, val in (("BLQH_SPMV_FIXED", "0"), ("BLQH_GS_FP64", "1")):
        monkeypatch.setenv(var, val)
        modes.append(run())
        monkeypatch.delenv(var)
    got = [r for r in sweep(ctx, run) if r is not None]
    assert len(got) == spare
    assert all(any(np.array_equal(r, m) for m in modes) for r in got)
    H.close()
    b.close()


@pytest.mark.parametrize("sec,prec", [r[:2] for r in RUNS], ids=str)
def test_lanczos_leaves_memory_to_later_calls(ctx, monkeypatch, sec, prec):
    """FP64-valued runs take their copies and planes only while half of the free memory holds them: with none of it
    they return the bits of the run without either. FP32-valued runs count on theirs."""
    import blqh_gb300 as B
    from blqh_gb300._lib import lib

    b = B.Basis(*sec, ctx=ctx)
    H = B.Hamiltonian(b, 0.9, precision=B.VAL_FP64 if prec == "f64" else B.VAL_FP32)

    def run():
        L = B.Lanczos(H, max_steps=40, tol=0.0, seed=3)
        L.iterate()
        r = np.concatenate([*L.coeffs(), L.ritz_vector().view(np.float64)])
        L.close()
        return r

    full = run()
    monkeypatch.setenv("BLQH_SPMV_FIXED", "0")
    monkeypatch.setenv("BLQH_GS_FP64", "1")
    bare = run()
    monkeypatch.undo()

    def allocations():
        lib().blqh_debug_fail_alloc(ctx.h, 100000)
        r = run()
        return r, 100000 - lib().blqh_debug_fail_alloc(ctx.h, 0)

    _, most = allocations()
    lib().blqh_debug_free_bytes(ctx.h, 1000)
    r, least = allocations()
    assert np.array_equal(r, bare if prec == "f64" else full)
    assert (least < most) == (prec == "f64")
    lib().blqh_debug_free_bytes(ctx.h, 1 << 40)
    r, n = allocations()
    assert n == most and np.array_equal(r, full)
    H.close()
    b.close()


def _batch(ctx, prec="f64"):
    import blqh_gb300 as B

    b = B.Batch([B.instance(8, 8, 4, 0, k, 0.9) for k in (1, 0, 2, 3)], lam=40, threads=256, lanes_per_row=8, ctx=ctx,
                precision=B.VAL_FP64 if prec == "f64" else B.VAL_FP32)
    b.solve()
    r = [np.concatenate([[x["energy"], x["ritz0"]], b.ground_state(i).view(np.float64)])
         for i, x in enumerate(b.results())]
    b.close()
    return r


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_batch(ctx, prec):
    """Each allocation of a batch fails in turn: without the planes' buffer its complex instances take the FP64 pass
    (energies and, up to the convergence of 40 steps, vectors agree), the real one the bits it always has."""
    full = _batch(ctx, prec)
    got = [r for r in sweep(ctx, lambda: _batch(ctx, prec), 2000) if r is not None]
    assert len(got) >= 1
    for r in got:
        assert np.array_equal(r[1], full[1])
        for a, f in zip(r, full):
            assert abs(a[0] - f[0]) < 1e-10 and np.max(abs(a - f)) < 1e-6


def test_batch_with_planes_for_some_instances(ctx):
    """As many complex instances as half of the free memory holds planes for take the fixed-point pass, the others the
    FP64 pass; the real instance (the second) is not concerned. 79 states, 158 doubles: two planes of 42 rows of 160."""
    from blqh_gb300._lib import lib

    full = _batch(ctx)
    out = {}
    for n in range(4):
        lib().blqh_debug_free_bytes(ctx.h, 2 * n * (2 * 42 * 160 * 4))
        out[n] = _batch(ctx)
    lib().blqh_debug_free_bytes(ctx.h, -1)
    for n in range(4):
        for i, rank in ((0, 1), (2, 2), (3, 3)):
            assert np.array_equal(out[n][i], full[i] if n >= rank else out[0][i])
        assert np.array_equal(out[n][1], full[1])
    assert any(not np.array_equal(out[0][i], full[i]) for i in (0, 2, 3))
