"""The batch's shape is tuned on what its solve runs."""
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_batches_with_and_without_planes_are_tuned_apart(tmp_path, monkeypatch):
    """Complex instances run another pass where there is no room for their planes: the two kinds of batch are two
    classes of the cache, each read back by the next of its kind. 79 states, 60 steps:
    energies converged to well below 1e-10 either way."""
    import blqh_gb300 as B
    from blqh_gb300._lib import lib

    cache = tmp_path / "tune.json"
    monkeypatch.setenv("BLQH_TUNE_CACHE", str(cache))
    monkeypatch.delenv("BLQH_TUNE", raising=False)
    ctx = B.Context(0)
    inst = [B.instance(8, 8, 4, 0, k, d) for k in (1, 3) for d in (0.7, 0.9)]
    energy, shape, keys = {}, {}, {}
    for free in (-1, 0, -1, 0):
        lib().blqh_debug_free_bytes(ctx.h, free)
        b = B.Batch(inst, lam=60, ctx=ctx)
        b.solve()
        e = np.array([r["energy"] for r in b.results()])
        s = b.shape()
        b.close()
        k = {k for k in json.loads(cache.read_text()) if k.startswith("batch|")}
        if free in energy:
            assert s == shape[free] and len(k) == 2
        energy[free], shape[free], keys[free] = e, s, k
    assert len(keys[-1]) == len(keys[0]) == 2
    assert np.max(np.abs(energy[-1] - energy[0])) < 1e-10
    ctx.close()
