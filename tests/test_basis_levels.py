"""The container-order emulation of the bases where its first growth levels (one block, up to 2,357 buckets) hand over
to the level kernels. The comment at each sector is the number of states inserted; a level ends at 13, 29, 59, 127,
257, 541, 1109, 2357 and 5087 of them. Everything is compared bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SECTORS = [
    (2, 2, 1, 0, 0),
    (11, 2, 1, 0, 0),   # 11
    (10, 3, 0, 0, 0),   # 12
    (9, 4, 0, 0, 0),    # 14
    (8, 3, 1, 0, 0),    # 28
    (11, 4, 0, 0, 0),   # 30
    (9, 5, 1, 0, 0),    # 126
    (9, 4, 2, 0, 0),    # 144
    (10, 5, 2, 0, 0),   # 540
    (8, 8, 4, 4, 4),
    (11, 7, 2, 0, 0),   # 2310, the largest that stays in the block
    (11, 6, 3, 2, 5),   # 2475, the first level beyond it
    (9, 8, 4, 3, 1),
    (12, 8, 2, 1, 0),   # 5072
    (12, 8, 2, 0, 0),   # 5092
    (8, 8, -1, 0, 1),
]


@pytest.mark.parametrize("sec", SECTORS, ids=str)
def test_representatives_and_periods(sec):
    import blqh_gb300 as B
    from oracle import oracle as O

    b, o = B.Basis(*sec), O.Basis(*sec)
    assert b.dim == o.dim
    assert np.array_equal(b.id, o.id)
    assert np.array_equal(b.period, o.period)
