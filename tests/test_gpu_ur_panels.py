"""u . r of a block over K panels sized by the number of queries and rows: one
panel, a short last one, several tiles of queries; honest responses and one
changed in its last row, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from bnutil import N, P, uniform_fp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,B,trials", [(1, 1, 20), (512, 3, 20), (513, 17, 3), (9001, 1, 20), (9001, 130, 23)])
def test_block_verify_panels(ctx, m, B, trials):
    from bn_b200 import capi as c

    m_enc = uniform_fp((m, N), 900 + m)
    f = c.Flat.build(ctx, m_enc, np.zeros(m * 128, np.uint64), np.zeros(m * 128, np.uint64), m)
    v = uniform_fp((B, N), 901 + B)
    r = O.matvec_batch(m_enc, m, N, v)
    bad = B - 1
    r[bad, m - 1] = (int(r[bad, m - 1]) + 1) % P
    seed = bytes([36]) * 32
    fl, ur, zv = f.verify_block(r, v, seed, trials)
    assert fl[bad] == 0 and all(fl[b] == -1 for b in range(bad))
    for b in sorted({0, B // 2, bad}):
        fo, uro, zvo = O.verify_response(r[b], m_enc, m, N, v[b], trials, seed)
        ran = trials if fo < 0 else fo + 1
        assert fl[b] == fo and np.array_equal(ur[:ran, b], uro) and np.array_equal(zv[:ran, b], zvo)
    f.close()
