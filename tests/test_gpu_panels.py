"""Protocol 2 panels chosen by the row count: one block, a few, ragged last
panels, panels of more than 4096 rows, several queries per call; every trial's
pair of sums against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from bnutil import N, P, uniform_fp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,trials", [(1, 3), (129, 20), (4999, 3), (20011, 20), (50001, 5)])
def test_verify_sums(ctx, m, trials):
    from bn_b200 import capi as c

    m_enc = uniform_fp((m, N), m)
    f = c.Flat.build(ctx, m_enc, np.zeros(m * 128, np.uint64), np.zeros(m * 128, np.uint64), m)
    v = uniform_fp((N,), m + 1)
    r = O.matvec(m_enc, m, N, v)
    assert np.array_equal(f.compute_products(v), r)
    seed = bytes([m % 256]) * 32
    for last in (0, 1):
        r2 = r.copy()
        r2[m - 1] = (r2[m - 1] + np.uint64(last)) % np.uint64(P)
        got, ur, zv = f.verify(r2, v, seed, trials)
        want, uo, zo = O.verify_response(r2, m_enc, m, N, v, trials, seed)
        assert got == want and np.array_equal(ur, uo) and np.array_equal(zv, zo)
    f.close()
