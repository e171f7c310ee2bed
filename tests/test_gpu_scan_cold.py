"""The scan right after a corpus is copied to the device: its first pass meets
cold pages, so the copies into the ring finish out of order.  Every residue
against the oracle, twice per corpus."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from bnutil import N, uniform_fp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [50001, 61440, 30003])
def test_first_scan_of_a_corpus(ctx, m):
    from bn_b200 import capi as c

    m_enc = uniform_fp((m, N), m)
    f = c.Flat.build(ctx, m_enc, np.zeros(m * 128, np.uint64), np.zeros(m * 128, np.uint64), m)
    for s in (1, 2):
        v = uniform_fp((N,), m + s)
        assert np.array_equal(f.compute_products(v), O.matvec(m_enc, m, N, v))
    f.close()
