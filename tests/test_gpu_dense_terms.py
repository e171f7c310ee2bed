"""AL g + H x by itself: the column shares of every n1, rows on both sides of a
block of 32 and of one round of CTAs, the largest residues; against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from bnutil import N, P, uniform_fp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n1,top", [(1, 64, False), (31, 512, True), (33, 256, False), (4737, 512, False),
                                      (18945, 128, True), (60001, 64, False)])
def test_dense_terms(ctx, m, n1, top):
    from bn_b200 import capi as c

    make = (lambda shape, seed: np.full(shape, P - 1, np.uint64)) if top else uniform_fp
    al, h, g, x = make((m, n1), 31), make((m, n1), 32), make(n1, 33), make(n1, 34)
    f = c.Flat.build(ctx, np.zeros((m, N), np.uint64), al, h, m, n1=n1)
    want = (O.matvec(al, m, n1, g).astype(object) + O.matvec(h, m, n1, x).astype(object)) % P
    assert np.array_equal(f.decode_dense_terms(g, x), want.astype(np.uint64))
    f.close()
