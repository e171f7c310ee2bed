"""Host copies and checks beside the kernels: the threads that share them stay the
same from call to call."""
from __future__ import annotations

import os

import numpy as np
import pytest

import oracle as O
from bnutil import N, uniform_fp

pytestmark = pytest.mark.gpu


def _threads():
    return set(os.listdir("/proc/self/task"))


def test_calls_do_not_make_threads(ctx):
    """Checks and copies of different sizes in turn: after the first round no call
    ends or makes a thread (a team of another size each time did)."""
    from bn_b200 import capi as c

    m = 9001
    m_enc = uniform_fp((m, N), 41)
    f = c.Flat.build(ctx, m_enc, np.zeros(m * 128, np.uint64), np.zeros(m * 128, np.uint64), m)
    v = uniform_fp((48, N), 42)
    want = O.matvec_batch(m_enc, m, N, v[:2])
    seen = None
    for turn in range(4):
        r = f.compute_products_batch(v[:20])  # 1.4 MB down
        assert np.array_equal(r[:2], want)
        fl, _, _ = f.verify_block(r, v[:20], bytes([3]) * 32, 2)  # checks 1.4 MB and 160 KB
        assert (fl == -1).all()
        assert np.array_equal(f.compute_products_batch(v)[:2], want)  # 3.4 MB down, checks 384 KB
        assert f.verify(r[0], v[0], bytes([3]) * 32, 2)[0] == -1
        if turn >= 1:
            assert seen is None or _threads() == seen
            seen = _threads()
    f.close()
