"""Host copies and checks beside the kernels: the threads that share them stay the
same from call to call, and pinned arrays may be reused when a call returns."""
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


def _pinned(a):
    import torch

    return torch.from_numpy(a.view(np.int64)).pin_memory().numpy().view(np.uint64)


def test_pinned_arrays_are_free_on_return(ctx):
    """Pinned sources are copied asynchronously: the call has to wait for them."""
    from bn_b200 import capi as c

    m = 6000
    off = np.array([0, 2500, m], np.uint64)
    m_enc, a_l, h = uniform_fp((m, N), 43), uniform_fp((m, 128), 44), uniform_fp((m, 128), 45)
    v = uniform_fp((N,), 46)
    pins = [_pinned(x.reshape(-1)) for x in (m_enc, a_l, h)]
    ivf = c.Ivf.build(ctx, off, np.arange(m, dtype=np.uint32), *pins)
    flat = c.Flat.build(ctx, *[_pinned(x.reshape(-1)) for x in (m_enc, a_l, h)], m)
    for p in pins:
        p[:] = 0
    want = O.matvec(m_enc, m, N, v)
    assert np.array_equal(ivf.compute_products(1, v), want[2500:])
    g = uniform_fp((2, 128), 47)
    assert np.array_equal(ivf.decode_dense_terms(1, g[0], g[1]), flat.decode_dense_terms(g[0], g[1])[2500:])
    r = _pinned(np.tile(want, 1))
    for bad in (False, True):
        r[m - 1] = (int(want[m - 1]) + bad) % O.P
        assert flat.verify(r, v, bytes([5]) * 32, 3)[0] == (0 if bad else -1)
        r[:] = 1
        r[:] = want
    ivf.close()
    flat.close()
