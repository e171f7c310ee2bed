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


def test_first_calls_of_a_new_thread(ctx):
    """A thread that has made no CUDA call yet, over handles that need no new memory."""
    import threading

    from bn_b200 import capi as c
    from bnutil import int8_matrix

    m, B = 2000, 2
    L = O.generate_subspace(bytes([3]) * 32)
    x = int8_matrix(m, 768, 48)
    f = c.Flat.build_keygen(ctx, x.reshape(-1), m, L, bytes([4]) * 32)
    off = np.array([0, 900, m], np.uint64)
    v = c.Ivf.build_keygen(ctx, off, np.arange(m, dtype=np.uint32), x.reshape(-1), L, 5)
    v.block_prepare()
    encs = [O.encode_query(int8_matrix(1, 768, 49 + b)[0], L, O.derive_h_seed(50, b)) for b in range(B)]
    q = (np.stack([e.v_enc for e in encs]), np.stack([e.g for e in encs]), [(e.t_idx, e.t_sign) for e in encs])
    seeds = [bytes([b]) * 32 for b in range(B)]
    probes = np.array([[0, 1], [1, 0]], np.uint32)
    r = f.compute_products_batch(q[0])
    calls = {
        "query": lambda: f.query(*q, seeds, 3, 5)[:2],
        "verify": lambda: f.verify(r[0], q[0][0], seeds[0], 3),
        "products": lambda: f.compute_products(q[0][0]),
        "dense": lambda: f.decode_dense_terms(q[1][0], q[1][1]),
        "list dense": lambda: v.decode_dense_terms(1, q[1][0], q[1][1]),
        "block": lambda: f.query_block(*q, seeds[0], 3, 5)[:2],
        "verify_block": lambda: f.verify_block(r, q[0], seeds[0], 3),
        "ivf": lambda: v.query(probes, *q, seeds, 3, 5),
        "ivf_block": lambda: v.query_block(probes, *q, seeds[0], 3, 5),
    }
    got = {}
    flat = lambda y: [z for w in y for z in flat(w)] if isinstance(y, (list, tuple)) else [y]  # noqa: E731
    for name, call in calls.items():
        want = call()
        t = threading.Thread(target=lambda: got.update({name: call()}))
        t.start()
        t.join()
        assert name in got, name  # the call raised
        assert all(np.array_equal(a, b) for a, b in zip(flat(got[name]), flat(want))), name
    f.close()
    v.close()
