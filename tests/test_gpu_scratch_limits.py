"""Calls in contexts and servers whose budget leaves room for z panels of 4096 rows,
a candidate list per eight decode units and u . r sums per 2048 list rows, but not for
the shorter ones that the schedules prefer: they are answered, with the same results.

ROOM holds the workspace of each call with the former, as the library allocated it
when it knew no others."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from bnutil import N, int8_matrix, uniform_fp

pytestmark = pytest.mark.gpu

M_FLAT = 1500
SIZES = [2600, 40, 5000, 300]
ROOM = {"query": 8957952, "verify": 1084928, "block": 758272, "verify_block": 654592, "ivf": 3392000,
        "ivf_block": 4295872, "ivf_verify_block": 2731520}
SERVER_ROOM = {"flat": 1170176, "flat_block": 1299712, "ivf": 3392000}


def _queries(L, B):
    encs = [O.encode_query(int8_matrix(1, 768, 300 + b)[0], L, O.derive_h_seed(301, b)) for b in range(B)]
    return (np.stack([e.v_enc for e in encs]), np.stack([e.g for e in encs]), [(e.t_idx, e.t_sign) for e in encs],
            [bytes([b + 1]) * 32 for b in range(B)])


class Case:
    """Handles in a context of their own; calls by name."""

    def __init__(self, budget=0):
        from bn_b200 import capi as c

        self.c, self.ctx = c, c.Context(0, vram_budget_bytes=budget)
        self.L = O.generate_subspace(bytes([3]) * 32)
        self.q = _queries(self.L, 8)
        x = int8_matrix(M_FLAT, 768, 310)
        self.flat = c.Flat.build_keygen(self.ctx, x.reshape(-1), M_FLAT, self.L, bytes([4]) * 32)
        self.flat.block_prepare()
        off = np.concatenate([[0], np.cumsum(SIZES)]).astype(np.uint64)
        rows = int(off[-1])
        y = int8_matrix(rows, 768, 311)
        self.ivf = c.Ivf.build_keygen(self.ctx, off, np.arange(rows, dtype=np.uint32), y.reshape(-1), self.L, 5)
        self.ivf.block_prepare()
        self.probes = np.array([[0, 2], [2, 1], [2, 3], [0, 3]] * 2, np.uint32)
        self.r = uniform_fp((8, M_FLAT), 312)
        self.ri = uniform_fp((sum(p[2] for p in self.ivf.pairs(self.probes)),), 313)
        self.keep = []

    def call(self, name):
        v, g, t, sd = self.q
        f, i = self.flat, self.ivf
        if name == "query":
            hits, fl, _, _ = f.query(v, g, t, sd, 40, 1000)
        elif name == "verify":
            return list(f.verify(self.r[0], v[0], sd[0], 40))
        elif name == "block":
            hits, fl, _ = f.query_block(v[:2], g[:2], t[:2], sd[0], 20, 10)
        elif name == "verify_block":
            return list(f.verify_block(self.r[:2], v[:2], sd[0], 20))
        elif name == "ivf":
            hits, fl, _ = i.query(self.probes[:1], v[:1], g[:1], t[:1], sd[:1], 20, 30)
        elif name == "ivf_block":
            hits, fl, _ = i.query_block(self.probes, v, g, t, sd[0], 20, 10)
        else:
            return list(i.verify_block(self.probes, self.ri, v, sd[0], 20))
        return [x for h in hits for x in h] + [fl]

    def left(self):
        budget, used, _ = self.ctx.memory()
        return budget - used

    def fill(self, room):
        """Holds memory until about `room` bytes are left of the budget (a little more)."""
        for B, k in ((8, 1024), (8, 100), (1, 1)):
            before = self.left()
            first = self.flat.plan(B, 0, k)
            step = before - self.left()
            first.close()
            while self.left() - step >= room:
                self.keep.append(self.flat.plan(B, 0, k))

    def close(self):
        for p in self.keep:
            p.close()
        self.flat.close()
        self.ivf.close()
        self.ctx.close()


@pytest.fixture(scope="module")
def ample():
    case = Case()
    yield case
    case.close()


NAMES = ["query", "verify", "block", "verify_block", "ivf", "ivf_block", "ivf_verify_block"]


@pytest.mark.parametrize("name", NAMES)
def test_call_at_its_scratch_limit(ample, name):
    want = ample.call(name)
    peak = ample.ctx.memory()[2]
    tight = Case(budget=peak + (64 << 20))
    tight.fill(ROOM[name])
    assert ROOM[name] <= tight.left() < ROOM[name] + (96 << 10)
    got = tight.call(name)
    assert len(got) == len(want) and all(np.array_equal(a, b) for a, b in zip(got, want))
    tight.close()


@pytest.mark.parametrize("kind", list(SERVER_ROOM))
def test_server_at_its_budget(ample, kind):
    """mem_budget as small as one request's (or one block of eight's) workspace."""
    c, (v, g, t, sd) = ample.c, ample.q
    room = SERVER_ROOM[kind]
    if kind == "flat":
        n, trials, k, block_min = 1, 40, 1024, 0
        want = ample.flat.query(v[:1], g[:1], t[:1], sd[:1], trials, k)[0]
    elif kind == "ivf":
        n, trials, k, block_min = 1, 20, 30, 0
        want = ample.ivf.query(ample.probes[:1], v[:1], g[:1], t[:1], sd[:1], trials, k)[0]
    else:
        n, trials, k, block_min = 8, 20, 10, 8
        want = ample.flat.query(v, g, t, sd, trials, k)[0]
    srv = c.Server(ample.flat, ample.ivf, max_batch=8, slots=1, mem_budget=room, max_wait_us=200000 if n > 1 else 0,
                   trials=trials, k=k, block_min=block_min)
    if kind == "ivf":
        tickets = [srv.submit_ivf(ample.probes[0], v[0], g[0], *t[0], sd[0])]
    else:
        tickets = [srv.submit_flat(v[b], g[b], *t[b], sd[b]) for b in range(n)]
    for ticket, (ids, sc) in zip(tickets, want):
        got = srv.wait(ticket)
        assert np.array_equal(got[0], ids) and np.array_equal(got[1], sc) and got[2] == -1
    st = srv.stats()
    assert st["peak_workspace_bytes"] <= room and st["block_batches"] == (1 if kind == "flat_block" else 0)
    srv.close()
