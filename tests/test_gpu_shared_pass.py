"""Several queries in one pass over the corpus (few trials each): groups of every
size, a smaller last group, rows, query counts and trials on both sides of the line; hits, products and both sums of every trial against the
oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from bnutil import N, cluster
from test_gpu_block import block_inputs, flat_from_cluster

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,B,trials", [(1, 2, 3), (1920, 4, 3), (1921, 4, 3), (5000, 5, 3), (2100, 17, 1), (2000, 3, 9),
                                        (3000, 2, 10), (1990, 5, 5), (2049, 13, 2), (12001, 4, 4), (2500, 3, 6)])
def test_shared_pass_matches_oracle(ctx, m, B, trials):
    M, L, cl = cluster(m, 90 + m + B)
    f = flat_from_cluster(ctx, M, L, cl)
    vs, encs = block_inputs(L, B, 91 + m)
    seeds = [bytes([m % 251, b]) * 16 for b in range(B)]
    v, g = np.stack([e.v_enc for e in encs]), np.stack([e.g for e in encs])
    t = [(e.t_idx, e.t_sign) for e in encs]
    hits, failed, r, _ = f.query(v, g, t, seeds, trials, 10, want_r=True)
    sh_hits, ur, zv = f.query_shard(v, g, t, seeds, trials, 10, 0, m)
    for b, e in enumerate(encs):
        want = O.matvec(cl.m_enc, m, N, e.v_enc)
        assert np.array_equal(r[b], want), b
        ids, sc = O.topk(O.to_signed(O.decode_scores(want, cl, L, e)), 10)
        for h in (hits[b], sh_hits[b]):
            assert np.array_equal(h[0], ids) and np.array_equal(h[1], sc), b
        fo, uo, zo = O.verify_response(want, cl.m_enc, m, N, e.v_enc, trials, seeds[b])
        assert failed[b] == fo == -1
        assert np.array_equal(ur[b], uo) and np.array_equal(zv[b], zo), b
    f.close()


def test_shared_pass_on_shards_with_an_offset(ctx):
    """Two shards of one corpus, whose draws start inside the whole corpus's: the sums
    of both shards' sides are the oracle's for the whole."""
    from bn_b200 import shard
    from test_shard import shard_cluster

    from bn_b200 import capi as c

    m, cut, B, trials = 5003, 2001, 4, 4
    M, L, cl = cluster(m, 97)
    vs, encs = block_inputs(L, B, 98)
    seeds = [bytes([m % 251, b]) * 16 for b in range(B)]
    args = (np.stack([e.v_enc for e in encs]), np.stack([e.g for e in encs]), [(e.t_idx, e.t_sign) for e in encs], seeds)
    parts = []
    for a, b in ((0, cut), (cut, m)):
        sub = shard_cluster(cl, a, b)
        f = c.Flat.build(ctx, sub.m_enc, sub.a_l, sub.h_mat, b - a)
        f.attach_client(L, sub.m_plain, sub.s_mat.rowptr, sub.s_mat.idx, sub.s_mat.sign)
        parts.append(f.query_shard(*args, trials, 10, a, m))
        f.close()
    for b, e in enumerate(encs):
        r = O.matvec(cl.m_enc, m, N, e.v_enc)
        fo, uo, zo = O.verify_response(r, cl.m_enc, m, N, e.v_enc, trials, seeds[b])
        failed, ur, zv = shard.combine_protocol2([p[1][b] for p in parts], [p[2][b] for p in parts])
        assert failed == fo == -1 and np.array_equal(ur, uo) and np.array_equal(zv, zo)
        ids, sc = O.topk(O.to_signed(O.decode_scores(r, cl, L, e)), 10)
        got = shard.merge_topk([p[0][b] for p in parts], 10)
        assert np.array_equal(got[0], ids) and np.array_equal(got[1], sc)


@pytest.mark.parametrize("B,trials", [(1, 20), (4, 3), (2, 23)])
def test_plans_back_to_back_on_two_streams(ctx, B, trials):
    """Runs of a plan follow one another without a wait, on each of two streams, with
    other inputs and seeds every time: nothing of a run is taken by the next."""
    import torch

    m, k = 3000, 10
    M, L, cl = cluster(m, 95)
    f = flat_from_cluster(ctx, M, L, cl)
    sets, want = [], []
    for i in range(5):
        vs, encs = block_inputs(L, B, 200 + 10 * i)
        seeds = [bytes([i + 1, b]) * 16 for b in range(B)]
        t, nnz = np.zeros((B, N), np.uint32), np.zeros(B, np.uint32)
        for b, e in enumerate(encs):
            nnz[b] = e.t_idx.size
            t[b, : nnz[b]] = e.t_idx | np.where(e.t_sign < 0, np.uint32(0x80000000), np.uint32(0))
        host = [np.stack([e.v_enc for e in encs]), np.stack([e.g for e in encs]), t, nnz,
                np.frombuffer(b"".join(seeds), np.uint8).copy()]
        ty = [np.int64, np.int64, np.int32, np.int32, np.uint8]
        sets.append([torch.from_numpy(a.view(y)).cuda() for a, y in zip(host, ty)])
        want.append([O.topk(O.to_signed(O.decode_scores(O.matvec(cl.m_enc, m, N, e.v_enc), cl, L, e)), k) for e in encs])
    plans, streams, runs = [f.plan(B, trials, k) for _ in range(2)], [torch.cuda.Stream() for _ in range(2)], []
    outs = [[torch.zeros((B, k), dtype=torch.int32, device="cuda"), torch.zeros((B, k), dtype=torch.int64, device="cuda"),
             torch.zeros(B, dtype=torch.int32, device="cuda"), torch.full((B,), 7, dtype=torch.int32, device="cuda")]
            for _ in range(20)]
    torch.cuda.synchronize()
    for n in range(20):
        i, w = (3 * n) % 5, n % 2
        plans[w].enqueue(*[x.data_ptr() for x in sets[i]], *[x.data_ptr() for x in outs[n]], streams[w].cuda_stream)
        runs.append(i)
    torch.cuda.synchronize()
    for i, (ids, sc, cnt, failed) in zip(runs, outs):
        assert (failed.cpu().numpy() == -1).all() and (cnt.cpu().numpy() == k).all()
        for b in range(B):
            assert np.array_equal(ids[b].cpu().numpy().view(np.uint32), want[i][b][0])
            assert np.array_equal(sc[b].cpu().numpy(), want[i][b][1])
    for p in plans:
        assert p.status() == 0
        p.close()
    f.close()
