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
