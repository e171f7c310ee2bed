"""Top-k of the block paths on both sides of the warp-list kernels' k <= 32:
scores with many ties (score desc, id asc), row counts around the tile sizes,
and verdicts summed over many K panels."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from bnutil import N, P, int8_matrix
from ivfutil import IvfCase
from test_gpu_block import block_inputs, flat_from_cluster

pytestmark = pytest.mark.gpu


def ivf_build(ctx, case):
    from bn_b200 import capi as c

    m_enc, a_l, h, rp, ix, sg = case.concat()
    v = c.Ivf.build(ctx, case.offsets, case.ids, m_enc, a_l, h)
    v.attach_client(case.L, case.M.reshape(-1), rp, ix, sg)
    return v


@pytest.mark.parametrize("m", [31, 513, 4099])
@pytest.mark.parametrize("k", [1, 31, 32, 33])
def test_block_topk_with_ties(ctx, m, k):
    M = int8_matrix(7, 768, 40 + m)[np.arange(m) % 7].copy()  # seven distinct rows: every score is tied m / 7 times
    L = O.generate_subspace(bytes([8]) * 32)
    cl = O.encrypt_cluster(M.reshape(-1), m, L, O.derive_h_seed(3, 0))
    f = flat_from_cluster(ctx, M, L, cl)
    _, encs = block_inputs(L, 3, 50 + m)
    hits, failed, mv = f.query_block(np.stack([e.v_enc for e in encs]), np.stack([e.g for e in encs]),
                                     [(e.t_idx, e.t_sign) for e in encs], bytes([4]) * 32, 33, k, want_mv=True)
    for b, enc in enumerate(encs):
        r = O.matvec(cl.m_enc, m, N, enc.v_enc)
        assert np.array_equal(mv[b], O.decode_scores(r, cl, L, enc))
        ids, sc = O.topk(O.to_signed(mv[b]), k)
        assert np.array_equal(hits[b][0], ids) and np.array_equal(hits[b][1], sc)
        assert failed[b] == -1
    f.close()


@pytest.mark.parametrize("k", [1, 32, 33])
def test_ivf_block_topk_odd_ranges(ctx, k):
    """Odd first entries of a query's range, ranges shorter than a pair, and an empty one."""
    case = IvfCase([1, 3, 0, 300, 17, 1, 129], seed=9)
    v = ivf_build(ctx, case)
    probes = np.array([[0, 1], [3, 5], [2, 2], [6, 4]], np.uint32)
    encs = [O.encode_query(int8_matrix(1, 768, 70 + b)[0], case.L, O.derive_h_seed(71, b)) for b in range(4)]
    hits, fc, ft = v.query_block(probes, np.stack([e.v_enc for e in encs]), np.stack([e.g for e in encs]),
                                 [(e.t_idx, e.t_sign) for e in encs], bytes([6]) * 32, 3, k)
    for b, enc in enumerate(encs):
        ids, sc = case.oracle_score(probes[b], enc, bytes([6]) * 32, 0, k)
        assert np.array_equal(hits[b][0], ids) and np.array_equal(hits[b][1], sc)
        assert fc[b] == ft[b] == -1
    v.close()
