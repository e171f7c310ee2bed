"""Protocol 2 over many short lists: the strip runs a panel is split into (1,
2, 4 or 8) and the verdicts of many single-panel segments."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from bnutil import N, P, int8_matrix
from ivfutil import IvfCase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlist,trials", [(148, 3), (70, 20), (160, 21), (12, 20)])
def test_short_lists_verdicts(ctx, nlist, trials):
    from bn_b200 import capi as c

    rng = np.random.default_rng(nlist)
    case = IvfCase([int(x) for x in rng.integers(1, 4, nlist)], seed=nlist)
    m_enc, a_l, h, rp, ix, sg = case.concat()
    v = c.Ivf.build(ctx, case.offsets, case.ids, m_enc, a_l, h)
    probes = np.stack([rng.permutation(nlist) for _ in range(2)]).astype(np.uint32)
    encs = [O.encode_query(int8_matrix(1, 768, 30 + b)[0], case.L, O.derive_h_seed(31, b)) for b in range(2)]
    seed = bytes([nlist % 256]) * 32
    r = [O.matvec(case.clusters[ci].m_enc, case.clusters[ci].m, N, encs[q].v_enc) for q, ci, _ in v.pairs(probes)]
    bad = 3 * nlist // 4  # one pair of the first query answers wrongly
    r[bad] = r[bad].copy()
    r[bad][0] = (r[bad][0] + np.uint64(1)) % np.uint64(P)
    fc, ft, ur, zv = v.verify_block(probes, np.concatenate(r), np.stack([e.v_enc for e in encs]), seed, trials)
    assert fc[0] == probes[0][bad] and ft[0] == 0 and fc[1] == ft[1] == -1
    for i, (q, ci, m) in enumerate(v.pairs(probes)):
        cl = case.clusters[ci]
        f, u, z = O.verify_response(r[i], cl.m_enc, m, N, encs[q].v_enc, trials, seed)
        ran = len(u)
        assert np.array_equal(ur[i][:ran], u) and np.array_equal(zv[i][:ran], z)
    v.close()
