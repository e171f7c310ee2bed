"""Both forms of the decode, a unit (32-row block) per CTA and a unit per warp:
unit counts on both sides of the line between them, segments that start and end
inside a block, wide slices of S and repeated columns, T lists of any length,
int8 and residue plaintext, both top-k forms; against the oracle or the
plaintext products."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from bnutil import N, P, int8_matrix, uniform_fp
from ivfutil import IvfCase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n1,k,uniform", [(1, 128, 10, False), (31, 64, 33, False), (33, 128, 32, True),
                                            (4801, 128, 10, False), (4801, 64, 100, True), (2000, 256, 10, True),
                                            (9000, 128, 1, True), (30011, 128, 10, False), (10007, 64, 33, True)])
def test_decode_matches_oracle(ctx, m, n1, k, uniform):
    from bn_b200 import capi as c

    M = uniform_fp((m, N), 20 + m) if uniform else int8_matrix(m, 768, 20 + m)
    L = O.generate_subspace(bytes([9]) * 32, n1=n1)
    cl = O.encrypt_cluster(M.reshape(-1), m, L, O.derive_h_seed(2, 0), n1=n1)
    f = c.Flat.build(ctx, cl.m_enc, cl.a_l, cl.h_mat, m, n1=n1)
    f.attach_client(L, M.reshape(-1), cl.s_mat.rowptr, cl.s_mat.idx, cl.s_mat.sign)
    encs = [O.encode_query(int8_matrix(1, 768, 21 + b)[0], L, O.derive_h_seed(22, b), n1=n1) for b in range(3)]
    hits, failed, _, mv = f.query(np.stack([e.v_enc for e in encs]), np.stack([e.g for e in encs]),
                                  [(e.t_idx, e.t_sign) for e in encs], None, 0, k, want_mv=True)
    for b, enc in enumerate(encs):
        want = O.decode_scores(O.matvec(cl.m_enc, m, N, enc.v_enc), cl, L, enc)
        assert np.array_equal(mv[b], want)
        ids, sc = O.topk(O.to_signed(want), k)
        assert np.array_equal(hits[b][0], ids) and np.array_equal(hits[b][1], sc)
    f.close()


def test_wide_slices_and_repeated_columns(ctx):
    """Rows of S with up to 700 entries (slices of more than 256 column slots)
    and columns named twice, beside ordinary ones: the products come out plain."""
    from bn_b200 import capi as c

    rng = np.random.default_rng(3)
    m = 200
    M = int8_matrix(m, 768, 77)
    L = O.generate_subspace(bytes([9]) * 32)
    H = uniform_fp((m, 128), 78)
    width = np.where(np.arange(m) % 64 == 5, 700, 90)
    cols = [rng.integers(0, N, w).astype(np.uint32) for w in width]  # repeats happen
    signs = [rng.choice([-1, 1], w).astype(np.int8) for w in width]
    rp = np.concatenate([[0], np.cumsum(width)]).astype(np.uint64)
    f = c.Flat.build_from_plain(ctx, M.reshape(-1), m, L, H, rp, np.concatenate(cols), np.concatenate(signs))
    q = int8_matrix(1, 768, 79)[0]
    enc = O.encode_query(q, L, bytes([1]) * 32)
    hits, failed, r, mv = f.query(enc.v_enc[None], enc.g[None], [(enc.t_idx, enc.t_sign)], [bytes([2]) * 32], 3, 10,
                                  want_r=True, want_mv=True)
    assert failed[0] == -1
    want = O.matvec(M.reshape(-1), m, N, q)
    assert np.array_equal(mv[0], want)
    # r = (M + H L^T + S) v
    S = np.zeros((m, N), object)
    for i in range(m):
        np.add.at(S[i], cols[i], signs[i].astype(object))
    row = 5
    enc_row = (M[row].astype(object) + H[row].astype(object) @ L.reshape(N, 128).astype(object).T + S[row]) % P
    assert int(r[0][row]) == int(enc_row @ enc.v_enc.astype(object)) % P
    f.close()


@pytest.mark.parametrize("t_len", [0, 1, 200, 513])
def test_t_lists_of_any_length(ctx, t_len):
    from bn_b200 import capi as c

    m = 300
    M = int8_matrix(m, 768, 60)
    L = O.generate_subspace(bytes([9]) * 32)
    cl = O.encrypt_cluster(M.reshape(-1), m, L, O.derive_h_seed(2, 0))
    f = c.Flat.build(ctx, cl.m_enc, cl.a_l, cl.h_mat, m)
    f.attach_client(L, M.reshape(-1), cl.s_mat.rowptr, cl.s_mat.idx, cl.s_mat.sign)
    enc = O.encode_query(int8_matrix(1, 768, 61)[0], L, bytes([1]) * 32)
    rng = np.random.default_rng(t_len)
    ti = rng.integers(0, N, t_len).astype(np.uint32)
    ts = rng.choice([-1, 1], t_len).astype(np.int8)
    _, _, r, mv = f.query(enc.v_enc[None], enc.g[None], [(ti, ts)], None, 0, 5, want_r=True, want_mv=True)
    _, _, _, mv0 = f.query(enc.v_enc[None], enc.g[None], [(ti[:0], ts[:0])], None, 0, 5, want_mv=True)
    Ms = O.to_signed(M.reshape(-1)).reshape(m, N)
    mt = Ms[:, ti].astype(np.int64) @ ts.astype(np.int64) if t_len else np.zeros(m, np.int64)
    assert [int(x) for x in mv[0]] == [(int(a) - int(b)) % P for a, b in zip(mv0[0], mt)]
    f.close()


def test_ivf_segments_inside_blocks(ctx):
    """Lists that share 32-row blocks, a query count that the CTAs do not divide by."""
    from bn_b200 import capi as c

    case = IvfCase([5, 40, 0, 1, 33, 300, 31, 64, 7], seed=4)
    m_enc, a_l, h, rp, ix, sg = case.concat()
    v = c.Ivf.build(ctx, case.offsets, case.ids, m_enc, a_l, h)
    v.attach_client(case.L, case.M.reshape(-1), rp, ix, sg)
    rng = np.random.default_rng(8)
    B = 23
    probes = np.stack([rng.permutation(case.nlist)[:4] for _ in range(B)]).astype(np.uint32)
    encs = [O.encode_query(int8_matrix(1, 768, 90 + b)[0], case.L, O.derive_h_seed(91, b)) for b in range(B)]
    seeds = [bytes([b]) * 32 for b in range(B)]
    for k in (10, 40):
        hits, fc, ft = v.query(probes, np.stack([e.v_enc for e in encs]), np.stack([e.g for e in encs]),
                               [(e.t_idx, e.t_sign) for e in encs], seeds, 2, k)
        for b, enc in enumerate(encs):
            ids, sc = case.oracle_score(probes[b], enc, seeds[b], 2, k)
            assert np.array_equal(hits[b][0], ids) and np.array_equal(hits[b][1], sc)
            assert fc[b] == ft[b] == -1
    v.close()


@pytest.mark.parametrize("m,k", [(300, 100), (1024, 256), (1024, 257), (1025, 256), (6001, 1000)])
def test_large_k(ctx, m, k):
    """k > 32 on both sides of the line between the forms: the oracle's hits, and a
    candidate list per eight units only (a list per unit cost more to merge than the
    whole decode) where a query has more than 32 units or k is above 256."""
    from bn_b200 import capi as c

    M = int8_matrix(m, 768, 30 + m)
    L = O.generate_subspace(bytes([9]) * 32)
    cl = O.encrypt_cluster(M.reshape(-1), m, L, O.derive_h_seed(2, 0))
    f = c.Flat.build(ctx, cl.m_enc, cl.a_l, cl.h_mat, m)
    f.attach_client(L, M.reshape(-1), cl.s_mat.rowptr, cl.s_mat.idx, cl.s_mat.sign)
    encs = [O.encode_query(int8_matrix(1, 768, 31 + b)[0], L, O.derive_h_seed(22, b)) for b in range(2)]
    hits, failed, _, mv = f.query(np.stack([e.v_enc for e in encs]), np.stack([e.g for e in encs]),
                                  [(e.t_idx, e.t_sign) for e in encs], None, 0, k, want_mv=True)
    for b, enc in enumerate(encs):
        want = O.decode_scores(O.matvec(cl.m_enc, m, N, enc.v_enc), cl, L, enc)
        assert np.array_equal(mv[b], want)
        ids, sc = O.topk(O.to_signed(want), k)
        assert np.array_equal(hits[b][0], ids) and np.array_equal(hits[b][1], sc)
    used = ctx.memory()[1]
    plan = f.plan(1, 0, k)
    grown = ctx.memory()[1] - used
    plan.close()
    units = (m + 31) // 32
    lists = units if units <= 32 and k <= 256 else (units + 7) // 8
    # beside the lists: r (8 m) and the query's own arrays (below 64 KB)
    assert grown <= 12 * k * lists + 16 * m + (64 << 10), (grown, lists)
    f.close()


@pytest.mark.parametrize("trials", [0, 3])
def test_decoded_residues_without_hits(ctx, trials):
    """k = 0 with the decoded residues asked for: those, and no hits."""
    from bn_b200 import capi as c

    m = 700
    M = int8_matrix(m, 768, 40)
    L = O.generate_subspace(bytes([9]) * 32)
    cl = O.encrypt_cluster(M.reshape(-1), m, L, O.derive_h_seed(2, 0))
    f = c.Flat.build(ctx, cl.m_enc, cl.a_l, cl.h_mat, m)
    f.attach_client(L, M.reshape(-1), cl.s_mat.rowptr, cl.s_mat.idx, cl.s_mat.sign)
    for turn in range(2):  # the second run would find the first one's in its workspace
        encs = [O.encode_query(int8_matrix(1, 768, 41 + 3 * turn + b)[0], L, O.derive_h_seed(42, b)) for b in range(3)]
        hits, failed, _, mv = f.query(np.stack([e.v_enc for e in encs]), np.stack([e.g for e in encs]),
                                      [(e.t_idx, e.t_sign) for e in encs], [bytes([b]) * 32 for b in range(3)], trials, 0,
                                      want_mv=True)
        for b, enc in enumerate(encs):
            assert len(hits[b][0]) == 0 and failed[b] == -1
            assert np.array_equal(mv[b], O.decode_scores(O.matvec(cl.m_enc, m, N, enc.v_enc), cl, L, enc))
    f.close()
