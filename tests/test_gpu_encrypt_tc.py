"""Encryption on the tensor cores against the oracle: every n1, row counts
around its tiles of 16 rows and past one pass, extreme residues; and the staged
copies that carry it (more chunks than slots, the first bad residue named)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from bnutil import N, P, uniform_fp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n1", [(1, 128), (15, 64), (17, 512), (300, 256), (1301, 128), (8209, 64)])
def test_encrypt_matches_oracle(ctx, m, n1):
    from bn_b200 import capi as c

    M = uniform_fp((m, N), m + n1)
    M[0] = P - 1
    L = O.generate_subspace(bytes([2]) * 32, n1=n1)
    cl = O.encrypt_cluster(M.reshape(-1), m, L, O.derive_h_seed(11, 0), n1=n1)
    m_enc, al = c.encrypt_cluster(ctx, M.reshape(-1), m, L, cl.h_mat, cl.s_mat.rowptr, cl.s_mat.idx, cl.s_mat.sign, n1)
    assert np.array_equal(al, cl.a_l.reshape(-1))
    assert np.array_equal(m_enc, cl.m_enc.reshape(-1))


def test_encrypt_without_room_for_the_scratch(ctx):
    """A budget that holds the results but not the tensor cores' scratch."""
    from bn_b200 import capi as c

    m = 4000
    M = uniform_fp((m, N), 5)
    L = O.generate_subspace(bytes([2]) * 32)
    cl = O.encrypt_cluster(M.reshape(-1), m, L, O.derive_h_seed(11, 0))
    need = 2 * m * N * 8 + 2 * m * 128 * 8 + 2 * N * 128 * 8 + (m + 1) * 8 + 5 * cl.s_mat.idx.size
    small = c.Context(0, need + (1 << 20))
    m_enc, al = c.encrypt_cluster(small, M.reshape(-1), m, L, cl.h_mat, cl.s_mat.rowptr, cl.s_mat.idx, cl.s_mat.sign)
    assert np.array_equal(al, cl.a_l.reshape(-1)) and np.array_equal(m_enc, cl.m_enc.reshape(-1))
    small.close()


@pytest.mark.parametrize("at", [0, 70000, 1200 * N - 1])
def test_the_first_bad_residue_is_named(ctx, at):
    from bn_b200 import capi as c

    m = 1200
    M = uniform_fp((m, N), 6).reshape(-1)
    M[at] = P if at else 2**64 - 1
    M[min(at + 100000, M.size - 1)] = max(int(M[min(at + 100000, M.size - 1)]), P)
    L = O.generate_subspace(bytes([2]) * 32)
    with pytest.raises(c.BnError, match=rf"m_q\[{at}\]"):
        c.Flat.build_keygen(ctx, M, m, L, bytes(32))
