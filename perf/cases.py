"""The work that users of this backend have it do, as cases that can be timed.

Every case is one call (or the two calls that belong together) of the public
Python API (bn_b200.capi) on a corpus that is already resident: a client or a
search service builds the encrypted corpus once and then sends queries to it.
The exception is the upload itself, which is a case of its own.

listed() gives the cases, draw(rng) another one of the same ranges,
prepare(case, seed) what the caller has in hand (handles, plans, encoded
queries), run(state) one pass, work(case) the bytes and operations a pass
cannot do without, exact(case, seed) the ranked plaintext products.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "secure-vector-search_b200"))

from bn_b200 import capi  # noqa: E402

N = capi.N  # padded dimension of the scheme
P = capi.P
N1 = 128  # the default secret dimension (delta = 3/10)
Q20 = 1 << 20  # the reference's default quantisation of f32 embeddings
DEV = "cuda:0"


def listed():
    return [
        # a small collection (one user's documents), one query at the
        # reference's default 3 Freivalds trials: latency and launches
        {"name": "flat_5k", "kind": "query", "rows": 5000, "d": 384, "data": "int8", "B": 1, "trials": 3, "k": 10},
        # the reference's own CPU benchmark size: 100k passages of a
        # 384-dimensional encoder, full 20 trials
        {"name": "flat_100k", "kind": "query", "rows": 100000, "d": 384, "data": "int8", "B": 1, "trials": 20, "k": 10},
        # the headline: a million 768-dimensional passages, one query
        {"name": "flat_1m", "kind": "query", "rows": 1000000, "d": 768, "data": "int8", "B": 1, "trials": 20, "k": 10},
        # embeddings quantised with the reference's default Q = 2^20 (not
        # int8-valued), a few queries with seeds of their own, a longer list
        {"name": "flat_q20", "kind": "query", "rows": 100003, "d": 768, "data": "q20", "B": 4, "trials": 3, "k": 100},
        # the server's half of a split deployment: r = M_enc v, sent to the client
        {"name": "products_150k", "kind": "products", "rows": 150001, "d": 768, "data": "int8", "B": 1},
        # the client's half: check the received r, then the dense terms of its decoding
        {"name": "client_150k", "kind": "client", "rows": 150001, "d": 768, "data": "int8", "B": 1, "trials": 20},
        # a service that batches a few requests (device buffers, a plan kept)
        {"name": "block_8", "kind": "block_plan", "rows": 200000, "d": 768, "data": "int8", "B": 8, "trials": 20, "k": 10},
        # offline scoring of many queries at once (device buffers, a plan kept)
        {"name": "block_512", "kind": "block_plan", "rows": 200000, "d": 768, "data": "int8", "B": 512, "trials": 20, "k": 10},
        # inverted lists, every query verified with its own seed
        {"name": "ivf_16x8", "kind": "ivf", "rows": 200000, "nlist": 400, "d": 768, "B": 16, "nprobe": 8, "trials": 20, "k": 10},
        # inverted lists, a server's batch of 64 with one verification seed: narrow and wide probes
        {"name": "ivf_block_64x8", "kind": "ivf_block", "rows": 327680, "nlist": 640, "d": 768, "B": 64, "nprobe": 8, "trials": 20, "k": 10},
        {"name": "ivf_block_64x64", "kind": "ivf_block", "rows": 327680, "nlist": 640, "d": 768, "B": 64, "nprobe": 64, "trials": 20, "k": 10},
        # the upload of one cluster: encrypt 4096 rows (host arrays in, host arrays out)
        {"name": "encrypt_4k", "kind": "encrypt", "rows": 4096, "d": 768, "data": "int8"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "query", "products", "client", "block_plan", "block_plan", "block", "ivf",
                       "ivf_block", "ivf_block", "encrypt"])
    d = rng.choice([384, 768])
    if kind == "query":
        rows, B = _log(rng, 2000, 400000), rng.choice([1, 1, 1, 2, 4])
        return {"kind": kind, "rows": max(rows // B, 500), "d": d, "data": rng.choice(["int8", "int8", "q20"]), "B": B,
                "trials": rng.choice([3, 20]), "k": rng.choice([10, 10, 100])}
    if kind in ("products", "client"):
        c = {"kind": kind, "rows": _log(rng, 5000, 200000), "d": d, "data": "int8", "B": 1}
        if kind == "client":
            c["trials"] = rng.choice([3, 20])
        return c
    if kind in ("block_plan", "block"):
        return {"kind": kind, "rows": _log(rng, 20000, 200000), "d": d, "data": "int8", "B": _log(rng, 2, 512),
                "trials": 20, "k": 10}
    if kind in ("ivf", "ivf_block"):
        rows = _log(rng, 60000, 327680)
        return {"kind": kind, "rows": rows, "nlist": max(64, rows // rng.choice([400, 512, 700])), "d": d,
                "B": rng.choice([1, 5, 16]) if kind == "ivf" else _log(rng, 8, 64),
                "nprobe": rng.choice([8, 16]) if kind == "ivf" else rng.choice([8, 32, 64]), "trials": 20, "k": 10}
    return {"kind": kind, "rows": _log(rng, 300, 6000), "d": d, "data": "int8"}


# ------------------------------------------------------------------ inputs
def _gen(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt) % (1 << 62))
    return g


def _unit(x):
    return x / x.norm(dim=1, keepdim=True).clamp_min(1e-12)


def _quantise(x, data):
    """Unit rows -> integers: int8 by per-row max-abs scaling, or round(x Q)."""
    x = _unit(x)
    if data == "q20":
        return torch.round(x * Q20).to(torch.int32)
    s = 127.0 / x.abs().amax(dim=1, keepdim=True).clamp_min(1e-12)
    return torch.clamp(torch.round(x * s), -127, 127).to(torch.int8)


def _vectors(rows, d, seed, salt, data):
    """Gaussian embeddings, normalised and quantised, on the GPU."""
    g = _gen(seed, salt)
    out = torch.empty((rows, d), dtype=torch.int32 if data == "q20" else torch.int8, device=DEV)
    for r0 in range(0, rows, 131072):
        r1 = min(rows, r0 + 131072)
        out[r0:r1] = _quantise(torch.randn((r1 - r0, d), generator=g, device=DEV), data)
    return out


def _residues(x):
    """Integer rows -> canonical residues mod p, zero-padded to N columns (host)."""
    x = x.cpu()
    out = np.zeros((x.shape[0], N), np.uint64)
    o = torch.from_numpy(out.view(np.int64))
    for r0 in range(0, x.shape[0], 65536):
        v = x[r0 : r0 + 65536].to(torch.int64)
        o[r0 : r0 + 65536, : x.shape[1]] = torch.where(v < 0, v + P, v)
    return out


def _seed32(seed, salt):
    return np.random.default_rng([int(seed), salt]).bytes(32)


def _mixture(case, seed):
    """Clustered embeddings: list sizes of a skewed partition, rows grouped by
    list, the lists' centroids, and queries near rows of the mixture."""
    rows, nlist, d = case["rows"], case["nlist"], case["d"]
    rng = np.random.default_rng([int(seed), 7])
    w = rng.lognormal(0.0, 0.8, nlist)
    sizes = rng.multinomial(rows, w / w.sum())
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    g = _gen(seed, 8)
    centres = _unit(torch.randn((nlist, d), generator=g, device=DEV))
    member = torch.from_numpy(np.repeat(np.arange(nlist), sizes)).to(DEV)
    x8 = torch.empty((rows, d), dtype=torch.int8, device=DEV)
    for r0 in range(0, rows, 131072):
        m = member[r0 : r0 + 131072]
        x8[r0 : r0 + 131072] = _quantise(
            centres[m] + (0.6 / math.sqrt(d)) * torch.randn((len(m), d), generator=g, device=DEV), "int8")
    pick = member[torch.randint(rows, (case["B"],), generator=g, device=DEV)]
    q8 = _quantise(centres[pick] + (0.6 / math.sqrt(d)) * torch.randn((case["B"], d), generator=g, device=DEV), "int8")
    cent = torch.zeros((nlist, d), dtype=torch.float32, device=DEV).index_add_(0, member, x8.to(torch.float32))
    cent /= torch.bincount(member, minlength=nlist).clamp_min(1)[:, None]
    ids = rng.permutation(rows).astype(np.uint32)
    return {"x": x8, "q": q8, "offsets": offsets, "ids": ids, "centroids": cent.cpu().numpy()}


def _encode(q, L, seed):
    """The client's encoded queries: v_enc, g, T, and each query's Protocol 2 seed."""
    vq = _residues(q)
    enc, seeds = [], []
    for i in range(vq.shape[0]):
        qs = _seed32(seed, 100 + i)
        enc.append(capi.host_encode_query(vq[i], L, qs))
        seeds.append(capi.host_domain_separate(qs))
    return (np.stack([e[0] for e in enc]), np.stack([e[1] for e in enc]), [(e[2], e[3]) for e in enc], seeds)


def prepare(case, seed):
    kind = case["kind"]
    L = capi.host_generate_subspace(_seed32(seed, 1), N1)
    ctx = capi.Context(0)
    st = {"kind": kind, "case": case, "ctx": ctx}
    if kind in ("ivf", "ivf_block"):
        mix = _mixture(case, seed)
        ivf = capi.Ivf.build_keygen(ctx, mix["offsets"], mix["ids"], _residues(mix["x"]).reshape(-1), L, int(seed), N1)
        ivf.set_centroids(mix["centroids"])
        if kind == "ivf_block":
            ivf.block_prepare()
        st.update(h=ivf, q=mix["q"].to(torch.float32).cpu().numpy(), enc=_encode(mix["q"], L, seed))
        return st
    if kind == "encrypt":
        x = _residues(_vectors(case["rows"], case["d"], seed, 2, case["data"]))
        h_seed = _seed32(seed, 3)
        st.update(L=L, m_q=x.reshape(-1), keys=capi.keygen_h_s(ctx, h_seed, case["rows"], N1))
        return st
    x = _vectors(case["rows"], case["d"], seed, 2, case["data"])
    flat = capi.Flat.build_keygen(ctx, _residues(x).reshape(-1), case["rows"], L, _seed32(seed, 3), N1)
    enc = _encode(_vectors(case["B"], case["d"], seed, 4, case["data"]), L, seed)
    st.update(h=flat, enc=enc)
    if kind == "client":  # an honest server's r, and the client's own L^T v
        st["r"] = flat.compute_products(enc[0][0])
        v, Lm = enc[0][0].astype(object), L.reshape(N, N1).astype(object)
        st["lt"] = np.array([int(t) % P for t in v @ Lm], np.uint64)
    if kind in ("block_plan", "block"):
        flat.block_prepare()
    if kind == "block_plan":
        B, k = case["B"], case["k"]
        t = np.zeros((B, N), np.uint32)
        nnz = np.zeros(B, np.uint32)
        for i, (ti, ts) in enumerate(enc[2]):
            nnz[i] = ti.size
            t[i, : ti.size] = ti | np.where(ts < 0, np.uint32(0x80000000), np.uint32(0))
        dev = lambda a, ty: torch.from_numpy(a.view(ty)).to(DEV)  # noqa: E731
        st.update(plan=flat.block_plan(B, case["trials"], k), v=dev(enc[0], np.int64), g=dev(enc[1], np.int64),
                  t=dev(t, np.int32), nnz=dev(nnz, np.int32),
                  s=torch.from_numpy(np.frombuffer(enc[3][0], np.uint8).copy()).to(DEV),
                  ids=torch.zeros((B, k), dtype=torch.int32, device=DEV),
                  sc=torch.zeros((B, k), dtype=torch.int64, device=DEV),
                  n=torch.zeros(B, dtype=torch.int32, device=DEV), f=torch.zeros(B, dtype=torch.int32, device=DEV))
    return st


def _joined(hits):
    return np.concatenate([h[0] for h in hits]), np.concatenate([h[1] for h in hits])


def run(st):
    kind, c = st["kind"], st["case"]
    if kind == "encrypt":
        H, rowptr, idx, sign = st["keys"]
        m_enc, al = capi.encrypt_cluster(st["ctx"], st["m_q"], c["rows"], st["L"], H, rowptr, idx, sign, N1)
        return {"m_enc": m_enc, "al": al}
    h = st["h"]
    v, g, t, seeds = st["enc"]
    if kind == "query":
        hits, failed, _, _ = h.query(v, g, t, seeds, c["trials"], c["k"])
        return [*_joined(hits), failed]
    if kind == "products":
        return h.compute_products(v[0])
    if kind == "client":
        failed, ur, zv = h.verify(st["r"], v[0], seeds[0], c["trials"])
        return {"failed": failed, "ur": ur, "zv": zv, "dense": h.decode_dense_terms(g[0], st["lt"])}
    if kind == "block_plan":
        st["plan"].enqueue(st["v"].data_ptr(), st["g"].data_ptr(), st["t"].data_ptr(), st["nnz"].data_ptr(),
                           st["s"].data_ptr(), st["ids"].data_ptr(), st["sc"].data_ptr(), st["n"].data_ptr(),
                           st["f"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return [st["ids"], st["sc"], st["f"], st["n"]]
    if kind == "block":
        hits, failed, _ = h.query_block(v, g, t, seeds[0], c["trials"], c["k"])
        return [*_joined(hits), failed]
    probes = h.route(st["q"], c["nprobe"])
    if kind == "ivf":
        hits, fc, ft = h.query(probes, v, g, t, seeds, c["trials"], c["k"])
    else:
        hits, fc, ft = h.query_block(probes, v, g, t, seeds[0], c["trials"], c["k"])
    return [*_joined(hits), fc, ft, probes]


# ------------------------------------------------------------------ work
# Bytes of a corpus row: M_enc, [AL | H], and per query the ~128 columns of M
# that T selects (one byte each, eight for residues) and S's ~128 entries (two bytes).
ROW_ENC, ROW_DENSE, ROW_S = 8 * N, 2 * 8 * N1, 2 * N // 8


def _row_t(data):
    return N // 8 * (8 if data == "q20" else 1)


def work(case):
    """Bytes read once and written once; operations are 2 per multiply-add mod p."""
    kind, rows = case["kind"], case["rows"]
    if kind == "encrypt":
        return {"bytes": rows * (2 * ROW_ENC + ROW_DENSE + 5 * N // 8), "flops": 4.0 * rows * N * N1}
    B, trials = case["B"], case.get("trials", 0)
    if kind == "products":
        return {"bytes": rows * (ROW_ENC + 8), "flops": 2.0 * rows * N}
    if kind == "client":
        return {"bytes": rows * (ROW_ENC + ROW_DENSE + 16), "flops": 2.0 * rows * (trials * (N + 1) + 2 * N1)}
    if kind == "query":
        # the corpus once for all of a call's queries; seeds differ, so the draws and products are per query
        per = rows * (N * (1 + trials) + trials + 2 * N1 + N // 4)
        return {"bytes": rows * (ROW_ENC + ROW_DENSE + _row_t("q20" if case["data"] == "q20" else "int8") + ROW_S),
                "flops": 2.0 * B * per}
    if kind in ("block_plan", "block"):
        # one seed per block: z once, then r, u . r and the decode per query
        return {"bytes": rows * (ROW_ENC + ROW_DENSE + N + ROW_S),
                "flops": 2.0 * rows * (trials * N + B * (N + trials + 2 * N1 + N // 4))}
    # IVF: expected rows a query probes, and the distinct rows of the batch
    frac = min(1.0, case["nprobe"] / case["nlist"])
    pairs = B * frac * rows
    distinct = rows * (1.0 - (1.0 - frac) ** B)
    z_rows = pairs if kind == "ivf" else distinct
    return {"bytes": distinct * (ROW_ENC + ROW_DENSE + N + ROW_S) + 4.0 * case["nlist"] * case["d"],
            "flops": 2.0 * (z_rows * trials * N + pairs * (N + trials + 2 * N1 + N // 4))}


# ------------------------------------------------------------------ exact
def _ranked(x, q, ids, k):
    """Top-k of x . q by (score desc, id asc); every product is below 2^53."""
    s = (x.to(torch.float64) @ q.to(torch.float64)).to(torch.int64).cpu().numpy()
    order = np.lexsort((ids, -s))[:k]
    return ids[order], s[order]


def exact(case, seed):
    """The ranked plaintext products of every query with an honest server's
    verdicts, where a case returns hits; None for encrypted values."""
    if case["kind"] not in ("query", "block") or case["rows"] * case["B"] > 4 << 20:
        return None
    x = _vectors(case["rows"], case["d"], seed, 2, case["data"])
    q = _vectors(case["B"], case["d"], seed, 4, case["data"])
    ids = np.arange(case["rows"], dtype=np.uint32)
    hits = [_ranked(x, q[b], ids, case["k"]) for b in range(case["B"])]
    return [*_joined(hits), np.full(case["B"], -1, np.int32)]
