"""The work that a user of this library has it do, as cases to time.

Most cases are searches, since that is what an index is for: one query, a
handful of queries (online serving), full batches in each precision and entry
mode, long rows, wide beams, and an uneven stream of batches through the
CUDA-graph batcher.  The rest is what an index costs before it serves: its
exact kNN graph, its PCA, and the training of its learned entry.

An index stands for the one that a serving program keeps: its base is made
from a fixed seed, and it is built once per process and shape.  What a call
gets (queries, training queries, the base of a graph or PCA build) is made
from the case's seed.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

import rt_entry_gb300 as rte

DEVICE = "cuda:0"
BASE_SEED = 1001
LEAF_SIZE = 32
EXPAND = 0.2
PRECISIONS = {"fp32": rte.PREC_FP32, "bf16": rte.PREC_BF16, "fp8": rte.PREC_FP8}
ENTRIES = {"random": rte.ENTRY_RANDOM, "kdtree": rte.ENTRY_KDTREE, "learned": rte.ENTRY_LEARNED}

# ---- shapes of the served indexes -----------------------------------------
# 1M x 128 integer values 0..255 over a degree-64 graph (SIFT-like)
SIFT = dict(data="flat", n=1_000_000, d=128, degree=64)
# long rows in [0, 1] over a degree-64 graph; the base is larger than L2
GIST = dict(data="minmax", n=200_000, d=960, degree=64)
# unit vectors over a degree-32 graph (angular)
DEEP = dict(data="unit", n=500_000, d=96, degree=32)
# the small configuration: 100k x 128, well-separated clusters
SMALL = dict(data="iso", n=100_000, d=128, degree=32)


def _search(name, index, nq, beam, width, k, precision, entry, hits=1):
    return dict(name=name, op="search", nq=nq, beam=beam, width=width, k=k, precision=precision, entry=entry,
                hits=hits, **index)


def listed():
    return [
        # a single interactive query with the default parameters
        _search("one_query", SIFT, 1, 64, 1, 10, "fp32", "kdtree"),
        # an online server's micro-batch
        _search("online_batch", SIFT, 37, 32, 1, 10, "bf16", "learned"),
        # offline batches: the plain method, and learned entries with
        # reduced-precision distances and the exact rerank
        _search("plain_10k", SIFT, 10_000, 32, 1, 10, "fp32", "kdtree"),
        _search("learned_10k", SIFT, 10_000, 16, 1, 10, "bf16", "learned"),
        # candidate generation: many neighbours per query, an odd batch size
        _search("candidates_k100", SIFT, 2_049, 128, 1, 100, "bf16", "kdtree"),
        # long rows, both ends of the precisions
        _search("long_rows_fp32", GIST, 1_000, 64, 1, 10, "fp32", "kdtree"),
        _search("long_rows_fp8", GIST, 1_000, 256, 4, 10, "fp8", "kdtree"),
        # angular data at the widest beam
        _search("angular_wide", DEEP, 10_000, 256, 4, 10, "bf16", "learned"),
        # a server that takes batches of uneven size from pinned host memory
        dict(name="uneven_stream", op="stream", batches=12, max_batch=8192, plan=4004, beam=32, width=1, k=10,
             precision="bf16", entry="learned", **SIFT),
        # before serving: the exact kNN graph of a new base
        dict(name="knn_graph", op="knn", data="iso", n=100_000, d=128, degree=32),
        # ... its PCA, with the base projected
        dict(name="build_pca", op="pca", data="flat", n=300_000, d=128, probe=1_000),
        # ... and one epoch of the learned entry (forward, backward, update)
        dict(name="train_entry", op="train", queries=131_072, batch=4096, epochs=1, probe=4_096, **SMALL),
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    op = rng.choices(("search", "stream", "knn", "pca", "train"), (60, 10, 12, 10, 8))[0]
    if op == "search":
        if rng.random() < 0.6:
            index = dict(rng.choice((SIFT, SIFT, GIST, DEEP, SMALL)))
        else:
            d = _log(rng, 32, 1000)
            data = rng.choice(("flat", "iso", "minmax", "unit"))
            index = dict(data=data, n=_log(rng, 20_000, 150_000), d=d, degree=rng.choice((16, 32, 64)))
        beam = rng.choice((16, 32, 64, 128, 256))
        widths = [w for w in (1, 2, 4) if w * index["degree"] <= 256 and w * 32 <= beam * 2]
        entry = rng.choice(("kdtree", "kdtree", "learned", "random"))
        k = rng.choice([k for k in (1, 10, 100) if k <= beam])
        hits = rng.choice((1, 1, 1, 2, 4)) if entry == "kdtree" else 1
        nq = min(_log(rng, 1, 10_000), 10_000 * 128 // max(128, index["d"]))
        c = _search("", index, nq, beam, rng.choice(widths), k, rng.choice(tuple(PRECISIONS)), entry, hits)
        del c["name"]
        return c
    if op == "stream":
        return dict(op="stream", batches=rng.randint(4, 16), max_batch=_log(rng, 64, 8192), plan=rng.randrange(1 << 20),
                    beam=rng.choice((16, 32, 64)), width=1, k=rng.choice((1, 10)),
                    precision=rng.choice(("fp32", "bf16")), entry=rng.choice(("kdtree", "learned")), **SIFT)
    if op == "knn":
        d = _log(rng, 32, 960)
        n = min(_log(rng, 2_000, 100_000), 100_000 * 128 // max(128, d))
        return dict(op="knn", data=rng.choice(("flat", "iso", "minmax", "unit")), n=n, d=d,
                    degree=rng.choice((16, 32, 64)))
    if op == "pca":
        d = _log(rng, 32, 256)
        return dict(op="pca", data=rng.choice(("flat", "iso", "minmax")), n=min(_log(rng, 5_000, 300_000), 300_000 * 128 // max(d, 128)),
                    d=d, probe=_log(rng, 100, 1_000))
    return dict(op="train", queries=_log(rng, 8_192, 131_072), batch=rng.choice((1024, 2048, 4096)), epochs=1,
                probe=_log(rng, 100, 4_096), **SMALL)


# ---- data -------------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


@functools.lru_cache(maxsize=16)
def _mixture(data: str, d: int):
    """Cluster centres (and spreads) of a data family, fixed per dimension."""
    g = _gen(BASE_SEED + 17 * d + sum(map(ord, data)))
    if data == "flat":     # 256 flat clusters whose centres lie on a low-dimensional subspace
        b = torch.linalg.qr(torch.randn(d, 8, generator=g, device=DEVICE).cpu())[0].to(DEVICE)
        cent = 128.0 + (torch.randn(256, 8, generator=g, device=DEVICE) * 50.0) @ b.T
        bases = torch.linalg.qr(torch.randn(256, d, 16, generator=g, device=DEVICE).cpu())[0].to(DEVICE)
        return cent, bases
    if data == "iso":      # 64 isotropic clusters, centres U[0, 100]
        return torch.rand(64, d, generator=g, device=DEVICE) * 100.0, None
    if data == "minmax":   # 128 clusters, N(0, 1) around N(0, 1), scaled to about [0, 1]
        return torch.randn(128, d, generator=g, device=DEVICE), None
    if data == "unit":     # 1024 clusters on the unit sphere
        return torch.randn(1024, d, generator=g, device=DEVICE), None
    raise ValueError(data)


def _sample(data: str, n: int, d: int, seed: int) -> torch.Tensor:
    cent, bases = _mixture(data, d)
    g = _gen(seed)
    lab = torch.randint(cent.shape[0], (n,), generator=g, device=DEVICE)
    if data == "flat":
        z = torch.randn(n, 16, generator=g, device=DEVICE) * 25.0
        x = cent[lab] + torch.randn(n, d, generator=g, device=DEVICE) * 6.0
        step = max(1, (1 << 26) // (16 * d))
        for s in range(0, n, step):
            x[s:s + step] += (bases[lab[s:s + step]] * z[s:s + step, None, :]).sum(-1)
        return x.clamp_(0, 255).round_()
    noise = torch.randn(n, d, generator=g, device=DEVICE)
    if data == "iso":
        return cent[lab] + 5.0 * noise
    if data == "minmax":
        return (cent[lab] + noise) / 12.0 + 0.5
    x = cent[lab] + 0.35 * noise
    return x / x.norm(dim=1, keepdim=True)


def _pca64(x: torch.Tensor):
    """Mean, eigenvectors (columns, largest component positive) and eigenvalues, descending, in 64 bits."""
    n, d = x.shape
    mean = torch.zeros(d, dtype=torch.float64, device=x.device)
    for s in range(0, n, 1 << 16):
        mean += x[s:s + (1 << 16)].double().sum(0)
    mean /= n
    cov = torch.zeros(d, d, dtype=torch.float64, device=x.device)
    for s in range(0, n, 1 << 16):
        c = x[s:s + (1 << 16)].double() - mean
        cov += c.T @ c
    w, v = np.linalg.eigh((cov / (n - 1)).cpu().numpy())
    w, v = w[::-1].copy(), v[:, ::-1].copy()
    v *= np.where(v[np.abs(v).argmax(0), np.arange(d)] < 0, -1.0, 1.0)
    return mean.cpu().numpy(), v, w


# ---- the indexes a program keeps ----------------------------------------------
@functools.lru_cache(maxsize=6)
def _index(data: str, n: int, d: int, degree: int, role: str) -> rte.Index:
    """`role` keeps the index that the training cases train apart from the ones that serve."""
    base = _sample(data, n, d, BASE_SEED)
    graph = rte.knn_graph(base, degree)
    mean, rot, _ = _pca64(base)
    idx = rte.Index.from_arrays(base, graph).set_pca(mean, rot).build_kdtree(LEAF_SIZE, EXPAND)
    idx.prepare(rte.COPY_BF16 | rte.COPY_FP8)
    return idx


@functools.lru_cache(maxsize=6)
def _trained(data: str, n: int, d: int, degree: int) -> rte.Index:
    idx = _index(data, n, d, degree, "serve")
    idx.train_learned(_sample(data, 131_072, d, BASE_SEED + 2), batch=4096, epochs=2)
    return idx


def _serving(case) -> rte.Index:
    shape = (case["data"], case["n"], case["d"], case["degree"])
    # the head takes projected rows of up to 256 dims in its fused form; a
    # trained index also serves kd-tree and random entries
    return _trained(*shape) if case["entry"] == "learned" else _index(*shape, "serve")


def _params(case) -> rte.SearchParams:
    prec = PRECISIONS[case["precision"]]
    return rte.default_params(beam=case["beam"], search_width=case["width"], k=case["k"], precision=prec,
                              rerank=int(prec != rte.PREC_FP32), entry_mode=ENTRIES[case["entry"]],
                              max_hits=case.get("hits", 1))


def _stream_sizes(case):
    rng = random.Random(case["plan"])
    return [max(1, int(math.exp(rng.uniform(0.0, math.log(case["max_batch"]))))) for _ in range(case["batches"])]


# ---- the measured calls ----------------------------------------------------------
def prepare(case, seed):
    op, d = case["op"], case["d"]
    s = dict(op=op)
    if op == "search":
        s["index"] = _serving(case)
        s["params"] = _params(case)
        s["queries"] = _sample(case["data"], case["nq"], d, seed)
    elif op == "stream":
        sizes = _stream_sizes(case)
        s["batcher"] = _serving(case).batcher(case["max_batch"], params=_params(case))
        q = _sample(case["data"], sum(sizes), d, seed).cpu()
        s["batches"] = []
        for part in torch.split(q, sizes):
            m = part.shape[0]
            s["batches"].append((part.contiguous().pin_memory(), torch.empty((m, case["k"]), dtype=torch.int32).pin_memory(),
                                 torch.empty((m, case["k"]), dtype=torch.float32).pin_memory()))
    elif op == "knn":
        s["base"] = _sample(case["data"], case["n"], d, seed)
        s["degree"] = case["degree"]
    elif op == "pca":
        n = case["n"]
        base = _sample(case["data"], n, d, seed)
        # the PCA does not read the graph: a ring of the smallest degree
        ring = (torch.arange(n, device=DEVICE)[:, None] + torch.arange(1, 17, device=DEVICE)) % n
        s["index"] = rte.Index.from_arrays(base, ring)
        s["probe"] = _sample(case["data"], case["probe"], d, seed + (1 << 30))
    else:
        s["index"] = _index(case["data"], case["n"], d, case["degree"], "train")
        s["train"] = _sample(case["data"], case["queries"], d, seed)
        s["probe"] = s["index"].project(_sample(case["data"], case["probe"], d, seed + (1 << 30)))
        s["batch"], s["epochs"] = case["batch"], case["epochs"]
    return s


def run(s):
    op = s["op"]
    if op == "search":
        return s["index"].search(s["queries"], s["params"])
    if op == "stream":
        return [s["batcher"].search(q, out_ids=ids, out_dists=dists) for q, ids, dists in s["batches"]]
    if op == "knn":
        return rte.knn_graph(s["base"], s["degree"])
    if op == "pca":
        mean, rotation, eigenvalues = s["index"].build_pca().pca()
        return dict(mean=mean, rotation=rotation, eigenvalues=eigenvalues, projected=s["index"].project(s["probe"]))
    # the head's weights have no accessor: the leaves that it proposes stand
    # for them, with the loss of the first and the last step
    report = s["index"].train_learned(s["train"], batch=s["batch"], epochs=s["epochs"])
    return dict(leaves=s["index"].learned_leaves(s["probe"]),
                loss=np.array([report["first_loss"], report["last_loss"]], np.float32))


def exact(case, seed):
    """Only the PCA has outputs that plain arithmetic gives: which neighbours
    a beam search reaches, and which leaves a trained head proposes, is
    decided step by step, and a graph is whole numbers."""
    if case["op"] != "pca":
        return None
    x = _sample(case["data"], case["n"], case["d"], seed)
    probe = _sample(case["data"], case["probe"], case["d"], seed + (1 << 30))
    mean, rot, w = _pca64(x)
    return dict(mean=mean, rotation=rot, eigenvalues=w, projected=(probe.double().cpu().numpy() - mean) @ rot)


def _search_work(case, nq):
    """What a beam search cannot do without: at least `beam` nodes are
    expanded per query, each reading its neighbour list, and about half of
    the listed neighbours are new and have their distance evaluated.  Rows
    that several queries share need to be read once, so the index bounds it."""
    n, d, degree, beam = case["n"], case["d"], case["degree"], case["beam"]
    size = {"fp32": 4, "bf16": 2, "fp8": 1}[case["precision"]]
    evals = beam + beam * degree / 2
    per_query = beam * 4 * degree + evals * size * d
    whole = n * (4 * degree + size * d)
    return dict(bytes=min(nq * per_query, whole) + nq * (4 * d + 8 * case["k"]), flops=3.0 * nq * evals * d)


def work(case):
    n, d = case["n"], case["d"]
    if case["op"] == "search":
        return _search_work(case, case["nq"])
    if case["op"] == "stream":
        return _search_work(case, sum(_stream_sizes(case)))
    if case["op"] == "knn":
        return dict(bytes=4.0 * n * (d + case["degree"]), flops=2.0 * n * n * d)
    if case["op"] == "pca":  # mean and covariance (its upper half), then the projected base
        return dict(bytes=8.0 * n * d + 4.0 * case["probe"] * 2 * d, flops=n * d * (d + 1.0) + 2.0 * n * d * d)
    # the labelling search (beam 64), then forward and backward of 256 -> 256 -> classes
    q, h, classes = case["queries"], 256, 4096
    label = _search_work(dict(case, beam=64, k=1, precision="fp32"), q)
    steps = q // case["batch"] * case["epochs"]
    params = d * h + h * h + h * classes
    return dict(bytes=label["bytes"] + steps * 20.0 * params,
                flops=label["flops"] + 6.0 * steps * case["batch"] * params)
