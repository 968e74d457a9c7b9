"""The workloads whose speed matters to a program that uses this library: quantising images'
descriptors with a vocabulary tree, training such trees, and retrieving images from an index.

``listed()`` names fixed cases, ``draw()`` gives further ones of the same ranges, ``prepare()``
makes a case's inputs and handles from a seed, ``run()`` is one pass through the public API,
``work()`` the bytes and operations such a pass cannot do without, and ``exact()`` its result
in plain torch (whole numbers exactly, computed numbers in 64 bits).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import rapidbow_b200 as rbw
from rapidbow_b200.synth import sift_like

DEV = "cuda"
FLT_MIN = float(np.finfo(np.float32).tiny)
ROWS = 1 << 17  # descriptors per step of the plain-torch tree code


def listed():
    return [
        # One photograph's descriptors to words: the call of a search front end, latency counts.
        {"name": "lookup_image", "kind": "lookup", "n": 731, "B": 16, "L": 4, "float": False},
        # A burst of photographs quantised together (a serving batch), ragged size.
        {"name": "lookup_burst", "kind": "lookup", "n": 60_013, "B": 16, "L": 4, "float": False},
        # Quantising a collection: 10M descriptors through 65,536 words (the benchmark's lookup).
        {"name": "lookup_10m", "kind": "lookup", "n": 10_000_000, "B": 16, "L": 4, "float": False},
        # The same through a deep, narrow tree of 1M words.
        {"name": "lookup_deep", "kind": "lookup", "n": 1_000_003, "B": 10, "L": 6, "float": False},
        # Words of a float-center vocabulary (FP64-exact assignment).
        {"name": "lookup_float", "kind": "lookup", "n": 200_003, "B": 10, "L": 4, "float": True},
        # A vocabulary from a small collection with the defaults (reference init, to convergence).
        {"name": "build_default_50k", "kind": "build", "n": 50_021, "B": 16, "L": 3, "init": "reference",
         "iterations": 1000, "words": False},
        # The benchmark's small build: k-means++, ten Lloyd steps.
        {"name": "build_200k", "kind": "build", "n": 200_000, "B": 16, "L": 3, "init": "kmeans++",
         "iterations": 10, "words": False},
        # A 1M-word vocabulary from 10M descriptors, which are then quantised with it.
        {"name": "build_10m", "kind": "build", "n": 10_000_000, "B": 10, "L": 6, "init": "kmeans++",
         "iterations": 10, "words": True},
        # A float-center vocabulary from chosen initial centers.
        {"name": "build_float_300k", "kind": "build_float", "n": 300_007, "B": 10, "L": 4, "iterations": 10},
        # One photograph's words against an index of 20,000 images: an interactive search.
        {"name": "query_image", "kind": "query", "docs": 20_000, "words": 1_733, "k": 100},
        # 256 searches at once against the same index (the benchmark's scoring).
        {"name": "query_batch", "kind": "query_batch", "docs": 20_000, "queries": 256, "k": 50},
        # A new index of a small collection, answered from at once.
        {"name": "index_3k", "kind": "index", "docs": 3_001, "queries": 16, "k": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lookup", "lookup", "lookup", "lookup_float", "build", "build", "build_float", "query",
                       "query_batch", "index"])
    if kind == "lookup":
        B, L = rng.choice([(16, 4), (16, 4), (16, 3), (10, 6), (10, 4)])
        return {"kind": "lookup", "n": _log(rng, 200, 10_000_000), "B": B, "L": L, "float": False}
    if kind == "lookup_float":
        return {"kind": "lookup", "n": _log(rng, 1_000, 1_000_000), "B": 10, "L": 4, "float": True}
    if kind == "build":
        B, L = rng.choice([(16, 3), (16, 4), (10, 4), (10, 6)])
        n = _log(rng, 20_000, 5_000_000)
        if rng.random() < 0.3:
            return {"kind": "build", "n": min(n, 200_000), "B": 16, "L": 3, "init": "reference", "iterations": 1000,
                    "words": False}
        return {"kind": "build", "n": n, "B": B, "L": L, "init": "kmeans++", "iterations": 10,
                "words": B ** L > 100_000}
    if kind == "build_float":
        return {"kind": "build_float", "n": _log(rng, 20_000, 1_000_000), "B": 10, "L": 4, "iterations": 10}
    if kind == "query":
        return {"kind": "query", "docs": _log(rng, 2_000, 40_000), "words": _log(rng, 300, 8_000),
                "k": rng.randint(10, 100)}
    if kind == "query_batch":
        return {"kind": "query_batch", "docs": _log(rng, 2_000, 20_000), "queries": _log(rng, 2, 256),
                "k": rng.randint(10, 100)}
    return {"kind": "index", "docs": _log(rng, 500, 6_000), "queries": _log(rng, 1, 64), "k": rng.randint(10, 50)}


# ------------------------------------------------------------------ inputs
def _level_beg(B, level):
    return sum(B ** i for i in range(level))


def _nodes(c):
    return _level_beg(c["B"], c["L"])


def _nearest(x, node, centers):
    """Index of the nearest of each row's node's centers, the lowest one on ties."""
    out = torch.empty(x.shape[0], dtype=torch.int64, device=x.device)
    idx = torch.arange(centers.shape[1], device=x.device)
    integer = centers.dtype == torch.uint8
    for i in range(0, x.shape[0], ROWS):
        # whole numbers: every sum is below 2^24, so fp32 is exact
        c = centers[node[i: i + ROWS]].to(torch.float32 if integer else torch.float64)
        v = x[i: i + ROWS].to(c.dtype)
        if integer:
            d = (c * c).sum(2) - 2 * torch.bmm(c, v.unsqueeze(2)).squeeze(2)
        else:
            d = (v.unsqueeze(1) - c).square().sum(2)
        out[i: i + ROWS] = torch.where(d == d.amin(1, keepdim=True), idx, centers.shape[1]).amin(1)
    return out


def _sums(x, word, words):
    """Exact sums and counts of the rows of every word."""
    counts = torch.bincount(word, minlength=words)
    total = torch.zeros(words, 128, dtype=torch.float64, device=x.device)
    if words <= 2048:  # as products with the one-hot matrix: few words would all be added to at once
        ids = torch.arange(words, device=x.device).unsqueeze(1)
        for i in range(0, x.shape[0], ROWS):
            hot = (word[i: i + ROWS].unsqueeze(0) == ids).to(torch.float32)
            # sums of 2^16 bytes at most stay below 2^24
            for j in range(0, hot.shape[1], 1 << 16):
                total += (hot[:, j: j + (1 << 16)] @ x[i + j: i + j + hot[:, j: j + (1 << 16)].shape[1]].float()).double()
    else:
        for i in range(0, x.shape[0], ROWS):
            total.index_add_(0, word[i: i + ROWS], x[i: i + ROWS].double())
    return total, counts


def _lloyd(x, node, centers, steps, integer):
    """`steps` Lloyd steps of every node of a level, stopping with the node; (centers, words)."""
    nb, B = centers.shape[:2]
    last = torch.zeros(x.shape[0], dtype=torch.int64, device=x.device)
    for step in range(steps):
        last = _nearest(x, node, centers)
        total, counts = _sums(x, node * B + last, nb * B)
        mean = total / counts.clamp_min(1).unsqueeze(1).double()
        new = mean.round().to(torch.uint8) if integer else mean.float()
        centers = torch.where((counts > 0).view(nb, B, 1), new.view(nb, B, 128), centers)
    return centers, node * B + last


def _members(node, nb, B, g):
    """B members of every node at random (again from the first one in small nodes, any row in empty ones)."""
    n = node.numel()
    order = torch.randperm(n, generator=g, device=node.device)
    order = order[torch.argsort(node[order], stable=True)]
    count = torch.bincount(node, minlength=nb)
    first = torch.cumsum(count, 0) - count
    k = torch.arange(B, device=node.device).unsqueeze(0) % count.clamp_min(1).unsqueeze(1)
    at = (first.unsqueeze(1) + k).clamp_max(n - 1)
    return order[at]


def _tree(x, B, L, steps, seed, integer):
    """A vocabulary tree of descriptors x by hierarchical k-means from random members: centers
    [nodes, B, 128], the descriptor each center began as [nodes, B], and counts [nodes * B]."""
    g = torch.Generator(device=x.device).manual_seed(seed)
    node = torch.zeros(x.shape[0], dtype=torch.int64, device=x.device)
    centers, picks, counts = [], [], []
    for level in range(L):
        nb = B ** level
        p = _members(node, nb, B, g)
        c = x[p] if integer else x[p].float()
        c, node = _lloyd(x, node, c, steps, integer)
        centers.append(c)
        picks.append(p)
        counts.append(torch.bincount(node, minlength=nb * B))
    return torch.cat(centers), torch.cat(picks), torch.cat(counts)


def _weights(counts, nb_doc):
    """idf weights in 64 bits."""
    w = torch.log(nb_doc / counts.double().clamp_min(1))
    return torch.where(counts > 0, w.clamp_min(FLT_MIN), torch.full_like(w, FLT_MIN))


def _descend(x, centers, B, L):
    node = torch.zeros(x.shape[0], dtype=torch.int64, device=x.device)
    for level in range(L):
        node = node * B + _nearest(x, _level_beg(B, level) + node, centers)
    return node


def _descriptors(n, seed, many=False):
    return sift_like(n, seed=seed, n_components=4096 if many else 256, zipf=1.1 if many else None, device=DEV)


def _lookup_inputs(case, seed):
    B, L = case["B"], case["L"]
    deep = B ** L > 100_000
    train = _descriptors(1_500_000 if deep else 400_000, seed * 3 + 1, deep)
    centers, _, counts = _tree(train, B, L, 2, seed, not case["float"])
    return centers, _weights(counts, train.shape[0] / 500), _descriptors(case["n"], seed * 3 + 2, deep)


def _vocabulary(B, L, centers, weights):
    make = rbw.vocabulary_from_host if centers.dtype == torch.uint8 else rbw.vocabulary_from_host_f32
    nodes = centers.shape[0]
    return make(B, L, centers.cpu().numpy(), np.full(nodes, (1 << B) - 1, np.uint32),
                weights.float().reshape(nodes, B).cpu().numpy())


# An index: images of 500 to 4,000 words (log-uniform) of a 65,536-word tree.
TREE_B, TREE_L = 16, 4


def _images(n, words, g, lo=500, hi=4_000):
    """Words of n images, drawn from quantised descriptors, as (words, offsets)."""
    size = torch.exp(torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * math.log(hi / lo)
                     + math.log(lo)).round().long()
    off = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(size, 0)
    return words[torch.randint(words.numel(), (int(off[-1]),), generator=g, device=DEV)], off


def _index_inputs(case, seed):
    """(weights, document words and offsets, query words and offsets); every other query shares
    60 % of its words with a document."""
    train = _descriptors(400_000, seed * 3 + 1)
    centers, _, counts = _tree(train, TREE_B, TREE_L, 1, seed, True)
    g = torch.Generator(device=DEV).manual_seed(seed)
    words = _descend(_descriptors(400_000, seed * 3 + 2), centers, TREE_B, TREE_L)
    dw, do = _images(case["docs"], words, g)
    if case["kind"] == "query":
        nq = 1
        qw, qo = _images(1, words, g, case["words"], case["words"])
    else:
        nq = case["queries"]
        qw, qo = _images(nq, words, g)
    for q in range(0, nq, 2):
        a, b = int(qo[q]), int(qo[q + 1])
        d = int(torch.randint(case["docs"], (1,), generator=g, device=DEV))
        own = dw[do[d]: do[d + 1]]
        take = min(own.numel(), int(0.6 * (b - a)))
        qw[a: a + take] = own[torch.randperm(own.numel(), generator=g, device=DEV)[:take]]
    return centers, _weights(counts, train.shape[0] / 500).float(), dw, do, qw, qo


def prepare(case, seed):
    kind = case["kind"]
    if kind == "lookup":
        centers, weights, desc = _lookup_inputs(case, seed)
        return {"case": case, "voc": _vocabulary(case["B"], case["L"], centers, weights), "desc": desc}
    if kind == "build":
        return {"case": case, "desc": _descriptors(case["n"], seed, case["B"] ** case["L"] > 100_000)}
    if kind == "build_float":
        desc = _descriptors(case["n"], seed)
        picks = _tree(desc, case["B"], case["L"], 2, seed, False)[1]
        return {"case": case, "desc": desc, "picks": picks.cpu().numpy().astype(np.uint32)}
    centers, weights, dw, do, qw, qo = _index_inputs(case, seed)
    state = {"case": case, "voc": _vocabulary(TREE_B, TREE_L, centers, weights),
             "ids": np.arange(case["docs"], dtype=np.uint32), "words": dw.cpu().numpy().astype(np.uint32),
             "offsets": do.cpu().numpy().astype(np.uint64), "q": qw.int(), "qo": qo,
             "q_host": qw.cpu().numpy().astype(np.uint32)}
    if kind != "index":
        db = rbw.create_database(state["voc"])
        db.add_docs(state["ids"], state["words"], state["offsets"])
        db.query(state["q_host"][:int(qo[1])], case["k"])  # the first query indexes the documents
        state["db"] = db
    return state


# ------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "lookup":
        return state["voc"].lookup(state["desc"])
    if kind == "build":
        desc = state["desc"]
        voc = rbw.build_vocabulary(desc, case["B"], nb_doc=max(1, case["n"] // 500), nb_levels=case["L"],
                                   max_iterations=case["iterations"], init=case["init"], seed=7)
        if case["words"]:
            return [voc.lookup(desc)] + [voc.level_weights(level) for level in range(case["L"])]
        return list(voc.tree())
    if kind == "build_float":
        voc = rbw.build_vocabulary(state["desc"], case["B"], nb_doc=max(1, case["n"] // 500), nb_levels=case["L"],
                                   max_iterations=case["iterations"], init="injected", injected=state["picks"],
                                   float_centers=True)
        return [voc.centers_f32()] + [voc.level_weights(level) for level in range(case["L"])]
    if kind == "query":
        return list(state["db"].query(state["q_host"], case["k"], with_scores=True))
    if kind == "query_batch":
        return list(state["db"].query_batched(state["q"], state["qo"], case["k"]))
    db = rbw.create_database(state["voc"])
    db.add_docs(state["ids"], state["words"], state["offsets"])
    return list(db.query_batched(state["q"], state["qo"], case["k"]))


def work(case):
    kind = case["kind"]
    if kind == "lookup":
        tree = min(_nodes(case), case["n"] * case["L"]) * case["B"] * 128 * (4 if case["float"] else 1)
        return {"bytes": case["n"] * 132 + tree, "flops": 2 * 128 * case["B"] * case["L"] * case["n"]}
    if kind in ("build", "build_float"):
        nodes = _nodes(case)
        # a build to convergence takes at least the four steps before its first check
        steps = min(case["iterations"], 10) if case["iterations"] <= 10 else 4
        flops = 2 * 128 * case["B"] * case["L"] * case["n"] * steps
        if kind == "build" and case["words"]:
            # the words and the weights come back; the descriptors are read to build and to quantise
            return {"bytes": case["n"] * (2 * 128 + 4) + nodes * case["B"] * 4,
                    "flops": flops + 2 * 128 * case["B"] * case["L"] * case["n"]}
        centers = nodes * case["B"] * 128 * (4 if kind == "build_float" else 1)
        return {"bytes": case["n"] * 128 + centers + nodes * case["B"] * 4, "flops": flops}
    mean = (4_000 - 500) / math.log(8)  # words of an image
    postings = case["docs"] * mean
    if kind == "index":
        # the documents in, an index entry (document, weight) per word out and the queries' lists in
        share = 1 - (1 - mean / TREE_B ** TREE_L) ** case["queries"]
        return {"bytes": int(postings * (4 + 8 + 8 * share) + case["queries"] * (mean * 4 + case["k"] * 8)),
                "flops": int(postings * 4)}
    queries, words = (1, case["words"]) if kind == "query" else (case["queries"], mean)
    # posting lists of the queries' words, once each however many queries ask for them
    share = 1 - (1 - words / TREE_B ** TREE_L) ** queries
    return {"bytes": int(postings * share * 8 + queries * (words * 4 + case["k"] * 8)),
            "flops": int(queries * postings * words / TREE_B ** TREE_L * 4)}


# ------------------------------------------------------------------ the same in plain torch
def _norms(word, owner, n, weights):
    total = torch.zeros(n, dtype=torch.float64, device=DEV)
    for level in range(TREE_L - 1, -1, -1):
        total.index_add_(0, owner, weights[_level_beg(TREE_B, level) * TREE_B + word])
        word = word // TREE_B
    return total


def _scores(case, seed):
    """Scores of the k best documents of every query: 2 + sum(|q - d| - (q + d)) over the shared
    words of every level, words above the leaves only while their documents are few."""
    centers, weights, dw, do, qw, qo = _index_inputs(case, seed)
    weights, nd, nq, k = weights.double(), do.numel() - 1, qo.numel() - 1, case["k"]
    owner = torch.repeat_interleave(torch.arange(nd, device=DEV), do.diff())
    d_rcp = 1 / _norms(dw, owner, nd, weights)
    q_owner = torch.repeat_interleave(torch.arange(nq, device=DEV), qo.diff())
    q_rcp = 1 / _norms(qw, q_owner, nq, weights)
    levels = []
    for level in range(TREE_L):
        span = TREE_B ** (TREE_L - 1 - level)
        size = TREE_B ** (level + 1)
        w = weights[_level_beg(TREE_B, level) * TREE_B:][:size]
        per_word = torch.bincount(dw // span, minlength=size)
        used = torch.ones_like(per_word, dtype=torch.bool) if span == 1 else per_word < 16 + 4 * k
        word = dw // span
        keep = used[word]
        key, tf = torch.unique(owner[keep] * size + word[keep], return_counts=True)
        doc, word = key // size, key % size
        levels.append((span, size, w, doc, word, tf * w[word] * d_rcp[doc]))
    best = torch.empty(nq, k, dtype=torch.float64, device=DEV)
    for q in range(nq):
        acc = torch.zeros(nd, dtype=torch.float64, device=DEV)
        touched = torch.zeros(nd, dtype=torch.bool, device=DEV)
        for span, size, w, doc, word, d in levels:
            qv = torch.bincount(qw[qo[q]: qo[q + 1]] // span, minlength=size) * w * q_rcp[q]
            at = torch.nonzero(qv[word] > 0).squeeze(1)
            v = qv[word[at]]
            acc.index_add_(0, doc[at], (v - d[at]).abs() - (v + d[at]))
            touched[doc[at]] = True
        s = torch.where(touched, acc + 2, torch.full_like(acc, math.inf))
        best[q] = torch.sort(s).values[:k]
    return best


def exact(case, seed):
    kind = case["kind"]
    if kind == "lookup":
        centers, _, desc = _lookup_inputs(case, seed)
        return _descend(desc, centers, case["B"], case["L"])
    if kind == "build":
        return None  # whole numbers: centers and words (the weights follow from whole counts)
    if kind == "build_float":
        B, L = case["B"], case["L"]
        desc = _descriptors(case["n"], seed)
        picks = _tree(desc, B, L, 2, seed, False)[1]
        node = torch.zeros(case["n"], dtype=torch.int64, device=DEV)
        centers, weights = [], []
        for level in range(L):
            p = picks[_level_beg(B, level): _level_beg(B, level + 1)]
            c, node = _lloyd(desc, node, desc[p].float(), case["iterations"], False)
            centers.append(c)
            weights.append(_weights(torch.bincount(node, minlength=B ** (level + 1)), max(1, case["n"] // 500))
                           .view(-1, B))
        return [torch.cat(centers).double()] + weights
    scores = _scores(case, seed)
    return [None, scores[0]] if kind == "query" else [None, scores, None]
