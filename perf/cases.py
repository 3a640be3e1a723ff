"""The work this library does for its users, as cases that can be timed.

Every case is a call, or a short sequence of calls, of the Python binding on
rows that are already on the device: exact k-NN of host queries, beam search of
host queries over a built graph, a k-NN graph, the rank prune of given pools,
and whole graph builds of every kind, with the results read back as a caller
reads them.  Shapes and flags are those of the workloads named in bench.py and
fastkcna_gb300/synth.py (c1 to c5) at their own size or scaled down; the rows
are drawn from the same kinds of mixtures on the GPU.
"""
import math

import numpy as np
import torch

from fastkcna_gb300 import kcna

C1 = dict(K=100, L=100, S=10, R=100, iterations=6, search_L=40, nsg_R=32, search_K=100, massq_S=10)
C2 = dict(K=500, L=500, S=12, R=100, iterations=12, search_L=80, nsg_R=50, search_K=500, massq_S=10, recall=0.99)
C3 = dict(K=200, L=200, S=10, R=100, iterations=6, search_L=40, nsg_R=40, search_K=200, massq_S=10)
C4 = dict(K=500, L=500, S=12, R=100, iterations=6, search_L=80, nsg_R=50, search_K=500, massq_S=10, tau=10.0)
BUILD_KEYS = ("K", "L", "S", "R", "iterations", "search_L", "nsg_R", "search_K", "massq_S", "recall", "tau", "screen",
              "learned_seed", "refine")


def listed():
    return [
        # one query against a small base: the latency of the smallest call
        dict(name="knn_one_query", op="knn", rows="gauss", n=20000, d=32, m=1, k=10),
        # ground truth for a recall curve over a base of full size
        dict(name="knn_ground_truth", op="knn", rows="int", n=1000000, d=128, m=1000, k=100),
        # interactive search: a single query over a small graph
        dict(name="search_one_query", op="search", rows="unit", n=20000, d=32, m=1, k=10, beam=40),
        # batched search at the beam width that the benchmark uses
        dict(name="search_batch", op="search", rows="unit", n=100003, d=128, m=10000, k=10, beam=100),
        # the k-NN graph alone, pools read back (the input of other index builders)
        dict(name="knn_graph", op="knn_graph", rows="unit", n=50021, d=96, recall=0.99,
             **dict(C3, K=140, L=140, S=8, search_K=140, iterations=8)),
        # the rank prune of the pools of a k-NN graph
        dict(name="rank_prune", op="rank_prune", rows="unit", n=150007, d=96, K=64),
        # a small index, plain FP32: launches and host round trips count
        dict(name="build_nsg_20k", op="build", kind="nsg", rows="gauss", n=20000, d=32, **C1),
        # the drop-in FP32 build
        dict(name="build_nsg_fp32_150k", op="build", kind="nsg", rows="int", n=150001, d=128, **C2),
        # the headline build (learned seed, BF16 Gram tiles) at the largest size whose builds repeat closely
        dict(name="build_nsg_learned_400k", op="build", kind="nsg", rows="int", n=400003, d=128, screen=1,
             learned_seed=1, **C2),
        # one layer of a layered index, unit rows, BF16 screening
        dict(name="build_hnsw_layer_150k", op="build", kind="hnsw", rows="unit", n=150007, d=96, screen=1,
             **dict(C3, K=260, L=260, search_K=260)),
        # high dimension, FP8-screened prune
        dict(name="build_taumng_960d", op="build", kind="taumng", rows="abs", n=40009, d=960, screen=1, **C4),
        # angle prune with the learned seed
        dict(name="build_alphapg_200k", op="build", kind="alphapg", rows="int", n=200000, d=128, screen=1,
             learned_seed=1, **C2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["knn", "search", "knn_graph", "rank_prune", "build", "build", "build"])
    if op == "knn":
        rows, d = rng.choice([("gauss", rng.randint(8, 64)), ("int", 128), ("unit", rng.randint(60, 200)),
                              ("abs", rng.randint(200, 960))])
        n = _log(rng, 2000, 400000)
        m = _log(rng, 1, max(1, min(5000, int(6e10 / (n * d)))))
        return dict(op=op, rows=rows, n=n, d=d, m=m, k=rng.randint(1, 200))
    if op == "search":
        beam = rng.randint(10, 200)
        return dict(op=op, rows="unit", n=_log(rng, 5000, 100000), d=rng.randint(20, 160), m=_log(rng, 1, 20000),
                    k=rng.randint(1, 10), beam=beam)
    if op == "knn_graph":
        K = rng.randint(129, 140)
        return dict(op=op, rows="unit", n=_log(rng, 5000, 60000), d=rng.choice([96, 100, 128]),
                    screen=rng.randint(0, 1), recall=0.99, **dict(C3, K=K, L=K, S=8, search_K=K, iterations=8))
    if op == "rank_prune":
        return dict(op=op, rows="unit", n=_log(rng, 10000, 150000), d=rng.choice([96, 128]), K=2 * rng.randint(8, 50))
    kind = rng.choice(["nsg", "hnsw", "taumng", "alphapg"])
    if kind == "taumng":
        d = rng.randint(256, 960)
        n = _log(rng, 3000, 30000)
        # clusters larger than the degree, the threshold at C4's share of the distances
        return dict(op=op, kind=kind, rows="abs", n=n, d=d, clusters=rng.randint(n // 700, n // 90),
                    screen=1 if n > 8000 else rng.randint(0, 1),
                    **dict(C4, search_L=rng.randint(40, 80), nsg_R=rng.randint(24, 60), tau=10.0 * d / 960))
    if kind == "hnsw":
        K = rng.choice([rng.randint(130, 145), rng.randint(260, 300)])
        return dict(op=op, kind=kind, rows="unit", n=_log(rng, 5000, 60000 if K < 200 else 180000), d=rng.choice([96, 100, 128]),
                    screen=rng.randint(0, 1), refine=rng.choice([0, 0, 1]), **dict(C3, K=K, L=K, search_K=K))
    if kind == "alphapg" or rng.random() < 0.6:
        learned = rng.randint(0, 1)
        K = rng.choice([130, 260, 500] if learned else [130, 260])
        lo = 400 * K  # clusters well above K rows
        return dict(op=op, kind=kind, rows="int", n=_log(rng, lo, 300000 if learned else 1.3 * lo), d=128,
                    screen=1 if learned else rng.randint(0, 1), learned_seed=learned,
                    **dict(C2, K=K, L=K, search_K=K, nsg_R=rng.randint(24, 60)))
    K = rng.randint(130, 150)
    return dict(op=op, kind=kind, rows="gauss", n=_log(rng, 3000, 60000), d=rng.randint(8, 64),
                **dict(C1, K=K, L=K, search_K=K))


def _draw_rows(rows, n, d, centres, gen):
    """n rows around the given centres, on the GPU."""
    lab = torch.randint(0, centres.shape[0], (n,), device="cuda", generator=gen)
    out = torch.empty((n, d), device="cuda")
    for s in range(0, n, 1 << 18):
        c = centres[lab[s:s + (1 << 18)]]
        if rows == "int":  # 256 clusters, Laplace noise of scale 12, integers 0..255
            u = torch.rand(c.shape, device="cuda", generator=gen) - 0.5
            x = c - 12.0 * torch.sign(u) * torch.log1p(-2.0 * u.abs().clamp(max=0.4999999))
            x = torch.round(x).clamp_(0.0, 255.0)
        else:
            x = c + {"gauss": 0.1, "unit": 0.35, "abs": 0.2}[rows] * torch.randn(c.shape, device="cuda", generator=gen)
            if rows == "unit":
                x = x / x.norm(dim=1, keepdim=True)
            elif rows == "abs":
                x = x.abs()
        out[s:s + (1 << 18)] = x
    return out


def _data(case, seed):
    """(base rows, query rows) on the GPU, one mixture."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 7919 + 2024)
    rows, d = case["rows"], case["d"]
    if rows == "int":
        cen = 160.0 * torch.rand((256, d), device="cuda", generator=gen)
    elif rows == "gauss":
        cen = 2.0 * torch.rand((16, d), device="cuda", generator=gen) - 1.0
    elif rows == "unit":
        cen = torch.randn((1024, d), device="cuda", generator=gen)
    else:
        cen = (0.5 * torch.randn((case.get("clusters", 512), d), device="cuda", generator=gen)).abs()
    X = _draw_rows(rows, case["n"], d, cen, gen)
    Q = _draw_rows(rows, case["m"], d, cen, gen) if "m" in case else None
    return X, Q


def prepare(case, seed):
    X, Q = _data(case, seed)
    torch.cuda.synchronize()
    ix = kcna.Index(0)
    ix.upload_device(X.data_ptr(), case["n"], case["d"], X.stride(0) * 4)
    s = dict(op=case["op"], ix=ix)
    if Q is not None:
        s.update(Q=Q.cpu().numpy(), k=case["k"])
    if case["op"] == "search":
        ix.build("hnsw", kcna.params(**dict(C3, K=260, L=260, search_K=260), screen=1))
        rng = np.random.default_rng(seed)
        s["beam"] = case["beam"]
        s["init"] = np.stack([rng.choice(case["n"], case["beam"], replace=False) for _ in range(min(case["m"], 64))])
        s["init"] = np.ascontiguousarray(s["init"][np.arange(case["m"]) % s["init"].shape[0]].astype(np.uint32))
    elif case["op"] != "knn":
        s["p"] = kcna.params(**{k: case[k] for k in BUILD_KEYS if k in case})
        s["kind"] = case.get("kind")
        if case["op"] == "rank_prune":
            ix.nndescent(kcna.params(**dict(C3, K=260, L=260, search_K=260), screen=1))
    return s


def run(s):
    ix, op = s["ix"], s["op"]
    if op == "knn":
        return dict(zip(("ids", "dists"), ix.knn_queries(s["Q"], s["k"])))
    if op == "search":
        return dict(zip(("ids", "dists"), ix.search(s["Q"], s["beam"], s["k"], init_ids=s["init"])))
    if op == "knn_graph":
        ix.nndescent(s["p"])
        ids, dists, counts = ix.pools()
        return {"ids": ids.view(np.int32), "dists": dists, "counts": counts.view(np.int32)}
    if op == "rank_prune":
        ix.prune("cagra", s["p"])
    else:
        ix.build(s["kind"], s["p"])
    return {"ids": ix.graph()[0].view(np.int32)}  # rows padded to the width: the degrees are in them


def work(case):
    n, d = case["n"], case["d"]
    if case["op"] == "knn":
        m, k = case["m"], case["k"]
        return {"bytes": 4 * (n * d + m * d + 2 * m * k), "flops": 3 * m * n * d}
    if case["op"] == "search":
        # about three rows of the base are met per beam entry
        m, met = case["m"], 3 * case["beam"]
        return {"bytes": 4 * (min(m * met, n) * d + m * d + 2 * m * case["k"]), "flops": 3 * m * met * d}
    K = case["K"]
    if case["op"] == "rank_prune":
        return {"bytes": n * (8 * K + 4 * (K // 2 + 2)), "flops": n * K * K}
    # about 20 K pairs are met per node until the graph stands
    return {"bytes": 4 * (n * d + n * (2 * K if case["op"] == "knn_graph" else case["nsg_R"] + 9)),
            "flops": 3 * n * 20 * K * d}


def exact(case, seed):
    """64-bit distances of the exact k-NN; the other calls are approximate or
    return whole numbers."""
    if case["op"] != "knn" or case["n"] * case["m"] * case["d"] > 4e11:
        return None
    X, Q = _data(case, seed)
    k, best = case["k"], []
    Xd = X.double()
    xn = (Xd * Xd).sum(1)
    for q in Q.double().split(max(1, int(2e8 // case["n"]))):
        near = torch.topk(xn[None, :] - 2.0 * (q @ Xd.T), min(case["n"], k + 8), dim=1, largest=False).indices
        dist = torch.stack([(Xd[i] - r[None, :]).square().sum(1) for r, i in zip(q, near)])
        best.append(dist.sort(dim=1).values[:, :k])
    return {"ids": None, "dists": torch.cat(best).cpu().numpy()}
