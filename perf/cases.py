"""The work that users of this framework have it do, as timed cases.

Every case goes through the package's public entry points: batched searches
of a resident index (device buffers or host buffers), the training of the
early-exit network, and the construction of a graph.  The sizes are those of
the workloads in song_gb300/datasets.py and of bench.py: 15k x 16 cosine
vectors, 1M x 128 integer-valued L2 vectors with 524,288 entry vertices,
960-d cosine rows and 256-d L2 rows (fewer of these two, still more than the
L2 cache holds), queue bounds from 10 to 1000, batches from one query to
10,000.

An index is a handle that a program makes once and then searches with one
batch of queries after another, so a process keeps one handle per base set
and settings; the queries, training samples and vectors to insert are drawn
from the seed.
"""
import math

import numpy as np
import torch

import song_gb300 as S
from song_gb300 import datasets as D

# Base sets: workload of song_gb300/datasets.py, vectors taken from it, its
# entry points (count, coarse, probes, starts); "flat" entry points: the
# nearest of 4096.
SETS = {
    "letters": {"workload": "small-15k-16d-cos", "n": 15_000, "two": (4096, 128, 4, 4)},
    "scale": {"workload": "scale-1m-128d-l2", "n": 1_000_000, "two": (524_288, 4096, 4, 4)},
    "wide": {"workload": "precision-1m-960d-cos", "n": 60_000, "two": (60_000, 1024, 8, 8)},
    "mid": {"workload": "learned-3m-256d-l2", "n": 150_000, "two": (65_536, 1024, 4, 4)},
}
FLAT = (4096, 4)  # entry vertices and starts of the flat choice
BATCH_DIV = 64


def _search(name, base, nq, pq, k, start="two", storage="f32", **more):
    return {"name": name, "op": "search", "base": base, "nq": nq, "pq": pq, "k": k, "start": start,
            "storage": storage, **more}


def listed():
    return [
        # one query at a time against a small base: a request path where latency and launches count
        _search("letters-1-query", "letters", 1, 50, 10, start="vertex0"),
        # the demo batch on the small base, the reference's start
        _search("letters-5000", "letters", 5000, 100, 10, start="vertex0"),
        # one query against the large base from its entry points
        _search("scale-1-query", "scale", 1, 100, 10),
        # a service's mixed batch with host buffers: copy in, search, copy out
        _search("scale-host-137", "scale", 137, 200, 100, host=True),
        # the headline batch: top-10 at recall 0.95
        _search("scale-10000-top10", "scale", 10_000, 43, 10),
        # the same base at recall 0.95 of the top 100
        _search("scale-10000-top100", "scale", 10_000, 150, 100),
        # the reference's own semantics: every query from vertex 0, the queue bound that recall 0.95 needs there
        _search("scale-vertex0-pq1000", "scale", 10_000, 1000, 10, start="vertex0"),
        # 960-d rows kept in BF16 with the FP32 re-rank
        _search("wide-bf16-1000", "wide", 1000, 75, 10, storage="bf16"),
        # 256-d rows kept in FP8 with the FP32 re-rank, an odd batch
        _search("mid-fp8-2501", "mid", 2501, 100, 10, storage="fp8"),
        # the early-exit network at work in the search
        _search("mid-exit-10000", "mid", 10_000, 150, 10, exit=True),
        # training of that network: forward, backward and Adam over traced hops
        {"name": "train-300k", "op": "train", "n": 300_001, "batch": 8192, "epochs": 6},
        # a graph for new vectors
        {"name": "build-20k", "op": "build", "n": 20_000, "dim": 128, "metric": "l2", "shift": 5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["search"] * 8 + ["train", "build"])
    if op == "train":
        return {"op": "train", "n": _log_int(rng, 20_000, 300_000), "batch": rng.choice([1024, 4096, 8192, 5000]),
                "epochs": rng.randint(2, 6)}
    if op == "build":
        return {"op": "build", "n": _log_int(rng, 3000, 15_000), "dim": rng.choice([16, 25, 64, 100, 128]),
                "metric": rng.choice(["l2", "ip", "cos"]), "shift": rng.choice([4, 5])}
    base = rng.choice(["letters", "scale", "scale", "scale", "wide", "mid"])
    kind = rng.choice(["plain", "plain", "storage", "multi", "exit"])
    start = rng.choice(["vertex0", "two", "two"] + (["flat"] if base in ("letters", "mid") else []))
    storage = rng.choice(["bf16", "fp8", "bits"] if base == "letters" else ["bf16", "fp8"]) if kind == "storage" else "f32"
    pq = _log_int(rng, 10, 500 if base == "wide" else 1000)
    nq = _log_int(rng, 1, 1000 if base == "wide" else 10_000)
    c = {"op": "search", "base": base, "nq": nq, "pq": pq, "k": min(pq, rng.choice([1, 10, 10, 100])),
         "start": start, "storage": storage}
    if kind == "exit":
        c["exit"] = True
    if kind == "multi":
        c["probes"], c["finish_cnt"], c["double_check"] = rng.choice([(2, 1, True), (4, 1, True), (1, 2, False)])
    if rng.random() < 0.25:
        c["host"] = True
    return c


# ---------------------------------------------------------------------------
# what a program has in hand
# ---------------------------------------------------------------------------

_bases = {}
_indexes = {}


def _base(name):
    """Vectors and graph of a base set (host arrays), made once."""
    if name not in _bases:
        w = D.WORKLOADS[SETS[name]["workload"]]
        data = D.base_vectors(w, SETS[name]["n"])
        graph = S.graph_build_gpu(data, w.metric, w.shift, w.search_degree, w.fixed_degree, 150, batch_div=BATCH_DIV)
        _bases[name] = (w, data, graph)
    return _bases[name]


def _exit_weights():
    """A network that fires once the top-k has stood still for about 32 hops."""
    p = np.zeros(S.MLP_PARAMS, dtype=np.float32)
    p[2] = 1.0             # W1[0][2]: log2(1 + hops since the last change) / 10
    p[192] = 1.0           # W2[0][0]
    p[1248] = 20.0         # w3[0]
    p[1280] = -10.0        # b3
    return p


def _index(c):
    multi = (c.get("probes", 1), c.get("finish_cnt", 1), c.get("double_check", False))
    key = (c["base"], c["start"], c["storage"], multi, c.get("exit", False))
    if key not in _indexes:
        w, data, graph = _base(c["base"])
        ix = S.Index(graph, data, w.shift, w.metric, storage=c["storage"])
        if c["storage"] == "bits":
            ix.set_hash_planes(S.hash_planes(w.dim))
        if c["start"] == "two":
            count, coarse, probes, starts = SETS[c["base"]]["two"]
            ix.set_entries(S.sample_entries(SETS[c["base"]]["n"], count, shuffle=True), starts=starts, coarse=coarse, probes=probes)
        elif c["start"] == "flat":
            ix.set_entries(S.sample_entries(SETS[c["base"]]["n"], FLAT[0]), starts=FLAT[1])
        ix.set_multiprobe(*multi)
        if c.get("exit"):
            ix.set_early_exit(_exit_weights(), 0.0, min_hops=8, every=4)
        _indexes[key] = ix
    return _indexes[key]


def _prepare_search(c, seed):
    ix = _index(c)
    w = D.WORKLOADS[SETS[c["base"]]["workload"]]
    q = D.query_vectors(w, nq=c["nq"], seed=1000 + seed)
    s = {"op": "search", "ix": ix, "pq": c["pq"], "k": c["k"], "nq": c["nq"], "host": bool(c.get("host"))}
    if s["host"]:
        s["q"] = q
    else:
        s["q"] = torch.from_numpy(q).cuda()
        s["out"] = torch.empty((c["nq"], c["k"]), dtype=torch.int64, device="cuda")
    return s


def _train_inputs(c, seed):
    """Traced hops: features of the ranges the search writes, labels that
    mostly follow the hops since the last change."""
    rng = np.random.default_rng(seed)
    n = c["n"]
    x = np.empty((n, 5), dtype=np.float32)
    hops = rng.integers(1, 400, n)
    since = (rng.random(n) * hops).astype(np.int64)
    x[:, 0] = np.log2(1 + hops) * 0.1
    x[:, 1] = np.log1p(rng.exponential(0.2, n))
    x[:, 2] = np.log2(1 + since) * 0.1
    x[:, 3] = rng.normal(0.0, 0.3, n)
    x[:, 4] = np.log2(1 + hops * rng.integers(4, 24, n)) * 0.1
    y = (x[:, 2] + 0.4 * x[:, 3] + 0.1 * rng.standard_normal(n) > 0.5).astype(np.float32)
    wt = np.where(y > 0.5, 1.0, 4.0).astype(np.float32)
    perm = np.concatenate([rng.permutation(n) for _ in range(c["epochs"])]).astype(np.int32)
    return x, y, wt, perm, S.mlp_init(seed & 0xffff)


def prepare(case, seed):
    if case["op"] == "search":
        return _prepare_search(case, seed)
    if case["op"] == "train":
        x, y, wt, perm, p = (torch.from_numpy(a).cuda() for a in _train_inputs(case, seed))
        return {"op": "train", "x": x, "y": y, "w": wt, "perm": perm, "init": p, "n": case["n"],
                "batch": case["batch"], "epochs": case["epochs"]}
    rng = np.random.default_rng(seed)
    centers = rng.uniform(0.0, 255.0, (64, case["dim"])).astype(np.float32)
    x = centers[rng.integers(0, 64, case["n"])] + 20 * rng.standard_normal((case["n"], case["dim"]), dtype=np.float32)
    # host vectors: the call takes host arrays and writes the host graph that is then saved
    return {"op": "build", "x": np.clip(np.rint(x), 0, 255).astype(np.float32), "metric": case["metric"],
            "shift": case["shift"]}


LR = 2e-3


def run(s):
    if s["op"] == "search":
        if s["host"]:
            return s["ix"].search(s["q"], s["pq"], s["k"]).view(np.int64)
        s["ix"].search_device(s["q"].data_ptr(), s["nq"], s["pq"], s["k"], s["out"].data_ptr(),
                              stream=torch.cuda.current_stream().cuda_stream)
        return s["out"]
    if s["op"] == "train":
        params = s["init"].clone()
        loss = torch.empty(s["epochs"], dtype=torch.float32, device="cuda")
        S.mlp_train_device(s["x"].data_ptr(), s["y"].data_ptr(), s["w"].data_ptr(), s["n"], s["perm"].data_ptr(),
                           s["epochs"], s["batch"], LR, params.data_ptr(), loss.data_ptr(),
                           torch.cuda.current_stream().cuda_stream)
        return {"params": params, "loss": loss}
    fixed = (1 << s["shift"]) - 1
    return S.graph_build_gpu(s["x"], s["metric"], s["shift"], fixed // 2, fixed, 150,
                             batch_div=BATCH_DIV).view(np.int64)


# ---------------------------------------------------------------------------
# work and exact values
# ---------------------------------------------------------------------------

def _row_bytes(dim, storage):
    return {"f32": 4 * dim, "bf16": 2 * dim, "fp8": dim + 4, "bits": 32}[storage]


def work(case):
    if case["op"] == "search":
        w = D.WORKLOADS[SETS[case["base"]]["workload"]]
        nq, pq = case["nq"], case["pq"]
        # the list of pq vertices has to fill, so at least pq vertices are
        # expanded, each bringing some vertices not seen before
        if case.get("exit"):
            pq = min(pq, EXIT_HOPS)
        evals = _evals(case["base"], pq)
        per_query = evals * _row_bytes(w.dim, case["storage"]) + pq * 4 * (1 << w.shift) + 4 * w.dim + 8 * case["k"]
        flops = evals * 3 * w.dim
        heads = {"two": SETS[case["base"]]["two"][1], "flat": FLAT[0], "vertex0": 0}[case["start"]]
        return {"bytes": nq * per_query + heads * 4 * w.dim, "flops": nq * (flops + heads * 2 * w.dim)}
    if case["op"] == "train":
        steps = case["epochs"] * -(-case["n"] // case["batch"])
        return {"bytes": case["epochs"] * case["n"] * (7 + 1) * 4 + steps * 1281 * 4 * 6,
                "flops": case["epochs"] * case["n"] * 6 * (5 * 32 + 32 * 32 + 32)}
    # every insertion reads the vertices that its search of result size 150 cannot do without
    n, dim = case["n"], case["dim"]
    return {"bytes": n * (150 * (4 * dim + (4 << case["shift"])) + 4 * dim + (8 << case["shift"])),
            "flops": n * 150 * 3 * dim}


# distances computed per query at these queue bounds, by the search's own
# counters, from the nearest entry points (the least work of the two starts)
EVALS_PQ = (10, 43, 100, 200, 400, 1000)
EVALS = {
    "letters": (109, 320, 515, 587, 576, 1507),
    "scale": (268, 914, 1673, 2326, 2129, 1697),
    "wide": (226, 430, 216, 635, 1214, 2534),
    "mid": (203, 217, 495, 1329, 2542, 5133),
}
EXIT_HOPS = 40  # with the early exit, a search of any bound ends after about this many expansions


def _evals(base, pq):
    return float(np.interp(math.log(pq), [math.log(v) for v in EVALS_PQ], EVALS[base]))


def exact(case, seed):
    if case["op"] != "train":
        return None  # ids
    x, y, wt, perm, p = _train_inputs(case, seed)
    x, y, wt, p = x.astype(np.float64), y.astype(np.float64), wt.astype(np.float64), p.astype(np.float64)
    n, batch = case["n"], case["batch"]
    m, v, t, losses = np.zeros_like(p), np.zeros_like(p), 0, []
    for ep in range(case["epochs"]):
        order, total, steps = perm[ep * n:(ep + 1) * n], 0.0, 0
        for a in range(0, n, batch):
            i = order[a:a + batch]
            xi, yi, wi = x[i], y[i], wt[i]
            w1, b1, w2, b2, w3, b3 = (p[:160].reshape(32, 5), p[160:192], p[192:1216].reshape(32, 32), p[1216:1248],
                                      p[1248:1280], p[1280])
            a1 = xi @ w1.T + b1
            h1 = np.maximum(a1, 0)
            a2 = h1 @ w2.T + b2
            h2 = np.maximum(a2, 0)
            z = h2 @ w3 + b3
            wsum = wi.sum()
            total += (wi * (np.maximum(z, 0) + np.log1p(np.exp(-np.abs(z))) - yi * z)).sum() / wsum
            steps += 1
            dz = wi * (1 / (1 + np.exp(-z)) - yi) / wsum
            da2 = (dz[:, None] * w3) * (a2 > 0)
            da1 = (da2 @ w2) * (a1 > 0)
            g = np.concatenate([(da1.T @ xi).ravel(), da1.sum(0), (da2.T @ h1).ravel(), da2.sum(0), h2.T @ dz,
                                [dz.sum()]])
            t += 1
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p = p - LR * (m / (1 - 0.9 ** t)) / (np.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
        losses.append(total / steps)
    return {"params": p, "loss": np.array(losses)}
