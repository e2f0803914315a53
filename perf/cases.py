"""The calls that a user of this framework makes, as cases to time: counting
(single calls, mode comparisons, batches on root samples, labeled patterns,
host graphs), instance sets, bag relations, device ingest and the plan scorer,
from the smallest graphs it ships to R-MAT 2^22.

A case is a dict of plain values.  prepare() makes the seeded inputs and keeps
what a program keeps (the device graph, the plans, a captured batch, the
scorer); run() is one pass through the public Python entry points.  Data
graphs are the repository's seeded generators' (Chung-Lu with exponent 2.1 to
2.3, R-MAT a=.57 b=.19 c=.19), so another seed is another graph
(or, where the output's size hangs on the graph, other vertex ids).
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "subgraph-enumeration_gb300"))
import sge  # noqa: E402


def _clique(k, drop=()):
    return [(a, b) for a in range(k) for b in range(a + 1, k) if (a, b) not in drop]


# the patterns that the benchmark, the tests and the recorded configurations count
PATTERNS = {
    "triangle": (3, _clique(3)),
    "cycle4": (4, [(0, 1), (1, 2), (2, 3), (0, 3)]),
    "diamond": (4, [(0, 1), (0, 2), (0, 3), (1, 2), (2, 3)]),
    "k4": (4, _clique(4)),
    "house": (5, [(0, 1), (0, 2), (0, 4), (1, 3), (1, 4), (2, 3)]),
    "k5_minus_e": (5, _clique(5, drop=[(3, 4)])),
    "near5clique_8e": (5, [(0, 1), (0, 2), (0, 3), (0, 4), (1, 2), (1, 3), (1, 4), (2, 3)]),
    "k5": (5, _clique(5)),
    "two_triangles_4cycle": (6, [(0, 1), (0, 2), (1, 2), (3, 4), (3, 5), (4, 5), (1, 3), (2, 4)]),
}
# a decomposition in the reference's printed form (global bag last)
BAG_TEXT = {"two_triangles_4cycle": "num bags: 5\n1,0,2\n3,1,2\n3,4,2\n3,4,5\n3,4,1,2\n"}
MODES = {"wcoj": (False, False), "wcoj-u": (False, True), "explore": (True, False), "explore-u": (True, True)}


def listed():
    return [
        # one interactive query on a collaboration-network-sized graph: all latency
        {"name": "diamond_n380", "do": "count", "graph": "chung_lu", "n": 380, "m": 915, "gamma": 2.3, "max_deg": 0,
         "patterns": "diamond", "modes": "wcoj-u"},
        # the four modes of the command line on a mid-sized graph, every root
        {"name": "modes_n7100", "do": "count", "graph": "chung_lu", "n": 7100, "m": 100000, "gamma": 2.1,
         "max_deg": 1000, "patterns": "house,k5_minus_e,near5clique_8e", "modes": "wcoj,wcoj-u,explore,explore-u"},
        # small motifs over every root edge of a web-graph-sized R-MAT
        {"name": "motifs_s18", "do": "count", "graph": "rmat", "scale": 18, "m": 2000003,
         "patterns": "triangle,diamond,k4", "modes": "wcoj-u"},
        # labeled matching (labels uniform over 8 values) over every root edge
        {"name": "labeled_s16", "do": "count", "graph": "rmat", "scale": 16, "m": 700001,
         "patterns": "triangle,diamond,house,k4", "modes": "wcoj-u", "labels": 8},
        # a service's batch of 16 six-vertex patterns on a root sample, replayed
        {"name": "batch16_k6_s20", "do": "batch", "graph": "rmat", "scale": 20, "m": 16000000, "random": 16, "k": 6,
         "e_lo": 11, "e_hi": 13, "pseed": 1000, "roots": 976, "cap": 1000},
        # the benchmark's 78 seven-vertex patterns on R-MAT 2^22 (half its root sample), replayed
        {"name": "batch78_k7_s22", "do": "batch", "graph": "rmat", "scale": 22, "m": 64000000, "random": 78, "k": 7,
         "e_lo": 16, "e_hi": 19, "pseed": 2000, "roots": 488, "cap": 1000},
        # end to end from host memory: upload, checks, index, one count, release
        {"name": "host_s19", "do": "host", "graph": "rmat", "scale": 19, "m": 6000001, "patterns": "triangle,k4",
         "modes": "wcoj-u", "roots": 90000},
        # the sorted instance set (-r) of a pattern
        {"name": "match_set_n7100", "do": "match_set", "graph": "chung_lu", "n": 7100, "m": 100000, "gamma": 2.1,
         "max_deg": 1000, "patterns": "k4"},
        # the bag-relation join: relations built, then a root sample counted through their tries
        {"name": "bags_s14", "do": "bags", "graph": "rmat", "scale": 14, "m": 200003,
         "patterns": "two_triangles_4cycle", "roots": 1500},
        # a data graph from an edge list in device memory (repeats and self-loops among it)
        {"name": "ingest_s20", "do": "ingest", "scale": 20, "m": 16000000},
        # the scorer over the shortlists of a 78-pattern batch (BF16)
        {"name": "score_4992", "do": "score", "rows": 4992},
        # training the scorer on a recorded set (FP32, Adam)
        {"name": "train_1152", "do": "train", "rows": 1152, "epochs": 4, "batch": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _some(rng, names, most):
    return ",".join(rng.sample(names, rng.randint(1, most)))


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    do = rng.choice(["small", "modes", "motifs", "labeled", "batch6", "batch7", "host", "match_set", "bags", "ingest",
                     "score", "train"])
    if do in ("small", "modes", "match_set"):
        n = _log(rng, 300, 1500) if do == "small" else _log(rng, 1200, 7100)
        c = {"do": "count", "graph": "chung_lu", "n": n, "m": round(n * rng.uniform(2.4, 6 if do == "small" else 14)),
             "gamma": rng.choice([2.1, 2.2, 2.3]), "max_deg": 0 if do == "small" else min(1000, n // 4)}
        if do == "match_set":
            return dict(c, do="match_set", patterns=rng.choice(["triangle", "k4"]))
        names = ["triangle", "diamond", "cycle4", "house", "k5_minus_e", "near5clique_8e", "k4", "k5"]
        return dict(c, patterns=_some(rng, names, 1 if do == "small" else 3), modes=_some(rng, list(MODES), 2))
    if do in ("motifs", "labeled", "host"):
        s = rng.randint(11, {"motifs": 18, "labeled": 16, "host": 19}[do])
        c = {"do": "count", "graph": "rmat", "scale": s, "m": round((1 << s) * rng.uniform(5, 11))}
        if do == "motifs":
            return dict(c, patterns=_some(rng, ["triangle", "diamond", "k4"], 3), modes=rng.choice(["wcoj", "wcoj-u"]))
        if do == "labeled":
            return dict(c, patterns=_some(rng, ["triangle", "diamond", "house", "k4"], 4), modes="wcoj-u",
                        labels=rng.randint(8, 16))
        return dict(c, do="host", patterns=_some(rng, ["triangle", "diamond", "k4"], 2), modes="wcoj-u",
                    roots=min(c["m"], _log(rng, 5000, 90000)))
    if do == "batch6":
        s = rng.randint(15, 20)
        return {"do": "batch", "graph": "rmat", "scale": s, "m": round((1 << s) * rng.uniform(9, 15.2)),
                "random": rng.randint(3, 16), "k": 6, "e_lo": 11, "e_hi": 13, "pseed": 1000, "roots": _log(rng, 60, 976),
                "cap": rng.randint(300, 1000)}
    if do == "batch7":
        s = rng.randint(16, 22)
        return {"do": "batch", "graph": "rmat", "scale": s, "m": round((1 << s) * rng.uniform(9, 15.2)),
                "random": rng.randint(8, 78), "k": 7, "e_lo": 16, "e_hi": 19, "pseed": 2000,
                "roots": _log(rng, 40, 400), "cap": rng.randint(300, 1000)}
    if do == "bags":
        s = rng.randint(10, 14)
        return {"do": "bags", "graph": "rmat", "scale": s, "m": round((1 << s) * rng.uniform(6, 12)),
                "patterns": "two_triangles_4cycle", "roots": _log(rng, 100, 1500)}
    if do == "ingest":
        s = rng.randint(13, 20)
        return {"do": "ingest", "scale": s, "m": round((1 << s) * rng.uniform(3, 15.2))}
    if do == "score":
        return {"do": "score", "rows": _log(rng, 61, 4992)}
    return {"do": "train", "rows": _log(rng, 200, 1152), "epochs": rng.randint(1, 4), "batch": rng.choice([64, 100, 128])}


# ------------------------------------------------------------------- inputs ----
def _pattern(name):
    k, edges = PATTERNS[name]
    return sge.PatternGraph.from_edges(k, edges)


def _root_first(k, edges):
    """One symmetry sequence and one root edge per pattern (the edge with the
    largest degree sum first, then falling degrees), as a program that counts
    root samples fixes them so that its plans agree on the sample."""
    deg = np.bincount(edges.reshape(-1), minlength=k)
    a, b = max(((int(x), int(y)) for x, y in edges), key=lambda e: (deg[e[0]] + deg[e[1]], -min(e), -max(e)))
    if deg[b] > deg[a]:
        a, b = b, a
    return [a, b] + sorted((v for v in range(k) if v not in (a, b)), key=lambda v: (-deg[v], v)), [a, b]


def _rmat_edges(scale, m, seed):
    """m R-MAT draws in device memory, repeats and self-loops included, with
    the vertex ids shuffled by the seed (so every seed has as many edges)."""
    gen = torch.Generator(device="cuda").manual_seed(m)
    e = torch.zeros(m, 2, dtype=torch.int32, device="cuda")
    for _ in range(scale):
        r = torch.rand(m, device="cuda", generator=gen)
        e[:, 0] = e[:, 0] * 2 + (r >= 0.76)
        e[:, 1] = e[:, 1] * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    ids = torch.randperm(1 << scale, generator=torch.Generator().manual_seed(seed)).to(device="cuda", dtype=torch.int32)
    return ids[e.long()].contiguous()


def _engine(case, seed):
    if case["graph"] == "rmat":
        return sge.Engine.rmat_device(case["scale"], case["m"], seed=seed)
    if case["do"] == "match_set":  # one graph with its vertex ids shuffled by the seed: every seed has as many rows
        g = sge.gen_chung_lu(case["n"], case["m"], case["gamma"], case["max_deg"], seed=1)
        ids = np.random.default_rng(seed).permutation(case["n"]).astype(np.uint32)
        return sge.Engine(sge.DataGraph.from_edges(ids[g.edge_array()], case["n"]))
    return sge.Engine(sge.gen_chung_lu(case["n"], case["m"], case["gamma"], case["max_deg"], seed=seed))


def _sample(case):
    """Root-sample options: about case["roots"] undirected root edges."""
    o = {}
    if case.get("roots", case["m"]) < case["m"]:
        o = {"root_stride": case["m"] // case["roots"], "root_offset": 1}
    if "cap" in case:
        o["root_max_degree"] = case["cap"]
    return o


def _scorer(case, seed):
    """Scorer weights (64 -> 128 -> 128 -> 1, Glorot-uniform) and plan features
    (64 values in [0, 1], two fifths of them 0) with log-runtime labels."""
    rng = np.random.default_rng(seed)
    h, d = 128, 64

    def uni(o, i):
        return rng.uniform(-1, 1, (o, i)) * math.sqrt(6 / (o + i))
    p = np.concatenate([uni(h, d).ravel(), rng.normal(0, 0.05, h), uni(h, h).ravel(), rng.normal(0, 0.05, h),
                        uni(1, h).ravel(), rng.normal(0, 0.05, 1)]).astype(np.float32)
    x = (rng.random((case["rows"], d)) * (rng.random((case["rows"], d)) < 0.6)).astype(np.float32)
    t = (rng.normal(1.5, 2.0, case["rows"])).astype(np.float32)
    return p, x, t


def prepare(case, seed):
    do = case["do"]
    if do == "ingest":
        return {"do": do, "n": 1 << case["scale"], "edges": _rmat_edges(case["scale"], case["m"], seed)}
    if do in ("score", "train"):
        p, x, t = _scorer(case, seed)
        mlp = sge.MLP(64, 128, seed=0)
        mlp.set_params(p)
        return {"do": do, "mlp": mlp, "p": p, "x": x, "t": t, "case": case}
    eng = _engine(case, seed)
    s = {"do": do, "eng": eng, "opts": _sample(case)}
    if do == "match_set":
        s["pattern"] = _pattern(case["patterns"])
    elif do == "bags":
        s["pattern"], s["text"] = _pattern(case["patterns"]), BAG_TEXT[case["patterns"]]
        s["plan"], _ = sge.plan_from_reference(s["pattern"], s["text"], eng, iep=True)
    elif do == "batch":
        plans = []
        for i in range(case["random"]):
            p = sge.PatternGraph.random(case["k"], case["e_lo"] + i % (case["e_hi"] - case["e_lo"] + 1),
                                        case["pseed"] + i)
            seq, root = _root_first(p.k, p.edges)
            plans.append(sge.plan(p, eng, symmetry_seq=seq, root_edge=root))
        s["batch"] = sge.Batch(eng, plans, **s["opts"])
    else:
        labels = None
        if case.get("labels"):
            rng = np.random.default_rng(seed)
            eng.set_labels(rng.integers(0, case["labels"], 1 << case["scale"]).astype(np.uint32))
            labels = []
        s["plans"] = []
        for mode in case["modes"].split(","):
            expl, iep = MODES[mode]
            for name in case["patterns"].split(","):
                p = _pattern(name)
                lab = None
                if labels is not None:
                    lab = [int(v) for v in rng.integers(0, case["labels"], p.k)]
                    labels.append(lab)
                s["plans"].append(sge.plan(p, eng, iep=iep, exploration=expl, labels=lab))
        s["labels"] = labels
        if do == "host":
            s["graph"] = eng.graph
            eng.close()
            del s["eng"]
    return s


# --------------------------------------------------------------------- runs ----
def _counts(c):
    return np.array(c, dtype=np.uint64).view(np.int64)


def run(s):
    do = s["do"]
    if do == "count":
        c, inst, _ = s["eng"].count(s["plans"], labels=s["labels"], **s["opts"])
        return {"counts": _counts(c), "instances": _counts(inst)}
    if do == "batch":
        c, inst, _ = s["batch"].run()
        return {"counts": _counts(c), "instances": _counts(inst)}
    if do == "host":
        c, _ = sge.count_host(s["graph"], s["plans"], **s["opts"])
        return {"counts": _counts(c)}
    if do == "match_set":
        return s["eng"].match_set(s["pattern"]).view(np.int32)
    if do == "bags":
        with s["eng"].bags(s["pattern"], s["text"]) as bags:
            info = bags.info()
            c, inst, _ = s["eng"].count([s["plan"]], bags=[bags], **s["opts"])
        return {"counts": _counts(c), "instances": _counts(inst), "rows": info["rows"]}
    if do == "ingest":
        e = s["edges"]
        with sge.Engine.from_device_edges(e.data_ptr(), e.shape[0], s["n"]) as eng:
            off, nb = eng.csr()
        return {"offsets": off.view(np.int32), "nbrs": nb.view(np.int32)}
    if do == "score":
        return s["mlp"].forward(s["x"], bf16=True)
    c, mlp = s["case"], s["mlp"]
    mlp.set_params(s["p"])
    loss = mlp.train(s["x"], s["t"], epochs=c["epochs"], batch=c["batch"], lr=2e-3, seed=7)
    return {"loss": np.float32(loss), "params": mlp.get_params()}


def work(case):
    """Bytes: the inputs of the call once and its outputs once.  A root sample
    needs two lists of at most `cap` (or of the mean length) per root.
    flops: the scorer's contractions (a counting call is integer work)."""
    do = case["do"]
    if do in ("score", "train"):
        fwd = 2 * case["rows"] * (64 * 128 + 128 * 128 + 128)
        if do == "score":
            return {"bytes": 4 * case["rows"] * 65 + 4 * 24961, "flops": fwd}
        return {"bytes": case["epochs"] * 4 * case["rows"] * 65 + 2 * 4 * 24961, "flops": 3 * case["epochs"] * fwd}
    n = case["n"] if "n" in case else 1 << case["scale"]
    csr = 4 * (n + 1) + 8 * case["m"]
    if do == "ingest":
        return {"bytes": 8 * case["m"] + csr, "flops": 0}
    if do == "host":
        return {"bytes": csr, "flops": 0}
    if do == "match_set":
        return {"bytes": csr + 16 * case["m"], "flops": 0}
    if "roots" in case and do != "bags":
        csr = min(csr, case["roots"] * 2 * 4 * case.get("cap", 2 * case["m"] // n))
    if "labels" in case:
        csr += 4 * n
    return {"bytes": csr, "flops": 0}


# -------------------------------------------------------------------- exact ----
def _forward64(p, x):
    h, d = 128, 64
    o = np.cumsum([0, h * d, h, h * h, h, h, 1])
    w1, b1, w2, b2, w3, b3 = (p[o[i]:o[i + 1]] for i in range(6))
    a1 = np.maximum(x @ w1.reshape(h, d).T + b1, 0)
    a2 = np.maximum(a1 @ w2.reshape(h, h).T + b2, 0)
    return a1, a2, a2 @ w3 + b3, w2.reshape(h, h), w3


def _mix(z):
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) % 2 ** 64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) % 2 ** 64
    return z ^ (z >> 31)


def _train64(case, p, x, t):
    """Adam on 0.5 mean (f(x)-t)^2, each epoch in the order of a Fisher-Yates
    shuffle drawn from splitmix64 (seed 7), in 64 bits."""
    golden = 0x9E3779B97F4A7C15
    state = _mix((7 ^ 0x5347454E5347454E) + golden & 2 ** 64 - 1)
    p, n = p.copy(), len(x)
    m, v, step = np.zeros_like(p), np.zeros_like(p), 0
    order = list(range(n))
    for _ in range(case["epochs"]):
        for i in range(n - 1, 0, -1):
            state = (state + golden) % 2 ** 64
            j = _mix(state) * (i + 1) >> 64
            order[i], order[j] = order[j], order[i]
        losses = []
        for s in range(0, n, case["batch"]):
            ids = order[s:s + case["batch"]]
            xb, tb = x[ids], t[ids]
            a1, a2, y, w2, w3 = _forward64(p, xb)
            losses.append(0.5 * np.mean((y - tb) ** 2))
            dy = (y - tb) / len(ids)
            d2 = np.outer(dy, w3) * (a2 > 0)
            d1 = (d2 @ w2) * (a1 > 0)
            g = np.concatenate([(d1.T @ xb).ravel(), d1.sum(0), (d2.T @ a1).ravel(), d2.sum(0), a2.T @ dy, [dy.sum()]])
            step += 1
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p -= 2e-3 * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
    return {"loss": np.float64(np.mean(losses)), "params": p}


def exact(case, seed):
    """The scorer's outputs in 64 bits; the other cases return whole numbers."""
    if case["do"] not in ("score", "train"):
        return None
    p, x, t = (a.astype(np.float64) for a in _scorer(case, seed))
    if case["do"] == "score":
        return _forward64(p, x)[2]
    return _train64(case, p, x, t)
