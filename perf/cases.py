"""Cases that stand for the work a user has this framework do, measured through its public API.

A case is one call sequence of a user's program: a whole IMM query (sampling, martingale rounds,
seed selection), the sampler or the selection alone, a batch of queries, the forward spread of a
seed set, or the upload of a host graph followed by its query.  Graphs are R-MAT (a, b, c = 0.57,
0.19, 0.19) or Erdos-Renyi with weighted-cascade, uniform or LT-normalised weights, drawn from the
case's seed; sizes follow bench.py's workloads and the test suite.

Every output is a whole number (seeds, counts, sets, reached vertices) or a ratio of two (f, a mean
count): the sampler's draws are a counter-based function of (seed, set, edge), so any correct
implementation of them returns the same bits, and the tolerance is "exact" throughout.  A 64-bit
recomputation of the floating outputs would be those same ratios, so there is no exact().
"""
import math

import numpy as np
import torch

import ripples_b200 as rb

WEIGHTS = {"uniform": rb.WEIGHTS_UNIFORM, "wc": rb.WEIGHTS_WC, "lt": rb.WEIGHTS_LT_NORMALIZED}
TIES = {"ref": rb.TIE_REF_HEAP, "lowest": rb.TIE_LOWEST_ID}
SAMPLERS = {"auto": rb.SAMPLER_AUTO, "plain": rb.SAMPLER_PLAIN, "fused": rb.SAMPLER_FUSED}


def listed():
    return [
        # The benchmark's smallest query: a graph that fits L2, sets of a third of its vertices.
        {"name": "imm_ic_rmat14", "kind": "imm", "graph": "rmat", "n": 1 << 14, "draws": 1 << 18,
         "model": "IC", "weights": "uniform", "hi": 0.1, "k": 20, "eps": 0.5, "tie": "ref"},
        # The LT workload of the benchmark: random walks, and picks with the reference's tie-break.
        {"name": "imm_lt_rmat20", "kind": "imm", "graph": "rmat", "n": 1 << 20, "draws": 16 << 20,
         "model": "LT", "weights": "lt", "hi": 1.0, "k": 50, "eps": 0.3, "tie": "ref"},
        # The headline workload: weighted cascade on 2^24 vertices, tight epsilon, 100 seeds.
        {"name": "imm_wc_rmat24", "kind": "imm", "graph": "rmat", "n": 1 << 24, "draws": 32 << 24,
         "model": "IC", "weights": "wc", "hi": 1.0, "k": 100, "eps": 0.13, "tie": "ref"},
        # An ordinary query at sizes that are no power of two, with picks on the device (lowest id).
        {"name": "imm_wc_er_lowest", "kind": "imm", "graph": "er", "n": 300007, "draws": 3600091,
         "model": "IC", "weights": "wc", "hi": 1.0, "k": 77, "eps": 0.3, "tie": "lowest"},
        # A supercritical graph of the serving workload: sets hold a large share of the graph.
        {"name": "imm_super_rmat18", "kind": "imm", "graph": "rmat", "n": 1 << 18,
         "draws": 16 << 18, "model": "IC", "weights": "uniform", "hi": 0.1, "k": 20, "eps": 0.5,
         "tie": "lowest"},
        # The fused multi-colour sampler, asked for by name (--gpu-batch-size), and its set counts.
        {"name": "sample_fused128", "kind": "sample", "graph": "rmat", "n": 1 << 14,
         "draws": 1 << 18, "model": "IC", "weights": "uniform", "hi": 0.05, "sampler": "fused",
         "colors": 128, "sets": 20011, "export": False},
        # A small GenerateRRRSets into host sets, as the drop-in gives them to the caller (LT walks).
        {"name": "generate_lt_rmat15", "kind": "sample", "graph": "rmat", "n": 1 << 15,
         "draws": 12 << 15, "model": "LT", "weights": "lt", "hi": 1.0, "sampler": "auto",
         "colors": 64, "sets": 4001, "export": True},
        # FindMostInfluentialSet alone on resident sets, the reference's tie-break, many seeds.
        {"name": "select_ref_rmat22", "kind": "select", "graph": "rmat", "n": 1 << 22,
         "draws": 16 << 22, "model": "IC", "weights": "wc", "hi": 1.0, "sets": 400000, "k": 200,
         "tie": "ref"},
        # Small and middle queries of many graphs run as one continuous batch.
        {"name": "batch_12", "kind": "batch", "graphs": 6, "n": 4099, "n_hi": 65537, "deg": 4,
         "deg_hi": 32, "queries": 12, "k": 10, "k_hi": 200, "eps": 0.1, "eps_hi": 0.5},
        # The simulator: spread of the 50 largest hubs, replica by replica, under IC ...
        {"name": "spread_ic_rmat20", "kind": "spread", "graph": "rmat", "n": 1 << 20,
         "draws": 16 << 20, "model": "IC", "weights": "uniform", "hi": 0.1, "k": 50,
         "replicas": 1500},
        # ... and under LT, which also reads the in-lists of the vertices that are tried.
        {"name": "spread_lt_rmat16", "kind": "spread", "graph": "rmat", "n": 1 << 16,
         "draws": 12 << 16, "model": "LT", "weights": "lt", "hi": 1.0, "k": 20, "replicas": 2000},
        # The imm tool's whole run after reading its file: a host graph uploaded, queried, dropped.
        {"name": "upload_imm_lt_rmat18", "kind": "upload", "graph": "rmat", "n": 1 << 18,
         "draws": 16 << 18, "model": "LT", "weights": "lt", "hi": 1.0, "k": 50, "eps": 0.5,
         "tie": "ref"},
    ]


def _between(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _drawn_graph(rng, lo, hi, deg_lo, deg_hi):
    n = _between(rng, lo, hi)
    if rng.random() < 0.5:
        return {"graph": "er", "n": n, "draws": n * rng.randint(deg_lo, deg_hi) + rng.randint(0, n)}
    scale = max(1, int(round(math.log2(n))))
    return {"graph": "rmat", "n": 1 << scale,
            "draws": (rng.randint(deg_lo, deg_hi) << scale) + rng.randint(0, 1 << scale)}


def draw(rng):
    kind = rng.choice(["imm_wc", "imm_wc", "imm_lt", "imm_lt", "imm_uniform", "sample_wc",
                       "sample_lt", "generate", "sample_fused", "select", "batch", "spread_ic",
                       "spread_lt", "upload"])
    k = _between(rng, 5, 200)
    eps = round(rng.uniform(0.13, 0.5), 3)
    tie = rng.choice(["ref", "lowest"])
    if kind == "imm_wc":
        return {"kind": "imm", **_drawn_graph(rng, 1 << 12, 1 << 22, 4, 32), "model": "IC",
                "weights": "wc", "hi": 1.0, "k": k, "eps": eps, "tie": tie}
    if kind == "imm_lt":
        return {"kind": "imm", **_drawn_graph(rng, 1 << 12, 1 << 21, 4, 32), "model": "LT",
                "weights": "lt", "hi": 1.0, "k": k, "eps": eps, "tie": tie}
    if kind == "imm_uniform":
        return {"kind": "imm", **_drawn_graph(rng, 1 << 12, 1 << 18, 4, 16), "model": "IC",
                "weights": "uniform", "hi": round(rng.uniform(0.02, 0.1), 3),
                "k": min(k, 50), "eps": max(eps, 0.4), "tie": tie}
    if kind == "sample_wc":
        return {"kind": "sample", **_drawn_graph(rng, 1 << 12, 1 << 21, 4, 32), "model": "IC",
                "weights": "wc", "hi": 1.0, "sampler": rng.choice(["auto", "plain"]), "colors": 64,
                "sets": _between(rng, 100, 200000), "export": False}
    if kind == "sample_lt":
        return {"kind": "sample", **_drawn_graph(rng, 1 << 12, 1 << 21, 4, 32), "model": "LT",
                "weights": "lt", "hi": 1.0, "sampler": "auto", "colors": 64,
                "sets": _between(rng, 100, 200000), "export": False}
    if kind == "generate":
        scale = rng.randint(12, 18)
        return {"kind": "sample", "graph": "rmat", "n": 1 << scale,
                "draws": (rng.randint(4, 32) << scale) + rng.randint(0, 1 << scale), "model": "LT",
                "weights": "lt", "hi": 1.0, "sampler": "auto", "colors": 64,
                "sets": _between(rng, 100, 30000), "export": True}
    if kind == "sample_fused":
        return {"kind": "sample", **_drawn_graph(rng, 1 << 10, 1 << 15, 4, 16), "model": "IC",
                "weights": "uniform", "hi": round(rng.uniform(0.02, 0.06), 3), "sampler": "fused",
                "colors": rng.choice([64, 128, 256]), "sets": _between(rng, 500, 20000),
                "export": False}
    if kind == "select":
        return {"kind": "select", **_drawn_graph(rng, 1 << 12, 1 << 22, 4, 16), "model": "IC",
                "weights": "wc", "hi": 1.0, "sets": _between(rng, 1000, 400000), "k": k, "tie": tie}
    if kind == "batch":
        return {"kind": "batch", "graphs": rng.randint(2, 6), "n": _between(rng, 4096, 8192),
                "n_hi": _between(rng, 16384, 65536), "deg": 4, "deg_hi": rng.randint(8, 32),
                "queries": rng.randint(4, 12), "k": 10, "k_hi": rng.randint(20, 200),
                "eps": round(rng.uniform(0.1, 0.2), 3), "eps_hi": 0.5}
    if kind == "spread_ic":
        return {"kind": "spread", **_drawn_graph(rng, 1 << 12, 1 << 20, 4, 16), "model": "IC",
                "weights": "uniform", "hi": round(rng.uniform(0.02, 0.1), 3), "k": k,
                "replicas": _between(rng, 100, 1500)}
    if kind == "spread_lt":
        return {"kind": "spread", **_drawn_graph(rng, 1 << 12, 1 << 16, 4, 12), "model": "LT",
                "weights": "lt", "hi": 1.0, "k": k, "replicas": _between(rng, 100, 2000)}
    return {"kind": "upload", **_drawn_graph(rng, 1 << 12, 1 << 18, 4, 16), "model": "LT",
            "weights": "lt", "hi": 1.0, "k": k, "eps": max(eps, 0.2), "tie": tie}


def _device_graph(ctx, case, seed):
    """The case's graph, built on the device from the seed."""
    args = (case["model"], WEIGHTS[case["weights"]], seed, seed + 1, 0.0, case["hi"])
    if case["graph"] == "rmat":
        g = rb.DeviceGraph.rmat_on_device(ctx, case["n"].bit_length() - 1, case["draws"], *args)
    else:
        g = rb.DeviceGraph.erdos_renyi_on_device(ctx, case["n"], case["draws"], *args)
    torch.cuda.empty_cache()  # the sorted keys' room goes back to the library's own allocations
    return g


def _host_graph(case, seed):
    if case["graph"] == "rmat":
        g = rb.HostGraph.rmat(case["n"].bit_length() - 1, case["draws"], seed=seed)
    else:
        g = rb.HostGraph.erdos_renyi(case["n"], case["draws"], seed=seed)
    return g.with_weights(WEIGHTS[case["weights"]], seed + 1, 0.0, case["hi"])


def _batch_specs(case, seed):
    """The graphs of a batch and its queries (graph, k, eps, seed): sizes from the case alone."""
    r = np.random.RandomState(case["n"] + case["n_hi"])
    span = lambda lo, hi, i, count: lo * (hi / lo) ** (i / max(1, count - 1))  # noqa: E731
    graphs = []
    for i in range(case["graphs"]):
        n = int(span(case["n"], case["n_hi"], i, case["graphs"])) | 1
        deg = int(r.randint(case["deg"], case["deg_hi"] + 1))
        graphs.append({"graph": "er" if i % 2 else "rmat", "model": "LT" if i % 3 else "IC",
                       "n": n if i % 2 else 1 << (n.bit_length() - 1), "draws": n * deg,
                       "weights": "lt" if i % 3 else "uniform", "hi": 0.05})
    queries = []
    for q in range(case["queries"]):
        queries.append((q % case["graphs"], int(r.randint(case["k"], case["k_hi"] + 1)),
                        float(r.uniform(case["eps"], case["eps_hi"])), seed + 7 * q))
    return graphs, queries


def _hubs(index, k):
    """The k vertices of the longest lists."""
    return np.argsort(-np.diff(index.astype(np.int64)), kind="stable")[:k].astype(np.uint32)


def prepare(case, seed):
    kind = case["kind"]
    ctx = rb.Context(0)
    state = {"case": case, "seed": seed, "ctx": ctx}
    if kind == "upload":
        state["host"] = _host_graph(case, seed)
        return state
    if kind == "batch":
        graphs, queries = _batch_specs(case, seed)
        state["graphs"] = [_device_graph(ctx, g, seed + 3 * i) for i, g in enumerate(graphs)]
        state["queries"] = queries
        return state
    if kind == "spread" and case["model"] == "LT":
        h = _host_graph(case, seed)
        f = h.transposed()
        state["back"] = rb.DeviceGraph(ctx, h, "LT")
        state["graph"] = rb.DeviceGraph(ctx, f, "IC")
        state["seeds"] = _hubs(f.index, case["k"])
        return state
    state["graph"] = _device_graph(ctx, case, seed)
    if kind == "spread":
        # the device graph's lists serve as out-lists: the forward CSR of the transposed R-MAT draw
        index, _ = state["graph"].export()
        state["seeds"] = _hubs(index, case["k"])
        return state
    state["pool"] = rb.Pool(state["graph"])
    if kind == "sample":
        state["pool"].configure(colors=case["colors"])
        if case["export"]:  # the caller's room for the sets (R-MAT walks take some tens of steps)
            state["sets"] = np.zeros(case["sets"] * 512, dtype=np.int32)
    if kind == "select":
        state["pool"].sample(case["sets"], seed)
    return state


def _padded(seeds, k):
    """Seeds as the caller's array of k (a selection that covers every set ends early)."""
    out = np.zeros(k, dtype=np.int32)
    out[: len(seeds)] = seeds.view(np.int32)
    return out


def _imm_outputs(case, seeds, rec):
    return {"seeds": _padded(seeds, case["k"]), "theta": int(rec.theta),
            "sets": int(rec.total_sets), "elements": int(rec.pool_elements), "f": float(rec.f),
            "rounds": int(rec.num_rounds),
            "deltas": np.array(rec.theta_prime_deltas[:], dtype=np.int64)}


def run(state):
    case, kind, seed = state["case"], state["case"]["kind"], state["seed"]
    if kind == "imm":
        pool = state["pool"]
        pool.clear()
        return _imm_outputs(case, *pool.imm(case["k"], case["eps"], 1.0, seed, TIES[case["tie"]]))
    if kind == "sample":
        pool = state["pool"]
        pool.clear()
        pool.sample(case["sets"], seed, SAMPLERS[case["sampler"]])
        if case["export"]:
            off, vtx = pool.export()
            state["sets"][: len(vtx)] = vtx.view(np.int32)
            return {"offsets": off.view(np.int64), "vertices": state["sets"]}
        return {"counts": pool.count().view(np.int32), "elements": pool.num_elements}
    if kind == "select":
        f, seeds, gains = state["pool"].select(case["k"], tiebreak=TIES[case["tie"]])
        return {"f": f, "seeds": _padded(seeds, case["k"]),
                "gains": _padded(gains.astype(np.uint32), case["k"])}
    if kind == "batch":
        qs = [rb.Query(state["graphs"][g], k, eps, seed=s) for g, k, eps, s in state["queries"]]
        rb.imm_batch(state["ctx"], qs)
        return [{"seeds": _padded(q.seeds, len(q.buf)), "theta": int(q.record.theta),
                 "sets": int(q.record.total_sets)} for q in qs]
    if kind == "spread":
        if case["model"] == "LT":
            mean, sizes = rb.spread_lt(state["graph"], state["back"], state["seeds"],
                                       case["replicas"], seed, with_sizes=True)
        else:
            mean, sizes = rb.spread_ic(state["graph"], state["seeds"], case["replicas"], seed,
                                       with_sizes=True)
        return {"mean": mean, "reached": sizes.view(np.int32)}
    graph = rb.DeviceGraph(state["ctx"], state["host"], case["model"])
    pool = rb.Pool(graph)
    out = _imm_outputs(case, *pool.imm(case["k"], case["eps"], 1.0, seed, TIES[case["tie"]]))
    pool.close()
    graph.close()
    return out


def work(case):
    """The graph read once and the outputs written once (the sampling itself is integer arithmetic
    and random access, which has no closed form in these sizes)."""
    if case["kind"] == "batch":
        graphs, _ = _batch_specs(case, 0)
        return {"bytes": sum(8 * g["draws"] + 4 * g["n"] for g in graphs), "flops": 0}
    graph = 8 * case["draws"] + 4 * (case["n"] + 1)
    if case["kind"] == "select":  # the resident sets' offsets, lengths and elements (about 8 a set)
        return {"bytes": 44 * case["sets"] + 4 * case["n"], "flops": 0}
    if case["kind"] == "upload":
        return {"bytes": graph + 8 * case["draws"] + 8 * case["n"], "flops": 0}
    if case["kind"] == "sample":  # the sets themselves are as many as the draws make them
        return {"bytes": graph + 12 * case["sets"] + 4 * case["n"], "flops": 0}
    if case["kind"] == "spread":
        return {"bytes": graph * (2 if case["model"] == "LT" else 1) + 4 * case["replicas"],
                "flops": 0}
    return {"bytes": graph, "flops": 0}


def tolerance(case):
    return "exact"
