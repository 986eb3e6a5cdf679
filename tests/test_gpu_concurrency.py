"""Concurrent queries on one device: IMMs run from several host threads, each
with its own context (graph copy and pool), return exactly what each query
returns when run alone.  bench.py times its IMM workloads this way (a query's
reference-heap selection waits on the host while another query's kernels use
the GPU), so the contexts must share nothing but the device."""
import threading

import numpy as np
import pytest

import ripples_b200 as rb

pytestmark = pytest.mark.gpu


def graphs():
    ic = rb.HostGraph.rmat(13, 8 << 13, seed=3).with_weights(rb.WEIGHTS_WC)
    lt = rb.HostGraph.rmat(13, 8 << 13, seed=4).with_weights(rb.WEIGHTS_LT_NORMALIZED, seed=5)
    return [("IC", ic), ("LT", lt)]


@pytest.mark.parametrize("model,g", graphs(), ids=["IC", "LT"])
def test_concurrent_contexts_match_alone(model, g):
    queries = [(20, 0.3, 100 + i) for i in range(8)]
    # alone: one context, one query after another
    alone = []
    cx = rb.Context(0)
    dg = rb.DeviceGraph(cx, g, model)
    pool = rb.Pool(dg)
    for k, eps, seed in queries:
        pool.clear()
        seeds, rec = pool.imm(k, eps, 1.0, seed=seed)
        alone.append((seeds.tolist(), rec.theta, rec.total_sets, rec.f))
    cx.close()
    # concurrent: four threads, a context each, two queries each
    n_clients = 4
    got = [None] * len(queries)
    errors = []

    def client(j):
        try:
            c = rb.Context(0)
            d = rb.DeviceGraph(c, g, model)
            p = rb.Pool(d)
            for i in range(j, len(queries), n_clients):
                k, eps, seed = queries[i]
                p.clear()
                seeds, rec = p.imm(k, eps, 1.0, seed=seed)
                got[i] = (seeds.tolist(), rec.theta, rec.total_sets, rec.f)
            c.close()
        except Exception as exc:  # reported after the join
            errors.append(repr(exc))

    threads = [threading.Thread(target=client, args=(j,)) for j in range(n_clients)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert got == alone
    # the queries differ from each other (the comparison is not vacuous)
    assert len({tuple(a[0]) for a in alone}) > 1
    assert np.all([a[1] > 0 for a in alone])


@pytest.mark.parametrize("model,sizes", [("IC", [450007, 700001, 1200007, 1800001]),
                                         ("IC", [9001, 100003, 30011, 200003]),
                                         ("LT", [9001, 20011, 30011, 12007]),
                                         ("LT", [40009, 65536, 50021, 60013])])
def test_concurrent_spreads_of_different_sizes(model, sizes):
    """Four threads launch one kernel with the shared memory their graphs take."""
    def spread(n, out):
        ctx = rb.Context(0)
        g = rb.HostGraph.erdos_renyi(n, 3 * n, seed=n)  # (replicas grow: bitmaps in shared memory)
        g = g.with_weights(rb.WEIGHTS_UNIFORM if model == "IC" else rb.WEIGHTS_LT_NORMALIZED, 1,
                           0.0, 1.0)
        fg = rb.DeviceGraph(ctx, g.forward(), "IC")
        assert model == "LT" or fg.branching > 1.1
        bg = rb.DeviceGraph(ctx, g, "LT") if model == "LT" else None
        for rep in range(30):
            args = ([1, 2, 3], 20, rep)
            out.append(rb.spread_lt(fg, bg, *args) if bg else rb.spread_ic(fg, *args))
        ctx.close()

    alone = [[] for _ in sizes]
    for n, out in zip(sizes, alone):
        spread(n, out)
    got, errors = [[] for _ in sizes], []

    def client(i):
        try:
            spread(sizes[i], got[i])
        except Exception as exc:  # reported after the join
            errors.append(repr(exc))

    threads = [threading.Thread(target=client, args=(i,)) for i in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert got == alone


def test_reference_heap_on_every_device():
    """Launch limits belong to a device: selections on each one in turn, in one
    process, answer alike (a heap of 17 levels needs more than 48 KB a block)."""
    import torch
    if torch.cuda.device_count() < 2:
        pytest.skip("one device")
    g = rb.HostGraph.rmat(16, 8 << 16, seed=3).with_weights(rb.WEIGHTS_WC, 4, 0.0, 1.0)
    answers = []
    for device in range(torch.cuda.device_count()):
        ctx = rb.Context(device)
        p = rb.Pool(rb.DeviceGraph(ctx, g, "IC"))
        p.sample(5000, seed=1)
        answers.append(p.select(20, tiebreak=rb.TIE_REF_HEAP)[1].tolist())
        ctx.close()
    assert all(a == answers[0] for a in answers)
