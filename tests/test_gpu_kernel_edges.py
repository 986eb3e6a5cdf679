"""Edges of the kernels' work division: list and set lengths around tiles,
blocks and hand-over sizes, thresholds at the ends of their range.  Everything
is integer work, so every comparison is exact."""
import numpy as np
import pytest

import ripples_b200 as rb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def hub_graph(hubs, lengths, probs, n=6000, seed=5):
    """`hubs` vertices with in-lists of the given lengths (cycled) and one
    probability each (cycled), half of their sources hubs; the other vertices
    have one in-edge from a hub at 0.4."""
    r = np.random.RandomState(seed)
    lists, w = [], []
    for v in range(n):
        if v < hubs:
            d = lengths[v % len(lengths)]
            s = np.where(r.rand(d) < 0.5, r.randint(0, hubs, d), r.randint(0, n, d))
            lists.append(np.sort(s).astype(np.uint32))
            w.append(np.full(d, probs[(v // len(lengths)) % len(probs)], dtype=np.float32))
        else:
            lists.append(np.array([v % hubs], dtype=np.uint32))
            w.append(np.array([0.4], dtype=np.float32))
    index = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum([len(x) for x in lists], out=index[1:])
    return rb.HostGraph(n, index, np.concatenate(lists), np.concatenate(w))


@pytest.mark.parametrize("threads", [128, 256, 1024])
@pytest.mark.parametrize("hubs,probs", [
    (64, [1e-3, 2.0 ** -16, 3e-4]),         # few live edges: deferred blocks
    (400, [0.02, 0.03]),                    # more long lists in a level than are listed
    (40, [0.5, 65535.5 / 65536, 1.0, 0.0]),  # more deferred blocks than there is room for
])
def test_heavy_set_list_tiles(ctx, threads, hubs, probs):
    # block counts around a tile (32), the listing length (128) and a CTA's width
    lengths = [1, 250, 256, 257, 1009, 1016, 1024, 1025, 1033, 2040, 2056, 4099]
    g = hub_graph(hubs, lengths, probs)
    dg = rb.DeviceGraph(ctx, g, "IC")
    assert dg.uniform_thresholds()
    p = rb.Pool(dg)
    p.heavy_batch(0)
    p.heavy_block(threads)
    p.work_caps(64, 0)
    p.sample(300, seed=9, sampler=rb.SAMPLER_PLAIN)
    off, vtx = p.export()
    thr = O.pack("IC", g.index, g.weights)
    ooff, ovtx, ost = O.sample("IC", g.n, g.index, g.src, thr, 9, 0, 300)
    assert np.array_equal(off, ooff) and np.array_equal(vtx, ovtx)
    st = p.stats()
    assert st[4] == ost[0] and st[5] == ost[1]
    dg.close()


@pytest.mark.parametrize("scale,weights,handed", [(15, "wc", False), (19, "wc", True),
                                                  (14, "uniform", True)])
def test_sets_are_handed_over_where_it_pays(ctx, scale, weights, handed):
    """Near-critical graphs below 2^21 edges keep their sets on the warps up to 2^18
    in-edges (one launch a sample); larger ones and supercritical ones hand them
    over at 2^14."""
    kind, hi = (rb.WEIGHTS_WC, 1.0) if weights == "wc" else (rb.WEIGHTS_UNIFORM, 0.2)
    g = rb.HostGraph.erdos_renyi(1 << scale, 16 << scale, seed=1).with_weights(kind, 2, 0.0, hi)
    dg = rb.DeviceGraph(ctx, g, "IC")
    p = rb.Pool(dg)
    for _ in range(2):  # (the first one grows the pool)
        p.clear()
        p.sample(4000, seed=3, sampler=rb.SAMPLER_PLAIN)
    assert (p.timing()[1] > 1) == handed
    off, vtx = p.export()
    thr = O.pack("IC", g.index, g.weights)
    ooff, ovtx, _ = O.sample("IC", g.n, g.index, g.src, thr, 3, 0, 400)
    assert np.array_equal(off[:401], ooff) and np.array_equal(vtx[: int(off[400])], ovtx)
    dg.close()


def test_heavy_block_goes_back_to_its_default(ctx):
    g = hub_graph(64, [257, 1033, 4099], [1e-3, 0.02])
    dg = rb.DeviceGraph(ctx, g, "IC")
    p = rb.Pool(dg)
    p.heavy_batch(0)
    p.work_caps(64, 0)
    sets = []
    for threads in (0, 128, 1024, 0):
        p.heavy_block(threads)
        p.clear()
        p.sample(300, seed=9, sampler=rb.SAMPLER_PLAIN)
        sets.append(p.export())
    assert all(np.array_equal(a, b) for s in sets[1:] for a, b in zip(s, sets[0]))
    for threads in (1, 64, 2048):
        with pytest.raises(rb.RipError):
            p.heavy_block(threads)
    dg.close()


SET_LENGTHS = [0, 1, 31, 32, 33, 63, 64, 65, 511, 512, 513, 1023, 1024, 1025, 5000]


@pytest.mark.parametrize("tie", [rb.TIE_REF_HEAP, rb.TIE_LOWEST_ID])
@pytest.mark.parametrize("copies,n", [(1, 6001), (40, 5003), (700, 5200)])
def test_selection_over_set_lengths(ctx, tie, copies, n):
    r = np.random.RandomState(copies)
    lens = np.array(SET_LENGTHS * copies) if copies < 100 else np.array(SET_LENGTHS[:10] * copies)
    r.shuffle(lens)
    off = np.zeros(len(lens) + 1, dtype=np.uint64)
    np.cumsum(lens, out=off[1:])
    vtx = np.concatenate([r.choice(n, d, replace=False) for d in lens]).astype(np.uint32)
    g = rb.HostGraph(n, np.zeros(n + 1, np.uint64), np.zeros(0, np.uint32), np.zeros(0, np.float32))
    dg = rb.DeviceGraph(ctx, g, "IC")
    p = rb.Pool(dg)
    p.import_sets(off, vtx)
    for s in (len(lens), len(lens) // 2 + 1):
        e = int(off[s])
        assert np.array_equal(p.count(s), np.bincount(vtx[:e], minlength=n))
        of, oseeds, ogains, _ = O.select(n, off[: s + 1], vtx[:e], 12, tie)
        if tie == rb.TIE_LOWEST_ID:  # device picks end with the last one that covers a set
            oseeds, ogains = oseeds[ogains > 0], ogains[ogains > 0]
        f, seeds, gains = p.select(12, s, tie)
        assert f == of and seeds.tolist() == oseeds.tolist() and gains.tolist() == ogains.tolist()
    dg.close()


@pytest.mark.parametrize("k,hot", [(6, 40), (30, 40), (60, 25000)])
def test_reference_heap_keeps_more_items(ctx, k, hot):
    """The first seed covers most sets, so the gains fall below the counts the
    host kept at first (n above what it keeps).  k = 6: they stay within them; 30:
    every set with members is covered and one without is left, counts of zero,
    which are some 500 times what was kept; 60: all counts in one step."""
    n, r = 40003, np.random.RandomState(hot)
    sets = [np.concatenate([[0], 1 + r.choice(hot, 30, replace=False)]) for _ in range(900)]
    sets += [np.array([hot + 1 + i, hot + 2 + i]) for i in range(0, 40, 2)] + [np.array([], int)]
    check_reference_heap(ctx, n, sets, k)


def test_reference_heap_keeps_a_large_next_bucket(ctx):
    """Few vertices in two sets each, many in one: the counts of one are 500 times
    the kept, and the gains fall to them."""
    first = 100 + 200 * 250
    sets = [np.concatenate([[i // 2], 100 + 250 * i + np.arange(250)]) for i in range(200)]
    sets += [np.array([first + i]) for i in range(40)]
    check_reference_heap(ctx, 60007, sets, 120)


def check_reference_heap(ctx, n, sets, k):
    off = np.zeros(len(sets) + 1, dtype=np.uint64)
    np.cumsum([len(x) for x in sets], out=off[1:])
    vtx = np.concatenate(sets).astype(np.uint32)
    g = rb.HostGraph(n, np.zeros(n + 1, np.uint64), np.zeros(0, np.uint32), np.zeros(0, np.float32))
    dg = rb.DeviceGraph(ctx, g, "IC")
    p = rb.Pool(dg)
    p.import_sets(off, vtx)
    of, oseeds, ogains, _ = O.select(n, off, vtx, k, rb.TIE_REF_HEAP)
    for guess in (0, 100, 3):  # adaptive, too high, too low first fetches
        p.select_guess(guess)
        f, seeds, gains = p.select(k, tiebreak=rb.TIE_REF_HEAP)
        assert f == of and seeds.tolist() == oseeds.tolist() and gains.tolist() == ogains.tolist()
    dg.close()


@pytest.mark.parametrize("model,n,sets,k", [("IC", 1 << 20, 1000, 200), ("LT", 1 << 18, 100, 60)])
def test_reference_heap_on_few_sampled_sets(ctx, model, n, sets, k):
    """Few sets on many vertices: nearly all counts are zero, most others one."""
    g = rb.HostGraph.erdos_renyi(n, 8 * n, seed=3).with_weights(
        rb.WEIGHTS_WC if model == "IC" else rb.WEIGHTS_LT_NORMALIZED, 1, 0.0, 1.0)
    dg = rb.DeviceGraph(ctx, g, model)
    p = rb.Pool(dg)
    for seed in (1, 2, 3):
        p.clear()
        p.sample(sets, seed=seed)
        off, vtx = p.export()
        of, oseeds, ogains, _ = O.select(n, off, vtx, k, rb.TIE_REF_HEAP)
        f, seeds, gains = p.select(k, tiebreak=rb.TIE_REF_HEAP)
        assert f == of and seeds.tolist() == oseeds.tolist() and gains.tolist() == ogains.tolist()
    dg.close()


def star_graph(degrees, weights, n=30000, seed=11):
    """Vertex v < len(degrees) has degrees[v] in-edges, the others one from a
    small vertex; weights 'equal', 'random', 'skewed' or 'short' (sum 0.5)."""
    r = np.random.RandomState(seed)
    lists, w = [], []
    for v in range(n):
        d = degrees[v] if v < len(degrees) else 1
        s = r.randint(0, len(degrees) if v >= len(degrees) or r.rand() < 0.3 else n, d)
        x = {"equal": np.ones(d), "random": r.rand(d) + 1e-9, "short": np.ones(d),
             "skewed": np.where(r.rand(d) < 0.02, 1.0, 1e-5)}[weights]
        lists.append(np.sort(s).astype(np.uint32))
        w.append((x / x.sum() * (0.5 if weights == "short" else 1.0)).astype(np.float32))
    index = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum([len(x) for x in lists], out=index[1:])
    return rb.HostGraph(n, index, np.concatenate(lists), np.concatenate(w))


@pytest.mark.parametrize("weights", ["equal", "random", "skewed", "short"])
def test_lt_walk_search_over_list_lengths(ctx, weights):
    # read whole up to 128 edges, one guessed read up to 4096, then two
    g = star_graph([1, 2, 31, 32, 33, 127, 128, 129, 160, 1023, 1024, 1025, 4095, 4096, 4097,
                    9000, 20000], weights)
    dg = rb.DeviceGraph(ctx, g, "LT")
    assert np.array_equal(dg.thresholds(), O.pack("LT", g.index, g.weights))
    p = rb.Pool(dg)
    p.sample(6000, seed=3)
    off, vtx = p.export()
    ooff, ovtx, ost = O.sample("LT", g.n, g.index, g.src, O.pack("LT", g.index, g.weights), 3, 0,
                               6000)
    assert np.array_equal(off, ooff) and np.array_equal(vtx, ovtx) and p.stats()[4] == ost[0]
    dg.close()


def test_lt_walk_revisits(ctx):
    """Walks that come back to their first, 32nd, 33rd, ... vertex: tails into
    cycles, one in-edge of weight 1 a vertex."""
    src = []
    for tail in (0, 1, 30, 31, 32, 33, 100, 700):
        for cycle in (1, 2, 31, 32, 33, 127, 128, 129, 161, 500):
            at = len(src)
            src += list(range(at + 1, at + tail + cycle)) + [at + tail]
    n = len(src)
    g = rb.HostGraph(n, np.arange(n + 1, dtype=np.uint64), np.array(src, dtype=np.uint32),
                     np.ones(n, dtype=np.float32))
    dg = rb.DeviceGraph(ctx, g, "LT")
    p = rb.Pool(dg)
    p.sample(4000, seed=3)
    off, vtx = p.export()
    ooff, ovtx, ost = O.sample("LT", n, g.index, g.src, O.pack("LT", g.index, g.weights), 3, 0,
                               4000)
    assert np.array_equal(off, ooff) and np.array_equal(vtx, ovtx) and p.stats()[4] == ost[0]
    dg.close()


@pytest.mark.parametrize("copies", [1, 25])
def test_device_picks_in_one_launch_and_grid_wide(ctx, copies):
    """Lowest-id picks by one cluster (up to 8 M elements) and by the grid-wide
    kernels (here 8.8 M): giant first covers (recounts) and small ones, ties."""
    n, r = 20011, np.random.RandomState(7)
    sets = [np.unique(np.concatenate([[5], r.randint(0, n, 6000)])) for _ in range(60)]
    sets += [r.choice(n, 1 + i % 40, replace=False) for i in range(2000)]
    sets = sets * copies
    off = np.zeros(len(sets) + 1, dtype=np.uint64)
    np.cumsum([len(x) for x in sets], out=off[1:])
    vtx = np.concatenate(sets).astype(np.uint32)
    assert (len(vtx) > 8 << 20) == (copies > 1)
    g = rb.HostGraph(n, np.zeros(n + 1, np.uint64), np.zeros(0, np.uint32), np.zeros(0, np.float32))
    dg = rb.DeviceGraph(ctx, g, "IC")
    p = rb.Pool(dg)
    p.import_sets(off, vtx)
    for s, k in ((len(sets), 40), (len(sets) - 777, 3), (61, 9)):
        e = int(off[s])
        of, oseeds, ogains, _ = O.select(n, off[: s + 1], vtx[:e], k, rb.TIE_LOWEST_ID)
        f, seeds, gains = p.select(k, s, rb.TIE_LOWEST_ID)
        assert f == of and seeds.tolist() == oseeds.tolist() and gains.tolist() == ogains.tolist()
    dg.close()


@pytest.mark.parametrize("n", [1 << 19, (1 << 19) + 1, 1100003])
def test_device_picks_by_the_number_of_chunks(ctx, n):
    """Small rounds of up to 512 chunks of 1024 vertices are one launch, those of more
    go pick by pick: the last chunks full, of one vertex, ragged."""
    r = np.random.RandomState(5)
    sets = [np.unique(np.concatenate([[n - 1 - i % 3], r.randint(0, n, 1 + i % 90)]))
            for i in range(3000)]
    off = np.zeros(len(sets) + 1, dtype=np.uint64)
    np.cumsum([len(x) for x in sets], out=off[1:])
    vtx = np.concatenate(sets).astype(np.uint32)
    g = rb.HostGraph(n, np.zeros(n + 1, np.uint64), np.zeros(0, np.uint32), np.zeros(0, np.float32))
    dg = rb.DeviceGraph(ctx, g, "IC")
    p = rb.Pool(dg)
    p.import_sets(off, vtx)
    for s, k in ((3000, 3), (2999, 60), (100, 40)):
        e = int(off[s])
        of, oseeds, ogains, _ = O.select(n, off[: s + 1], vtx[:e], k, rb.TIE_LOWEST_ID)
        oseeds, ogains = oseeds[ogains > 0], ogains[ogains > 0]
        f, seeds, gains = p.select(k, s, rb.TIE_LOWEST_ID)
        assert f == of and seeds.tolist() == oseeds.tolist() and gains.tolist() == ogains.tolist()
    dg.close()


@pytest.mark.parametrize("total", [0.7, 5.0])
def test_lt_pack_over_list_lengths(ctx, total):
    """Cumulative weights of lists that end on and off the scan's 32-edge and
    1024-edge steps, long ones side by side, empty ones between; sums past 1
    saturate."""
    lens = [0, 1, 31, 32, 33, 64, 0, 1023, 1024, 1025, 1024, 4096, 4097, 0, 0, 5000, 7, 100] * 9
    r = np.random.RandomState(3)
    index = np.zeros(len(lens) + 1, dtype=np.uint64)
    np.cumsum(lens, out=index[1:])
    m = int(index[-1])
    w = np.concatenate([r.rand(d) * (2 * total / max(d, 1)) for d in lens]).astype(np.float32)
    g = rb.HostGraph(len(lens), index, r.randint(0, len(lens), m).astype(np.uint32), w)
    dg = rb.DeviceGraph(ctx, g, "LT")
    assert np.array_equal(dg.thresholds(), O.pack("LT", g.index, g.weights))
    dg.close()


@pytest.mark.parametrize("n,hi", [(20011, 0.2), (500009, 0.2), (1900003, 0.2), (20011, 0.002),
                                  (500009, 0.001)])
def test_spread_bitmap_places(ctx, n, hi):
    """The reached bitmap in shared memory (four CTAs an SM, one) and in global
    memory (large graphs, and wide ones whose replicas stay small); small levels
    packed over a CTA; out-lists around a tile and past what a level lists."""
    r = np.random.RandomState(n % 97)
    lens = [1, 7, 8, 9, 255, 1016, 1024, 1025, 2049, 5000] * 30
    src = np.repeat(np.arange(len(lens)), lens)  # out-lists of the first vertices
    dst = r.randint(0, n, len(src))
    hub = r.rand(len(src)) < 0.2
    dst[hub] = r.randint(0, len(lens), hub.sum())
    g = rb.HostGraph.from_edges(n, src, dst, r.rand(len(src)) * hi)
    dg = rb.DeviceGraph(ctx, g.forward(), "IC")
    assert (dg.branching > 1.1) == (hi > 0.1)
    seeds = list(range(12))
    mean, sizes, levels = rb.spread_ic(dg, seeds, 200, seed=5, with_sizes=True, with_levels=True)
    f = g.forward()
    _, o_sizes, o_levels = O.spread_ic(f.n, f.index, f.src, O.pack("IC", f.index, f.weights), seeds,
                                       200, seed=5, with_levels=True)
    assert np.array_equal(sizes, o_sizes) and np.array_equal(levels, o_levels)
    dg.close()


@pytest.mark.parametrize("n", [2011, 33000, 65536, 65537])
def test_spread_lt_swept_and_scanned(ctx, n):
    """Replicas that stay below the sweep's share of out-edges and replicas that
    go on over kept sources: 16-bit ids up to 65536 vertices, deep levels."""
    r = np.random.RandomState(n)
    chain = 300  # the last ids: one in-edge each
    src, dst = r.randint(0, n - chain, 4 * n), r.randint(0, n - chain, 4 * n)
    src[: 2 * n] = r.randint(0, 40, 2 * n)  # hubs
    src = np.concatenate([src, [7], np.arange(n - chain, n - 1)])
    dst = np.concatenate([dst, np.arange(n - chain, n)])
    g = rb.HostGraph.from_edges(n, src, dst).with_weights(rb.WEIGHTS_LT_NORMALIZED, 3, 0.0, 1.0)
    fg, bg = rb.DeviceGraph(ctx, g.forward(), "IC"), rb.DeviceGraph(ctx, g, "LT")
    few = [n - 5, 1000, 1000, n - chain]
    for seeds, replicas in ((few, 40), (few + [7], 40), (list(range(40)), 20), ([], 5)):
        _, sizes, levels = rb.spread_lt(fg, bg, seeds, replicas, seed=23, with_sizes=True,
                                        with_levels=True)
        _, o_sizes, o_levels = O.spread_lt(g, seeds, replicas, seed=23, with_levels=True)
        assert np.array_equal(sizes, o_sizes) and np.array_equal(levels, o_levels)
    bg.close()
    fg.close()


@pytest.mark.parametrize("n,chain", [(2011, 2000), (33000, 5000), (35000, 34000), (65536, 65535)])
def test_spread_lt_deep_chains(ctx, n, chain):
    """Chains of kept sources as long as the graph, cycles, self-loops, vertices that
    keep no in-edge; sizes with levels and alone (kernels of their own)."""
    r = np.random.RandomState(n)
    dst = np.arange(1, n)
    src = np.where(dst < chain, dst - 1, r.randint(0, n, n - 1))  # past the chain: trees and cycles
    loops = r.choice(n - 1, 50, replace=False)
    src[loops[loops > chain]] = dst[loops[loops > chain]]
    w = np.where(dst < chain, 1.0, 0.9).astype(np.float32)
    # a second in-edge from far behind for some vertices of the chain
    more = np.arange(chain // 3, chain, 37)
    src, dst, w = np.append(src, more // 2), np.append(dst, more), np.append(w, 0.0 * more)
    w[more - 1], w[n - 1:] = 0.999, 0.001
    g = rb.HostGraph.from_edges(n, src, dst, w)
    fg, bg = rb.DeviceGraph(ctx, g.forward(), "IC"), rb.DeviceGraph(ctx, g, "LT")
    for seeds, replicas in (([0], 12), ([n - 1, 5, chain // 2], 300), (list(range(0, n, 97)), 12)):
        _, sizes, levels = rb.spread_lt(fg, bg, seeds, replicas, seed=23, with_sizes=True,
                                        with_levels=True)
        mean, alone = rb.spread_lt(fg, bg, seeds, replicas, seed=23, with_sizes=True)
        _, o_sizes, o_levels = O.spread_lt(g, seeds, replicas, seed=23, with_levels=True)
        assert np.array_equal(sizes, o_sizes) and np.array_equal(levels, o_levels)
        assert np.array_equal(alone, o_sizes) and mean == o_sizes.mean()
    bg.close()
    fg.close()


@pytest.mark.parametrize("grid", [False, True])
@pytest.mark.parametrize("colors,sets", [(64, 60), (128, 300), (256, 500), (256, 4500)])
def test_colour_pairs(ctx, grid, colors, sets):
    """Multi-colour levels: masks of one set and of all 256, lists around a
    window's and a tile's blocks, more long entries in a level than a CTA lists;
    a fresh pool that its sets overflow."""
    lengths = [1, 7, 8, 9, 16, 31, 63, 127, 128, 129, 250, 1016, 1024, 1025, 4099]
    g = hub_graph(400, lengths, [0.02, 0.03, 1e-3, 1.0])
    dg = rb.DeviceGraph(ctx, g, "IC")
    p = rb.Pool(dg)
    p.configure(colors=colors)
    if grid:  # batches of the whole grid
        p.heavy_batch(1)
        p.work_caps(64, 0)
    p.sample(sets, seed=9, sampler=rb.SAMPLER_PLAIN if grid else rb.SAMPLER_FUSED)
    off, vtx = p.export()
    thr = O.pack("IC", g.index, g.weights)
    ooff, ovtx, ost = O.sample("IC", g.n, g.index, g.src, thr, 9, 0, sets)
    assert np.array_equal(off, ooff) and np.array_equal(vtx, ovtx)
    st = p.stats()
    assert st[4] == ost[0] and st[5] == ost[1]
    dg.close()


@pytest.mark.parametrize("threads", [0, 128, 512, 1024])
def test_record_tiles(ctx, threads):
    """Lists with a threshold per edge, read 32 coin blocks at a time: ends on and
    off blocks, tiles and the listing length; one warp per set and CTAs."""
    r = np.random.RandomState(4)
    g = hub_graph(300, [7, 247, 248, 249, 255, 256, 257, 263, 511, 513, 1000, 1025, 4099], [0.5])
    w = (r.rand(g.m) * 0.01).astype(np.float32)
    w[r.rand(g.m) < 0.002] = 1.0
    w[-5000:] = 0.4
    g = rb.HostGraph(g.n, g.index, g.src, w)
    dg = rb.DeviceGraph(ctx, g, "IC")
    p = rb.Pool(dg)
    p.heavy_batch(0)
    if threads:
        p.heavy_block(threads)
        p.work_caps(64, 0)
    else:
        p.work_caps(0, 0)  # no set is handed over
    p.sample(400, seed=9, sampler=rb.SAMPLER_PLAIN)
    off, vtx = p.export()
    ooff, ovtx, ost = O.sample("IC", g.n, g.index, g.src, O.pack("IC", g.index, g.weights), 9, 0,
                               400)
    assert np.array_equal(off, ooff) and np.array_equal(vtx, ovtx)
    st = p.stats()
    assert st[4] == ost[0] and st[5] == ost[1]
    dg.close()


def budget_calls():
    """Calls and device budgets (bytes) that are enough for them: a few KB above the
    least, which is what the graph, the sets and the smallest scratch take."""
    def graph(draws, n, weights, hi):
        return rb.HostGraph.erdos_renyi(n, draws, seed=1).with_weights(weights, 2, 0.0, hi)

    def sample(ctx):
        p = rb.Pool(rb.DeviceGraph(ctx, graph(1 << 14, 1 << 12, rb.WEIGHTS_UNIFORM, 0.05), "IC"))
        p.sample(200000, seed=3, sampler=rb.SAMPLER_PLAIN)

    def spread(ctx):
        g = graph(400000, 100000, rb.WEIGHTS_LT_NORMALIZED, 1.0)
        fg, bg = rb.DeviceGraph(ctx, g.forward(), "IC"), rb.DeviceGraph(ctx, g, "LT")
        rb.spread_lt(fg, bg, [1, 2, 3], 50, 1)

    def select(ctx):
        p = rb.Pool(rb.DeviceGraph(ctx, graph(400000, 100000, rb.WEIGHTS_WC, 1.0), "IC"))
        vtx = np.random.RandomState(1).randint(0, 100000, 400000).astype(np.uint32)
        p.import_sets(np.arange(0, 400001, 2, dtype=np.uint64), vtx)
        p.select(20, tiebreak=rb.TIE_REF_HEAP)

    return [pytest.param(sample, 6100000, id="sets that may be handed over"),
            pytest.param(select, 13850000, id="reference heap"),
            pytest.param(spread, 12050000, id="LT lists packed")]


@pytest.mark.parametrize("call,budget", budget_calls())
def test_budgets_that_are_enough(call, budget):
    ctx = rb.Context(0, budget)
    try:
        call(ctx)
    finally:
        ctx.close()
