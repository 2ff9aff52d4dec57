"""The forms a traversal may take, at the sizes where they change: the fused
and the launched level loop, row gather items and heavy in-lists, row chunks
skipped by bounds, slot lists and flattened pairs of a scatter, padded rows,
depth planes added on the way, union-find sampling, and results copied out
through pinned slots.  Everything is compared with the CPU oracle for
equality (distances are the same sums in the same order: exact)."""
import numpy as np
import pytest

import cgp_b200 as cgp
import oracle

pytestmark = pytest.mark.gpu


def _path(n):
    v = np.arange(n - 1)
    return cgp.csr_from_edges(n, v, v + 1)


def _stars(degrees, extra=40):
    """Hubs of exactly the given degrees: shared leaves, and a path through the hubs."""
    leaves = max(degrees) + extra
    src, dst = [], []
    for h, d in enumerate(degrees):
        n = d - (h > 0) - (h + 1 < len(degrees))
        src += [h] * n
        dst += list(range(len(degrees), len(degrees) + n))
    src += list(range(len(degrees) - 1))
    dst += list(range(1, len(degrees)))
    return cgp.csr_from_edges(len(degrees) + leaves, src, dst)


def _run(graph, kind, src, loop="auto", **kw):
    o = cgp.RunOptions(level_loop=loop, **kw)
    return cgp.run(kind, graph, src, options=o, layout="query").values


@pytest.mark.parametrize("loop", ["auto", "chunks"])
@pytest.mark.parametrize("n,q", [(1, 1), (2, 3), (33, 31), (300, 64), (700, 20)])
def test_path_graphs_in_both_loops(n, q, loop):
    """Depths past 15 and 255 add depth planes; 700 vertices take more levels
    than one launch of the fused loop; two vertices and one take none."""
    g = _path(n).with_weights("u32", 1, 9, seed=5) if n > 1 else cgp.csr_from_edges(1, [], [])
    graph = cgp.CsrGraph(g)
    src = np.arange(q) % n
    np.testing.assert_array_equal(_run(graph, "bfs", src, loop), oracle.batch("bfs", g, src)[0])
    if n > 1:
        np.testing.assert_array_equal(_run(graph, "sssp", src, loop).view(np.uint32),
                                      oracle.batch("sssp", g, src)[0])


@pytest.mark.parametrize("loop", ["auto", "chunks"])
@pytest.mark.parametrize("kinds", [("bfs",), ("sssp",), ("bfs", "sssp", "khop")])
def test_grid_levels_swept_or_cleared(kinds, loop):
    """Road-like graph: the fused loop zeroes masks as it reads them and clears
    nothing between levels; mixed groups clear as before."""
    g = cgp.gen_grid(37, 41, 0.1, 0.002, seed=3).with_weights("f32", 1.0, 100.0, seed=4)
    graph = cgp.CsrGraph(g)
    src = g.pick_sources(45, seed=6)
    descs = [cgp.QueryDescriptor(int(s), kinds[i % len(kinds)], 3 + i % 9) for i, s in enumerate(src)]
    r = cgp.run_batch(graph, descs, cgp.RunOptions(level_loop=loop), layout="query").values
    for i, d in enumerate(descs):
        if d.kind == "sssp":
            np.testing.assert_array_equal(r[i].view(np.float32), oracle.sssp(g, d.source))
        else:
            want = oracle.bfs(g, d.source, d.k if d.kind == "khop" else -1)
            np.testing.assert_array_equal(r[i].view(np.int32), want)


@pytest.mark.parametrize("loop", ["auto", "chunks"])
@pytest.mark.parametrize("q,words", [(45, 0), (90, 0), (126, 4)])
def test_bfs_push_beside_an_sssp_gather(q, words, loop):
    """BFS pushes while SSSP gathers, in one group whose kinds alternate by slot
    (so they share the row vectors the gather writes back), on a grid: no
    in-list is long enough for the heavy gather to come between the two."""
    for seed in range(4):
        g = cgp.gen_grid(61 + seed, 67, 0.1, 0.002, seed=seed).with_weights("f32", 1.0, 100.0, seed=4)
        graph = cgp.CsrGraph(g)
        src = g.pick_sources(q, seed=60 + seed)
        descs = [cgp.QueryDescriptor(int(s), "sssp" if i % 2 else "bfs") for i, s in enumerate(src)]
        o = cgp.RunOptions(level_loop=loop, mask_words=words, sssp_pull_edge_ratio=0.01,
                           sssp_pull_pair_ratio=0.0, pull_edge_ratio=2.0, pull_frontier_ratio=2.0)
        r = cgp.run_batch(graph, descs, o, layout="query")
        assert r.pull_levels == 0 and r.counters["sssp_pull_edges"] > 0
        np.testing.assert_array_equal(r.values[::2].view(np.int32), oracle.batch("bfs", g, src[::2])[0])
        np.testing.assert_array_equal(r.values[1::2].view(np.uint32),
                                      oracle.batch("sssp", g, src[1::2])[0].view(np.uint32))


@pytest.mark.parametrize("mode", ["pull", "hybrid", "push"])
@pytest.mark.parametrize("q", [1, 2, 6, 63, 129, 257, 500])
def test_in_degrees_around_the_gather_and_tile_limits(q, mode):
    """In-degrees 1, 32, 33, 255 .. 257 and 2047 .. 2049 beside items of one to
    32 vertices; slot counts that pad to the next multiple of 4."""
    g = _stars([1, 31, 32, 33, 255, 256, 257, 2047, 2048, 2049]).with_weights("u32", 1, 50, seed=8)
    graph = cgp.CsrGraph(g)
    src = g.pick_sources(q, seed=9)
    got = _run(graph, "sssp", src, traversal_mode=mode, sssp_pull_edge_ratio=0.05,
               sssp_pull_pair_ratio=0.01)
    np.testing.assert_array_equal(got.view(np.uint32), oracle.batch("sssp", g, src)[0])


@pytest.mark.parametrize("q", [32, 64, 100, 256, 320])
@pytest.mark.parametrize("weights", ["unit", "small", "zero", "huge", "lognormal", "f32zero"])
def test_bounds_skip_no_improvement(weights, q):
    """Every gather level after the first may skip row chunks by bounds.  Two
    components (the hub is unreachable for some slots), weights whose sums pass
    2^30 and saturate, zero weights, and float weights over a wide range."""
    a = cgp.gen_rmat(10, 8, seed=11)
    s = np.repeat(np.arange(a.num_vertices), a.degrees())
    off = a.num_vertices
    g = cgp.csr_from_edges(off + 60, np.r_[s, off + np.arange(59)],
                           np.r_[a.col_indices, off + 1 + np.arange(59)])
    if weights == "small":
        g = g.with_weights("u32", 1, 64, seed=12)
    elif weights == "zero":
        g = g.with_weights("u32", 0, 2, seed=12)
    elif weights == "huge":
        g = g.with_weights("u32", 1 << 28, 3000000000, seed=12)
    elif weights == "lognormal":
        g = g.with_weights("f32", 0.0, 2.0, seed=12, lognormal=True)
    elif weights == "f32zero":
        g = g.with_weights("f32", 0.0, 1e-3, seed=12)
    graph = cgp.CsrGraph(g)
    src = np.r_[g.pick_sources(q - 3, seed=13), off, off + 30, off + 59]
    ref = oracle.batch("sssp", g, src)[0] if weights != "unit" else None
    for mode in ("pull", "hybrid"):
        for loop in ("auto", "chunks"):
            got = _run(graph, "sssp", src, loop, traversal_mode=mode)
            if ref is None:  # unit weights: hop counts
                hops = oracle.batch("bfs", g, src)[0].view(np.uint32)
                want = np.where(hops == 0x7fffffff, np.uint32(0xffffffff), hops)
            else:
                want = ref
            np.testing.assert_array_equal(got.view(want.dtype), want)


@pytest.mark.parametrize("k", [1, 6, 7, 31, 32, 33, 64, 65, 200, 1024])
def test_scatter_of_k_slots_at_one_vertex(k):
    """k queries from one source: every vertex carries k active slots, below
    and above the list limit, in whole and partial runs of 32; lists of 40, 257
    and 2100 edges go to tiles and to the heavy queue."""
    g = _stars([3, 40, 257, 2100]).with_weights("u32", 1, 30, seed=15)
    graph = cgp.CsrGraph(g)
    src = np.full(k, g.num_vertices - 45)
    got = _run(graph, "sssp", src, traversal_mode="push", mask_words=16 if k > 512 else 0)
    want = oracle.sssp(g, int(src[0]))
    np.testing.assert_array_equal(got.view(np.uint32), np.tile(want, (k, 1)))


@pytest.mark.parametrize("frontier", [3000, 40000])
def test_scatter_lists_queued_and_in_place(frontier):
    """The second level holds `frontier` vertices of 70 active slots each: small
    frontiers scatter their lists in the tile, larger ones queue them."""
    n = frontier
    src = np.zeros(n, np.int64)
    ring = np.arange(n)
    g = cgp.csr_from_edges(n + 1, np.r_[src, 1 + ring], np.r_[1 + ring, 1 + (ring + 1) % n])
    g = g.with_weights("u32", 1, 40, seed=17)
    graph = cgp.CsrGraph(g)
    want = oracle.sssp(g, 0)
    got = _run(graph, "sssp", np.zeros(70, np.int64), traversal_mode="push")
    np.testing.assert_array_equal(got.view(np.uint32), np.tile(want, (70, 1)))


@pytest.mark.parametrize("make", [
    lambda: cgp.csr_from_edges(1, [], []),
    lambda: _path(1000),
    lambda: cgp.gen_grid(150, 130, 0.45, 0.0, seed=21),     # many components
    lambda: cgp.gen_rmat(12, 8, seed=22),
    lambda: cgp.csr_from_edges(4000, np.arange(0, 4000, 2), np.arange(1, 4000, 2)),  # pairs
    lambda: cgp.csr_from_edges(3000, np.arange(2999), np.arange(1, 3000)[::-1], symmetrize=False),
    lambda: cgp.csr_from_edges(5000, np.arange(1, 5000), np.zeros(4999), symmetrize=False),
])
def test_wcc_sampling(make):
    g = make()
    got = cgp.run("wcc", cgp.CsrGraph(g), [0]).values[:, 0].view(np.uint32)
    np.testing.assert_array_equal(got, oracle.wcc_components(g))


@pytest.mark.parametrize("n,q", [(100, 1), (131072, 1), (131073, 4), (65536, 37)])
@pytest.mark.parametrize("layout", ["vertex", "query"])
def test_results_into_pageable_and_pinned_memory(n, q, layout):
    """Result sizes below, at and beyond the copy slots and their count."""
    import torch
    g = _path(n) if n < 1000 else cgp.csr_from_edges(n, np.zeros(n - 1), np.arange(1, n))
    graph = cgp.CsrGraph(g, symmetric=True)
    src = (np.arange(q) * 7) % n
    descs = [cgp.QueryDescriptor(int(s), "bfs") for s in src]
    want = oracle.batch("bfs", g, src)[0]
    want = want if layout == "query" else want.T
    np.testing.assert_array_equal(cgp.run_batch(graph, descs, layout=layout).values, want)
    pinned = torch.empty(want.shape, dtype=torch.int32, pin_memory=True)
    cgp.run_batch(graph, descs, layout=layout, out=pinned)
    np.testing.assert_array_equal(pinned.numpy(), want)


@pytest.mark.parametrize("q", [1, 65, 129, 257, 513, 1024])
@pytest.mark.parametrize("depth", ["planes", "direct"])
def test_pull_masks_shared_by_lanes(q, depth):
    """Masks of 1 to 16 words: one lane each, or 16 bytes per lane; light, mid
    and heavy in-lists; queries of two components, k-hop bounds among them."""
    a = cgp.gen_rmat(11, 12, seed=31)
    s = np.repeat(np.arange(a.num_vertices), a.degrees())
    off = a.num_vertices
    g = cgp.csr_from_edges(off + 50, np.r_[s, off + np.arange(49)],
                           np.r_[a.col_indices, off + 1 + np.arange(49)])
    graph = cgp.CsrGraph(g)
    src = np.r_[g.pick_sources(q, seed=32), off][1:]
    descs = [cgp.QueryDescriptor(int(v), "khop" if i % 5 == 4 else "bfs", 1 + i % 4)
             for i, v in enumerate(src)]
    for mode in ("pull", "hybrid"):
        for loop in ("auto", "chunks"):
            o = cgp.RunOptions(traversal_mode=mode, level_loop=loop, depth_mode=depth,
                               heavy_degree=200)
            r = cgp.run_batch(graph, descs, o, layout="query").values.view(np.int32)
            for i in {0, q // 2, q - 1, 4 % q, min(q - 1, 64)}:
                d = descs[i]
                np.testing.assert_array_equal(
                    r[i], oracle.bfs(g, d.source, d.k if d.kind == "khop" else -1))


@pytest.mark.parametrize("offsets64", [False, True])
@pytest.mark.parametrize("weights", ["none", "u32", "f32"])
@pytest.mark.parametrize("q", [5, 70, 200])
def test_directed_gathers_over_the_transpose(q, weights, offsets64):
    """Vertices without in-edges, in-lists from 1 to 700, asymmetric weights."""
    r = np.random.default_rng(41)
    n, m = 900, 14000
    dst = (n * r.random(m) ** 3).astype(np.int64) + 20
    g = cgp.csr_from_edges(n + 20, r.integers(0, n + 20, m), np.minimum(dst, n + 19),
                           symmetrize=False)
    if weights == "u32":
        g.weights = r.integers(0, 40, g.num_edges).astype(np.uint32)
    elif weights == "f32":
        g.weights = r.random(g.num_edges).astype(np.float32) * 10
    graph = cgp.CsrGraph(g, offsets64=offsets64)
    src = r.integers(0, n + 20, q)
    if weights == "none":
        hops = oracle.batch("bfs", g, src)[0].view(np.uint32)
        want = np.where(hops == 0x7fffffff, np.uint32(0xffffffff), hops)
    else:
        want = oracle.batch("sssp", g, src)[0]
    for mode in ("pull", "hybrid"):
        for loop in ("auto", "chunks"):
            got = _run(graph, "sssp", src, loop, traversal_mode=mode)
            np.testing.assert_array_equal(got.view(want.dtype), want)


def test_rows_stay_unpadded_without_room():
    """9 SSSP slots over 16M vertices in memory that holds their 576 MB value
    matrix but not one of 10 or 12 slots per row beside the rest of the group."""
    import torch
    n = 1 << 24
    g = cgp.csr_from_edges(n, np.zeros(n - 1), np.arange(1, n))
    graph = cgp.CsrGraph(g, symmetric=True)
    src = [0, 1, 5, n - 1, 77, 4096, n // 2, 3, 2]
    descs = [cgp.QueryDescriptor(s, "sssp") for s in src]
    out = torch.empty((len(src), n), dtype=torch.int32, device="cuda")
    cgp.run_batch(graph, descs[:4], layout="query", out=out)  # the 4-slot group's memory stays
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (416 << 20), dtype=torch.uint8, device="cuda")
    cgp.run_batch(graph, descs, layout="query", out=out)
    del fill
    torch.cuda.empty_cache()
    want = torch.full((n,), 2, dtype=torch.int32, device="cuda")
    want[0] = 1
    for i, s in enumerate(src):
        w = want.clone() if s else torch.ones_like(want)
        w[s] = 0
        assert torch.equal(out[i], w)


@pytest.mark.parametrize("loop", ["auto", "chunks"])
@pytest.mark.parametrize("words", [2, 4, 8, 16])
def test_pull_edges_counted_for_any_words(words, loop):
    """One BFS in the last slot of a wide group whose other slots have stopped
    (0-hop): the pull reads, and counts, the in-edges the query alone would."""
    for g in (cgp.gen_grid(40, 50, 0.1, 0.01, seed=5), cgp.gen_rmat(11, 8, seed=6)):
        graph = cgp.CsrGraph(g)
        s = int(g.pick_sources(1, seed=7)[0])
        o = dict(traversal_mode="pull", level_loop=loop, depth_mode="direct")
        alone = cgp.run_batch(graph, [cgp.QueryDescriptor(s, "bfs")], cgp.RunOptions(**o))
        descs = [cgp.QueryDescriptor(i % g.num_vertices, "khop", 0) for i in range(64 * words - 1)]
        r = cgp.run_batch(graph, descs + [cgp.QueryDescriptor(s, "bfs")],
                          cgp.RunOptions(mask_words=words, **o))
        np.testing.assert_array_equal(r.values[:, -1].view(np.int32), oracle.bfs(g, s, -1))
        assert r.mask_words == words
        for k in ("pull_vertices", "pull_edges", "new_pairs"):
            assert r.counters[k] == alone.counters[k], k


@pytest.mark.parametrize("kind", ["bfs", "sssp"])
def test_calls_beside_one_another_launch_their_levels(kind):
    """A traversal that would take the whole GPU for its levels runs them one
    launch each while others are on the device, and as one launch alone."""
    import threading
    import time
    g = cgp.gen_rmat(15, 16, seed=51).with_weights("u32", 1, 64, seed=52)
    graph = cgp.CsrGraph(g)
    src = g.pick_sources(48, seed=53)
    want = oracle.batch(kind, g, src)[0]
    descs = [cgp.QueryDescriptor(int(s), kind) for s in src]
    launched, exact = [0, 0, 0], [0, 0, 0]

    def caller(i):
        for _ in range(15):
            r = cgp.run_batch(graph, descs, layout="query")
            exact[i] += np.array_equal(r.values, want)
            launched[i] += r.kernel_launches > 2 * r.iterations

    threads = [threading.Thread(target=caller, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert exact == [15, 15, 15] and sum(launched) > 0
    time.sleep(0.3)  # callers count as side by side for 0.1 s
    alone = cgp.run_batch(graph, descs, layout="query")
    assert alone.kernel_launches < alone.iterations + 3
    np.testing.assert_array_equal(alone.values, want)


@pytest.mark.parametrize("q,fused", [(1, True), (3, True), (4, False), (64, False)])
def test_scatter_only_groups_by_edges_and_slots(q, fused):
    """Push mode over short lists: few (edge, slot) pairs in one launch, more
    than 2^21 level by level."""
    r = np.random.default_rng(71)
    n = 60000
    g = cgp.csr_from_edges(n, r.integers(0, n, 10 * n), r.integers(0, n, 10 * n), symmetrize=False)
    g = g.with_weights("u32", 1, 64, seed=72)
    assert 3 * g.num_edges <= 1 << 21 < 4 * g.num_edges and g.degrees().max() <= 32
    src = r.integers(0, n, q)
    got = cgp.run("sssp", cgp.CsrGraph(g), src, options=cgp.RunOptions(traversal_mode="push"),
                  layout="query")
    assert (got.kernel_launches < got.iterations) == fused
    np.testing.assert_array_equal(got.values.view(np.uint32), oracle.batch("sssp", g, src)[0])


def _islands(sizes, degree, seed):
    """Random components of the given sizes, about `degree` entries per vertex."""
    r = np.random.default_rng(seed)
    src, dst, at = [], [], 0
    for n in sizes:
        src.append(at + np.tile(np.arange(n), degree))
        dst.append(at + r.integers(0, n, n * degree))
        at += n
    return at, np.concatenate(src), np.concatenate(dst)


def _two_dense_with_hubs(n):
    """Two components, each a ring of 9 neighbours a side and a hub: one of them
    is outside whatever root is sampled, with a list of n entries."""
    r = np.arange(n)
    src = np.concatenate([np.full(n, n)] + [r] * 9)
    dst = np.concatenate([r] + [(r + j) % n for j in range(1, 10)])
    return cgp.csr_from_edges(2 * n + 2, np.r_[src, n + 1 + src], np.r_[dst, n + 1 + dst])


def _directed_with_sinks(n, sinks):
    """A dense directed component and vertices that only its out-entries lead to
    (high ids, so that they are nobody's first or second neighbour)."""
    r = np.random.default_rng(61)
    src = np.r_[np.tile(np.arange(n), 14), r.integers(0, n, sinks)]
    dst = np.r_[r.integers(0, n, 14 * n), n + np.arange(sinks)]
    return cgp.csr_from_edges(n + sinks, src, dst, symmetrize=False)


@pytest.mark.parametrize("offsets64", [False, True])
@pytest.mark.parametrize("make,launches", [
    (lambda: cgp.csr_from_edges(*_islands([900, 40, 1000, 3, 950, 1], 9, 62)), 10),
    (lambda: cgp.csr_from_edges(*_islands([33] * 200, 12, 63)), 10),
    (lambda: _two_dense_with_hubs(700), 10),
    (lambda: cgp.csr_from_edges(*_islands([2000, 1999, 30], 12, 64), symmetrize=False), 11),
    (lambda: _directed_with_sinks(1500, 400), 11),
    (lambda: cgp.csr_from_edges(*_islands([500, 20], 3, 65)), 4),
])
def test_wcc_by_sampling_and_by_every_entry(make, launches, offsets64):
    """From 8 entries per vertex on the neighbours are sampled (8 kernels, 9 with
    the transpose of a directed graph, then labels and a column), below every
    entry is linked."""
    g = make()
    graph = cgp.CsrGraph(g, offsets64=offsets64)
    assert (g.num_edges >= 8 * g.num_vertices) == (launches > 4)
    for _ in range(3):
        r = cgp.run("wcc", graph, [0])
        assert r.kernel_launches == launches
        np.testing.assert_array_equal(r.values[:, 0].view(np.uint32), oracle.wcc_components(g))
