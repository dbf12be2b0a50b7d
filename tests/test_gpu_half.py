"""Half-rank layers (repeated labels under the default plan) against the oracle
and the list layers: one to six labels, odd and even degrees, both sides of the
limits that send a start to the general paths, directed sets and the wide
starts of more than 16 positions."""
import random

import pytest

from oracle import graph_oracle as G
from oracle import packed_oracle as P

pytestmark = pytest.mark.gpu


def _search(graph, **plan):
    from multigpubfs_b200 import GraphDefinition
    from multigpubfs_b200.engine import NativeGraph
    with NativeGraph(GraphDefinition.from_dict(graph)) as e:
        info = e.plan(**plan)
        r = e.run()
        words = sorted(e.frontier_words().tolist()) if info["packed"] else None
        return r, e.sample(0, 1000), e.sample(1, 1000), words


def _start(rng, n, labels):
    names = rng.sample(range(-50, 50), labels)
    start = [names[i % labels] for i in range(n)]
    rng.shuffle(start)
    return start


# Repeated labels, domains small enough for a quick comparison.
@pytest.mark.parametrize("n,labels", [(n, labels) for n in (2, 3, 7, 8, 9, 13, 15, 16) for labels in range(1, 8)
                                      if labels < n and (n <= 13 or labels <= 4)])
def test_packed_starts(n, labels):
    rng = random.Random(100 * n + labels)
    closed = labels % 2 == 0
    gens = G.lrx_generators(n) if closed else [rng.sample(range(n), n) for _ in range(3)]
    graph = G.permutation_graph(gens, _start(rng, n, labels))
    lists, last, small, words = _search(graph, visited="bitmap", dedup="atomic")
    r, current, previous, front = _search(graph)
    assert r.layer_sizes == lists.layer_sizes
    assert (r.states, r.successors, r.visited_tests) == (lists.states, lists.successors, lists.visited_tests)
    assert previous == small and front == words
    if r.layer_sizes[-1] <= 1000:
        assert current == last
    if n <= 9:
        assert r.layer_sizes == P.packed_bfs(gens, graph["start"])[0]


@pytest.mark.parametrize("n,labels", [(17, 1), (17, 2), (18, 2), (17, 3), (17, 4), (17, 5), (24, 2), (37, 2)])
@pytest.mark.parametrize("closed", [True, False])
def test_wide_starts(n, labels, closed):
    """More than 16 positions, against the wide hash (visited="hash" asks for
    it); 17 positions of five labels and 37 of two keep the hash by default."""
    rng = random.Random(10 * n + labels)
    start = [0] * (n - 3) + [1, 1, 2][:3] if n == 37 else _start(rng, n, labels)
    if n == 37:
        start = [min(x, 1) for x in start]
    gens = G.lrx_generators(n) if closed else G.lrx_generators(n)[::2]
    if labels == 5:
        start = [0] * (n - 4) + [1, 2, 3, 4]
    graph = G.permutation_graph(gens, start)
    lists, last, small, _ = _search(graph, visited="hash")
    r, current, previous, _ = _search(graph)
    assert r.complete and r.layer_sizes == lists.layer_sizes
    assert (r.states, r.successors, r.visited_tests) == (lists.states, lists.successors, lists.visited_tests)
    assert previous == small
    if r.layer_sizes[-1] <= 1000:
        assert current == last


def test_the_bitmap_is_the_list_layers(tmp_path):
    """A checkpoint of a finished search loads, and one of list layers goes on
    to the same table."""
    from multigpubfs_b200 import GraphDefinition
    from multigpubfs_b200.engine import NativeGraph
    g = GraphDefinition.from_dict(G.permutation_graph(G.lrx_generators(12), [i % 4 for i in range(12)]))
    with NativeGraph(g) as e:
        e.plan()
        full = e.run()
        e.checkpoint(tmp_path / "done.bin")
        e.run(max_layers=9)
        e.checkpoint(tmp_path / "part.bin")
    for name in ("done.bin", "part.bin"):
        with NativeGraph(g) as e:
            e.plan()
            e.resume(tmp_path / name)
            assert e.run().layer_sizes == full.layer_sizes


def _terms(gens):
    """Displacement terms of a generator set: the distinct shifts of each."""
    return sum(len({x - i for i, x in enumerate(g)}) for g in gens)


@pytest.mark.parametrize("case", ["below", "above", "reversals"])
def test_wide_starts_of_many_generators(case):
    """Half-rank layers hold 512 displacement terms; the sets on both sides of
    that (random permutations of 24 positions, all 31 prefix reversals of 32)
    are searched under the default plan."""
    if case == "reversals":
        gens = [list(range(k))[::-1] + list(range(k, 32)) for k in range(2, 33)]
        start = [1, 1, 1] + [0] * 29
    else:
        rng = random.Random(24)
        gens = [rng.sample(range(24), 24) for _ in range(32)]
        while case == "below" and _terms(gens) > 512:
            gens.pop()
        start = [1] * 4 + [0] * 20
    assert (_terms(gens) <= 512) == (case == "below") and len(gens) > 16
    graph = G.permutation_graph(gens, start)
    lists, last, small, _ = _search(graph, visited="hash")
    r, current, previous, _ = _search(graph)
    assert r.complete and r.layer_sizes == lists.layer_sizes
    assert previous == small
    if r.layer_sizes[-1] <= 1000:
        assert current == last


@pytest.mark.parametrize("limit", [1, 999, 1000, 1001, 1820, 5000])
def test_samples_of_a_large_deepest_layer(limit):
    """Star transpositions on 20 positions, four of them marked: 1,820 states
    in the deepest layer, more than the rows a search copies to the host."""
    from multigpubfs_b200 import GraphDefinition
    from multigpubfs_b200.engine import NativeGraph
    n, start = 20, [7] * 4 + [-3] * 16
    gens = []
    for i in range(1, n):
        g = list(range(n))
        g[0], g[i] = i, 0
        gens.append(g)
    graph = GraphDefinition.from_dict(G.permutation_graph(gens, start))
    with NativeGraph(graph) as e:
        e.plan(visited="hash")
        whole = e.run()
        rows = e.sample(0, 5000)
    with NativeGraph(graph) as e:
        e.plan()
        r = e.run()
        got = e.sample(0, limit)
    assert r.layer_sizes == whole.layer_sizes and len(rows) == r.layer_sizes[-1] == 1820
    assert len(got) == min(limit, 1820) and got == sorted(got)
    assert len({tuple(x) for x in got}) == len(got) and {tuple(x) for x in got} <= {tuple(x) for x in rows}


def test_lists_that_do_not_fit_leave_the_search_to_the_hash():
    """C(30, 15) = 155 M arrangements bound the layers of a shift's 30 states:
    with 1.5 GB left on the device when the search runs, half-rank layers do not
    get their two lists of 1.24 GB, and the wide hash needs a few MB."""
    import torch
    from multigpubfs_b200 import GraphDefinition, native
    from multigpubfs_b200.engine import NativeGraph
    shift = list(range(1, 30)) + [0]
    graph = GraphDefinition.from_dict(G.permutation_graph([shift, [29] + list(range(29))], [1] * 15 + [0] * 15))
    native.trim_memory(0)
    torch.cuda.empty_cache()
    with NativeGraph(graph) as e:
        e.plan()
        free, _ = torch.cuda.mem_get_info()
        hold = torch.empty(free - (1536 << 20), dtype=torch.uint8, device="cuda")
        try:
            r = e.run()
            rows = e.sample(0)
        finally:
            del hold
            torch.cuda.empty_cache()
        assert r.complete and r.layer_sizes == [1] + [2] * 14 + [1]
        assert rows == [[0] * 15 + [1] * 15]
        assert e.run().layer_sizes == r.layer_sizes and e.sample(0) == rows
