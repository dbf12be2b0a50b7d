"""Coset-word layers (the default plan of a Lehmer bitmap) against the oracle
and the list layers: every degree from the embedded ones (below 7) through both
word widths, directed and inverse-closed sets, sets with and without an even
generator, the smallest and largest number of generators, small orbits."""
import random

import pytest

from oracle import graph_oracle as G
from oracle import packed_oracle as P

pytestmark = pytest.mark.gpu


def _search(graph, **plan):
    from multigpubfs_b200 import GraphDefinition
    from multigpubfs_b200.engine import NativeGraph
    with NativeGraph(GraphDefinition.from_dict(graph)) as e:
        e.plan(**plan)
        r = e.run()
        return r, e.sample(0, 1000), e.sample(1, 1000)


def _generators(rng, n, count, kind):
    gens = []
    for _ in range(count):
        g = list(range(n))
        if kind == "odd":  # transpositions: no edge inside a layer
            i, j = rng.sample(range(n), 2)
            g[i], g[j] = g[j], g[i]
        elif kind == "cycle":  # one orbit of a cyclic group
            g = g[1:] + g[:1]
        else:
            rng.shuffle(g)
        gens.append(g)
    return gens


def _closed(gens):
    out = [list(g) for g in gens]
    for g in gens:
        inv = sorted(range(len(g)), key=lambda i: g[i])
        if inv not in out:
            out.append(inv)
    return out


@pytest.mark.parametrize("n", range(2, 12))
@pytest.mark.parametrize("kind", ["any", "odd", "cycle", "closed"])
def test_matches_the_oracle(n, kind):
    rng = random.Random(1000 * n + len(kind))
    for count in (1, 2, 3, 32) if n <= 9 else (2, 4):
        gens = _generators(rng, n, count, kind)
        gens = _closed(gens)[:32] if kind == "closed" else gens
        start = list(range(n))
        rng.shuffle(start)
        sizes, last, _ = P.packed_bfs(gens, start, sample=1 << 20)
        r, current, _ = _search(G.permutation_graph(gens, start))
        assert r.complete and r.layer_sizes == sizes, (n, kind, count)
        assert r.successors == len(gens) * sum(sizes)
        if sizes[-1] <= 1000:
            assert current == last, (n, kind, count)


@pytest.mark.parametrize("n,count,closed", [(7, 3, True), (8, 33, False), (9, 2, False), (10, 2, True), (12, 2, False),
                                            (12, 4, True), (13, 2, True), (13, 2, False)])
def test_matches_the_list_layers(n, count, closed):
    """Tables, samples and counts of the same search in list layers (33
    generators take them under the default plan too)."""
    rng = random.Random(n * 100 + count)
    gens = _generators(rng, n, count, "any")
    gens = _closed(gens) if closed else gens
    graph = G.permutation_graph(gens, rng.sample(range(n), n))
    lists, last, small = _search(graph, visited="bitmap", dedup="bucket" if n > 12 else "atomic")
    r, current, previous = _search(graph)
    assert r.layer_sizes == lists.layer_sizes
    assert (r.successors, r.visited_tests, r.states) == (lists.successors, lists.visited_tests, lists.states)
    assert previous == small
    if r.layer_sizes[-1] <= 1000:
        assert current == last


def test_a_finished_search_is_checkpointed_and_read_back(tmp_path):
    """The checkpoint of a finished search holds the Lehmer bitmap, which the
    coset-word layers do not make: it loads, and its search is over."""
    from multigpubfs_b200 import GraphDefinition
    from multigpubfs_b200.engine import NativeGraph
    g = GraphDefinition.from_dict(G.permutation_graph(G.lrx_generators(8), [3, 1, 4, 0, 5, 7, 2, 6]))
    with NativeGraph(g) as e:
        e.plan()
        full = e.run()
        words = sorted(e.frontier_words().tolist())
        e.checkpoint(tmp_path / "done.bin")
    with NativeGraph(g) as e:
        e.plan()
        e.resume(tmp_path / "done.bin")
        assert e.run().layer_sizes == full.layer_sizes
        assert sorted(e.frontier_words().tolist()) == words


def test_a_sweep_of_every_degree_and_width():
    """One batch of degrees 2 to 13, directed and closed: 32- and 64-bit words
    take separate waves; with predicted capacities it keeps list layers and
    gives the same tables."""
    from multigpubfs_b200.batch import BatchSweep
    rng = random.Random(5)
    graphs = []
    for n in (13, 2, 3, 6, 7, 8, 9, 10, 11):
        gens = _generators(rng, n, 2, "any")
        graphs.append(G.permutation_graph(_closed(gens) if n % 2 else gens, rng.sample(range(n), n)))
    with BatchSweep(graphs) as sweep:
        st = sweep.run()
        tables = sweep.layer_tables()
        assert st["complete_instances"] == len(graphs) and st["waves"] >= 2 and st["fatal"] == 0
        for g, table in zip(graphs, tables):
            if len(g["start"]) <= 10:
                assert table == P.packed_bfs(g["action"]["generators"], g["start"])[0]
        sweep.run(capacities=[1 << 30] * len(graphs))
        assert sweep.layer_tables() == tables
        with pytest.raises(Exception):
            sweep.run(max_depth=4)


def test_rows_by_orbits():
    """Degree 13 and 14 in one wave, rows ordered by the orbits of a generator:
    of the full length, of lengths that differ (cycles of 3, 4 and 5), of the
    rank where no generator has order 3."""
    from multigpubfs_b200.batch import BatchSweep

    def cycles(n, *lengths):
        g, at = list(range(n)), 0
        for k in lengths:
            g[at:at + k] = g[at + 1:at + k] + g[at:at + 1]
            at += k
        return g

    odd = _generators(random.Random(3), 13, 3, "odd")
    graphs = [G.permutation_graph(gens, list(range(len(gens[0])))) for gens in (
        [cycles(13, 13)], odd, [cycles(13, 3, 4, 5)], _closed([cycles(14, 14)]), [cycles(14, 5, 9)],
        _closed([cycles(13, 5, 3), cycles(13, 3, 2)]))]
    with BatchSweep(graphs) as sweep:
        st = sweep.run()
        assert st["complete_instances"] == len(graphs) and st["fatal"] == 0
        tables = sweep.layer_tables()
    for g, table in zip(graphs, tables):
        assert table == P.packed_bfs(g["action"]["generators"], g["start"], max_states=1 << 20)[0]


def test_a_checkpoint_that_list_layers_cannot_make(tmp_path):
    """Coset words fit a budget of 96 MB that the list layers of the same search
    do not: the search completes, its checkpoint is refused, and the handle
    keeps the table and the states."""
    import torch
    from multigpubfs_b200 import GraphDefinition, native
    from multigpubfs_b200.engine import NativeGraph
    rng = random.Random(11)
    graph = GraphDefinition.from_dict(G.permutation_graph(_closed(_generators(rng, 11, 4, "any")), list(range(11))))
    with NativeGraph(graph) as e:
        e.plan()
        want = e.run()
        words, samples = sorted(e.frontier_words().tolist()), (e.sample(0), e.sample(1))
        assert max(want.layer_sizes) > 6 << 20  # more than (96 MB - the bitmap) / 16 bytes
        native.trim_memory(0)
        torch.cuda.empty_cache()
        # The plan's free memory may be some seconds old: its own capacity (16
        # bytes a state beside the bitmap) says what budget a reserve leaves.
        reserve = torch.cuda.mem_get_info()[0] - (300 << 20)
        info = e.plan(reserve_bytes=reserve)
        assert info["capacity"] < info["state_bound"]
        reserve += 16 * info["capacity"] + info["bitmap_bits"] // 8 - (96 << 20)
        info = e.plan(reserve_bytes=reserve)
        assert 5 << 20 < info["capacity"] < 6 << 20 and e.search_form() == "coset"
        r = e.run()
        assert r.complete and r.layer_sizes == want.layer_sizes
        path = tmp_path / "refused.bin"
        with pytest.raises(native.NativeError):
            e.checkpoint(path)
        assert not path.exists()
        assert e.layer_table()[0] == want.layer_sizes
        assert sorted(e.frontier_words().tolist()) == words
        assert (e.sample(0), e.sample(1)) == samples


def test_list_layers_after_another_plan_hold_no_coset_words():
    """A handle that ran S12 in coset words (two buffers of 61 MB, a table of 13
    MB) and is planned again for list layers holds their 60 MB bitmap and small
    frontiers."""
    import torch
    from multigpubfs_b200 import GraphDefinition, native
    from multigpubfs_b200.engine import NativeGraph
    graph = GraphDefinition.from_dict(G.permutation_graph(G.lrx_generators(12), list(range(12))))

    def free():
        native.trim_memory(0)
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    with NativeGraph(graph) as e:
        e.plan()
        sizes = e.run().layer_sizes
    before = free()
    with NativeGraph(graph) as e:
        e.plan()
        assert e.run().layer_sizes == sizes
        e.plan(dedup="atomic")
        assert e.run(max_layers=5).layer_sizes == sizes[:5]
        assert before - free() < 110 << 20


def _wreath(k, blocks):
    """S_k wr S_blocks on k * blocks points: two generators of one block, two of
    the blocks."""
    n = k * blocks
    return [list(range(1, k)) + [0] + list(range(k, n)), [1, 0] + list(range(2, n)),
            [(i + k) % n for i in range(n)], list(range(k, 2 * k)) + list(range(k)) + list(range(2 * k, n))]


@pytest.mark.parametrize("name,form", [("C12", "coset"), ("C13", "lists"), ("AGL(1,13)", "lists"), ("S2 wr S7", "lists"),
                                       ("S7 wr S2", "lists"), ("A13", "coset"), ("LRX13", "coset"), ("S13", "coset"),
                                       ("S14", "coset")])
def test_small_orbits_of_wide_words_are_searched_in_lists(name, form):
    """At 13 and 14 symbols a group other than A_n and S_n keeps list layers;
    its table is that of the oracle, or of its bound."""
    from multigpubfs_b200 import GraphDefinition
    from multigpubfs_b200.engine import NativeGraph
    rng = random.Random(14)
    gens = {"C12": lambda: _closed([list(range(1, 12)) + [0]]), "C13": lambda: _closed([list(range(1, 13)) + [0]]),
            "AGL(1,13)": lambda: [[(i + 1) % 13 for i in range(13)], [2 * i % 13 for i in range(13)]],
            "S2 wr S7": lambda: _closed(_wreath(2, 7)), "S7 wr S2": lambda: _wreath(7, 2),
            "A13": lambda: [list(range(1, 13)) + [0], [1, 2, 0] + list(range(3, 13))],
            "LRX13": lambda: G.lrx_generators(13),
            "S13": lambda: [rng.sample(range(13), 13) for _ in range(3)],
            "S14": lambda: _closed([rng.sample(range(14), 14) for _ in range(2)])}[name]()
    graph = G.permutation_graph(gens, rng.sample(range(len(gens[0])), len(gens[0])))
    with NativeGraph(GraphDefinition.from_dict(graph)) as e:
        e.plan()
        assert e.search_form() == form
        if name in ("A13", "LRX13", "S13", "S14"):
            return
        r = e.run()
        assert r.complete and e.search_form() == form
        if name == "S7 wr S2":
            assert sum(r.layer_sizes) == 2 * 5040 ** 2
        else:
            assert r.layer_sizes == P.packed_bfs(gens, graph["start"], max_states=1 << 20)[0]
