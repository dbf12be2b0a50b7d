"""Unipotent-ring layers (2x2 matrices over a prime field under the default plan)
against the list layers: the smallest and largest prime of each ring width, the
switch from list layers, singular and non-unit starts, determinants that
spread slowly, at once or not at all."""
import pytest

from multigpubfs_b200 import workloads

pytestmark = pytest.mark.gpu


def _search(graph, **plan):
    from multigpubfs_b200 import GraphDefinition
    from multigpubfs_b200.engine import NativeGraph
    with NativeGraph(GraphDefinition.from_dict(graph)) as e:
        e.plan(**plan)
        r = e.run()
        return r, e.sample(0, 1000), e.sample(1, 1000), sorted(e.frontier_words().tolist())


# 13 is below the rings' primes; 101 and 103 lie on the two sides of
# the node count from which list layers go first.
@pytest.mark.parametrize("p", [13, 17, 31, 37, 61, 67, 101, 103, 127, 131])
@pytest.mark.parametrize("start", [[1, 0, 0, 1], [2, 5, 3, 1], [0, 0, 4, 7], [0, 3, 0, 0]])
def test_matches_the_list_layers(p, start):
    graph = workloads.gl2_graph(p)
    graph["start"] = start
    lists, last, small, words = _search(graph, visited="bitmap", dedup="atomic")
    r, current, previous, front = _search(graph)
    assert r.complete and r.layer_sizes == lists.layer_sizes
    assert (r.states, r.successors, r.visited_tests) == (lists.states, lists.successors, lists.visited_tests)
    assert previous == small and front == words
    if r.layer_sizes[-1] <= 1000:
        assert current == last
    assert len(r.layer_seconds) == len(r.layer_sizes) - 1


def test_largest_prime_and_composite_modulus():
    """257 is a ring of nine words; a composite modulus keeps list layers."""
    for m, states in ((257, (257 ** 2 - 1) * (257 ** 2 - 257)), (221, None)):
        graph = workloads.gl2_graph(257)
        if m != 257:
            graph["action"]["generators"] = [{"matrix": [1, 1, 0, 1], "modulo": m}, {"matrix": [1, m - 1, 0, 1], "modulo": m},
                                             {"matrix": [0, 1, 1, 0], "modulo": m}]
            graph["generator_names"] = ["a", "b", "c"]
        r, _, small, words = _search(graph)
        lists, _, expect, front = _search(graph, visited="bitmap", dedup="atomic")
        assert r.layer_sizes == lists.layer_sizes and small == expect and words == front
        assert states is None or r.states == states


def _closed(p, matrices):
    """A graph of the matrices and their inverses mod p."""
    every = []
    for a, b, c, d in matrices:
        i = pow(a * d - b * c, -1, p)
        for m in ((a, b, c, d), (d * i % p, -b * i % p, -c * i % p, a * i % p)):
            if list(m) not in every:
                every.append(list(m))
    graph = workloads.gl2_graph(p)
    graph["action"]["generators"] = [{"matrix": m, "modulo": p} for m in every]
    graph["generator_names"] = [str(i) for i in range(len(every))]
    return graph


# Six to eight words a ring; determinant 1 only, many at once, and a small
# group over all of them; long searches that stay below the rings' layers, and
# one that comes to them late.
@pytest.mark.parametrize("p,matrices", [
    (163, [(1, 1, 0, 1), (1, 0, 1, 1), (2, 0, 0, 1)]),
    (193, [(1, 1, 0, 1), (1, 0, 1, 1)]),
    (223, [(0, 1, 222, 0), (1, 1, 0, 1), (222, 0, 0, 222)]),
    (251, [(1, 1, 0, 1), (0, 1, 1, 0), (6, 0, 0, 1)]),
    (67, [(3, 1, 4, 7), (5, 2, 0, 9), (0, 1, 11, 0), (2, 0, 0, 1), (6, 6, 1, 3)]),
    (61, [(2, 0, 0, 1), (0, 1, 1, 0)]),
    (37, [(1, 1, 0, 1)]),
    (127, [(3, 0, 0, 1), (0, 1, 1, 0)]),
    (113, [(1, 1, 0, 1), (3, 0, 0, 1), (1, 0, 0, 3)]),
])
def test_generator_sets(p, matrices):
    graph = _closed(p, matrices)
    graph["start"] = [1, 2, 0, 3]
    lists, last, small, words = _search(graph, visited="bitmap", dedup="atomic")
    r, current, previous, front = _search(graph)
    assert r.complete and r.layer_sizes == lists.layer_sizes
    assert previous == small and front == words
    if r.layer_sizes[-1] <= 1000:
        assert current == last


def test_a_finished_search_is_checkpointed_and_read_back(tmp_path):
    from multigpubfs_b200 import GraphDefinition
    from multigpubfs_b200.engine import NativeGraph
    g = GraphDefinition.from_dict(workloads.gl2_graph(37))
    with NativeGraph(g) as e:
        e.plan()
        full = e.run()
        e.checkpoint(tmp_path / "done.bin")
    with NativeGraph(g) as e:
        e.plan()
        e.resume(tmp_path / "done.bin")
        assert e.run().layer_sizes == full.layer_sizes
