"""The rule that decides which forwards are captured into CUDA graphs (CPU)."""
import random

import pytest

from ittai_b200.graphs import Graphs


def _run(g, keys):
    """Captures among the forwards of ``keys``, and forwards that replayed a graph."""
    captures = replays = 0
    for k in keys:
        new, graph, capture = g.use(k)
        assert not (new and capture) and not (graph and capture) and (graph is None or graph == k)
        if capture:
            g.put(k, k)
            captures += 1
        replays += graph is not None
        assert len(g.graphs) <= g.limit and len(g.seen) <= g.keys
    return captures, replays


@pytest.mark.parametrize("limit", [1, 9, 16])
def test_few_keys_are_captured_on_their_second_use(limit):
    g = Graphs(limit)
    keys = [f"k{i}" for i in range(limit)] * 10
    assert _run(g, keys) == (limit, 8 * limit)


@pytest.mark.parametrize("n,limit", [(17, 16), (56, 16), (64, 9)])
def test_more_keys_than_graphs_do_not_throw_one_another_out(n, limit):
    rng = random.Random(n)
    for keys in ([f"k{i % n}" for i in range(40 * n)], [f"k{rng.randrange(n)}" for _ in range(40 * n)]):
        captures, replays = _run(Graphs(limit), keys)
        assert captures <= 2 * limit and replays >= 0.8 * limit / n * len(keys)


def test_an_unused_graph_gives_way():
    g = Graphs(2, idle=10)
    _run(g, ["a", "a", "b", "b"])
    assert _run(g, ["c"] * 7) == (0, 0)                     # "a" was used last in the second forward
    assert _run(g, ["c", "c", "b"]) == (1, 2) and set(g.graphs) == {"b", "c"}


def test_many_keys_are_forgotten_but_graphs_stay():
    g = Graphs(2, keys=4)
    _run(g, ["a", "a"] + [f"x{i}" for i in range(20)])
    new, graph, _ = g.use("a")
    assert graph == "a" and len(g.seen) <= 4


def test_no_graphs():
    assert _run(Graphs(0), ["a"] * 5) == (0, 0)
