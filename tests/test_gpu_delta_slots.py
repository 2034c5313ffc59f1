"""Iterations of the delta loop that one block begins alone and that turn out to hold long rows, many
of them in one fixpoint: each such iteration is finished by all blocks, and the counters of the next one
have to be clean whichever way it was reached."""
import numpy as np
import pytest

from oracle import oracle as O
from xlog_b200 import programs
from xlog_b200.plan import CompiledRule, ExecutionPlan, Join, Project, Scan, Scc

from test_gpu_delta_loop import U2, both

pytestmark = pytest.mark.gpu


def two_rules():
    # p(X,Y) :- s(X,Y).  p(Y,Z) :- p(X,Y), e(Y,Z).  p(Y,Z) :- p(X,Y), f(Y,Z).
    ids = {"s": 0, "e": 1, "f": 2, "p": 3}
    step = [CompiledRule("p", Project(Join(Scan(3), Scan(r), [1], [0]), [1, 3]), U2) for r in (1, 2)]
    return ExecutionPlan([Scc(0, True, [CompiledRule("p", Scan(0), U2)] + step)], ids)


def hub_ladder(width, parents, hubs, gap, leaves=600):
    """`width` paths side by side; every `gap` levels `parents` of them step to a node with `leaves`
    successors (and on)."""
    levels = (hubs + 1) * gap
    node = lambda level, k: 1 + level * width + k  # noqa: E731
    top = 1 + (levels + 1) * width
    e, f = [], []
    for level in range(levels):
        for k in range(width):
            (e if k % 2 else f).append((node(level, k), node(level + 1, k)))
        if level % gap == gap - 1 and level // gap < hubs:
            hub = top + (level // gap) * (leaves + 1)
            e += [(node(level, k), hub) for k in range(parents)]
            f += [(hub, hub + 1 + i) for i in range(leaves)]
    cols = lambda rows: [np.array(c, dtype=np.uint32) for c in zip(*rows)]  # noqa: E731
    return {"s": cols([(0, node(0, k)) for k in range(width)]), "e": cols(e), "f": cols(f)}


def twin_tree(hubs, gap, twins, children):
    """`twins` paths below one root; every `gap` levels each of their nodes has `children` children, the first
    of which the path goes on with."""
    edge, at, top = [], list(range(1, twins + 1)), twins + 1
    edge += [(0, x) for x in at]
    for level in range((hubs + 1) * gap):
        n = children if level % gap == gap - 1 and level // gap < hubs else 1
        for k, x in enumerate(at):
            edge += [(x, top + i) for i in range(n)]
            at[k] = top
            top += n
    return [np.array(c, dtype=np.uint32) for c in zip(*edge)]


@pytest.mark.parametrize("width,parents,hubs,gap", [(50, 1, 7, 6), (200, 1, 7, 6), (200, 40, 7, 6), (1400, 3, 5, 7), (60, 60, 4, 1)])
def test_many_iterations_with_long_rows(width, parents, hubs, gap, monkeypatch):
    rels = hub_ladder(width, parents, hubs, gap)
    got, it, cand = both(two_rules(), rels, "p", monkeypatch)
    want, stats = O.run_program(two_rules(), rels, ["p"])
    assert it == (hubs + 1) * gap + 1
    assert len(got[0]) == sum(len(r[0]) for r in rels.values())
    for g, w in zip(got, want["p"]):
        assert np.array_equal(g, w)


@pytest.mark.parametrize("hubs,gap,twins,children", [(7, 6, 2, 23), (6, 4, 5, 23), (5, 7, 3, 40)])
def test_same_generation_of_large_families(hubs, gap, twins, children, monkeypatch):
    edge = twin_tree(hubs, gap, twins, children)
    got, _, _ = both(programs.same_generation(), {"edge": edge}, "sg", monkeypatch)
    want, _ = O.run_program(programs.same_generation(), {"edge": edge}, ["sg"])
    for g, w in zip(got, want["sg"]):
        assert np.array_equal(g, w)
