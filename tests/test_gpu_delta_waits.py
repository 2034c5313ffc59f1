"""Waits inside the delta loop: they last as long as the others get on, however long that is, and a
fixpoint whose wait did run out is evaluated by the routes that have none."""
import numpy as np
import pytest

from oracle import oracle as O
from xlog_b200 import programs, workloads
from xlog_b200.executor import run_program
from xlog_b200.plan import CompiledRule, ExecutionPlan, Join, Project, Scan, Scc
from xlog_b200.provider import KernelProvider

from test_gpu_delta_loop import U2, chain
from test_gpu_delta_slots import hub_ladder, two_rules

pytestmark = pytest.mark.gpu


def run(monkeypatch, plan, inputs, out, polls=None):
    if polls is not None:
        monkeypatch.setenv("XLB_DELTA_POLLS", str(polls))
    p = KernelProvider(device=0)
    try:
        got, stats = run_program(p, plan, inputs, [out])
    finally:
        p.close()
    return got[out], stats


def steps(rules):
    # p(X,Y) :- s(X,Y).  p(Y,Z) :- p(X,Y), e(Y,Z).  (the second rule twice over: e and f)
    ids = {"s": 0, "e": 1, "f": 2, "p": 3}
    return ExecutionPlan([Scc(0, True, [CompiledRule("p", Scan(0), U2)] + [CompiledRule("p", Project(Join(Scan(3), Scan(r), [1], [0]), [1, 3]), U2) for r in (1, 2)[:rules]])], ids)


@pytest.mark.parametrize("rules", [1, 2])
def test_a_long_phase_of_one_block_is_waited_for(rules, monkeypatch):
    # 60 000 iterations by one block, some 50 ms; the others may see nothing for about 10 ms
    n = 60_000
    e = chain(n)
    rels = {"s": [np.array([0], np.uint32), np.array([1], np.uint32)], "e": [e[0][1:], e[1][1:]], "f": [np.array([n], np.uint32), np.array([n], np.uint32)]}
    got, stats = run(monkeypatch, steps(rules), rels, "p", polls=10_000)
    assert np.array_equal(got[0], e[0]) and np.array_equal(got[1], e[1])
    assert stats["iterations"] == n - 1 and stats["kernel_launches"] < 100  # by the loop, not iteration by iteration


@pytest.mark.parametrize("name,plan,rels,out", [
    ("ladder", two_rules(), hub_ladder(50, 1, 3, 4), "p"),
    ("same generation", programs.same_generation(), {"edge": list(workloads.tree_dag(300, 0.05)[:2])}, "sg"),
    ("doubling", programs.transitive_closure_nonlinear(), {"edge": list(workloads.uniform_digraph(200, 500, 5))}, "reach"),
], ids=lambda x: x if isinstance(x, str) else "")
def test_a_wait_that_runs_out_falls_back(name, plan, rels, out, monkeypatch):
    by_loop, fast = run(monkeypatch, plan, rels, out)
    # (one poll: less than any iteration takes)
    got, stats = run(monkeypatch, plan, rels, out, polls=1)
    want, _ = O.run_program(plan, rels, [out])
    for g, w, b in zip(got, want[out], by_loop):
        assert np.array_equal(g, w) and np.array_equal(b, w)
    assert stats["kernel_launches"] > fast["kernel_launches"]
    assert (stats["iterations"], stats["candidate_tuples"]) == (fast["iterations"], fast["candidate_tuples"])


# No wait of any block is given a second look: of some 2000, all would have to be over at the first for the kernel to finish
@pytest.mark.parametrize("name,plan,rels,out", [
    ("same generation", programs.same_generation(), {"edge": list(workloads.tree_dag(1200, 0.05)[:2])}, "sg"),
    ("same generation of 13 bits", programs.same_generation(), {"edge": list(workloads.tree_dag(5000, 0.05)[:2])}, "sg"),
    ("points-to", programs.andersen(), {k: list(v) for k, v in workloads.andersen_program(0.0002, 11).items()}, "pt"),
    ("points-to of 12 bits", programs.andersen(), {k: list(v) for k, v in workloads.andersen_program(0.001, 11).items()}, "pt"),
    ("ladder", two_rules(), hub_ladder(50, 1, 3, 4), "p"),
], ids=lambda x: x if isinstance(x, str) else "")
def test_a_wait_that_is_not_over_falls_back(name, plan, rels, out, monkeypatch):
    by_kernel, fast = run(monkeypatch, plan, rels, out)
    got, stats = run(monkeypatch, plan, rels, out, polls=0)
    for g, b in zip(got, by_kernel):
        assert np.array_equal(g, b)
    assert stats["kernel_launches"] > fast["kernel_launches"] + 10  # iteration by iteration
    if "bits" not in name:  # (the others take the oracle long)
        for g, w in zip(got, O.run_program(plan, rels, [out])[0][out]):
            assert np.array_equal(g, w)
    assert (stats["iterations"], stats["candidate_tuples"]) == (fast["iterations"], fast["candidate_tuples"])


@pytest.mark.parametrize("name,plan,rels,out", [
    ("same generation", programs.same_generation(), {"edge": list(workloads.tree_dag(1200, 0.05)[:2])}, "sg"),
    ("points-to", programs.andersen(), {k: list(v) for k, v in workloads.andersen_program(0.0002, 11).items()}, "pt"),
], ids=lambda x: x if isinstance(x, str) else "")
def test_waits_of_the_kernels_by_rows(name, plan, rels, out, monkeypatch):
    # (whether one poll is enough is a matter of luck: the result and the counts are the same either way)
    got, fast = run(monkeypatch, plan, rels, out)
    again, stats = run(monkeypatch, plan, rels, out, polls=1)
    for g, a in zip(got, again):
        assert np.array_equal(g, a)
    assert (stats["iterations"], stats["candidate_tuples"]) == (fast["iterations"], fast["candidate_tuples"])
