"""The delta loop (linear recursive rules run to their fixpoint by one kernel) against the oracle and
against the general loop: iterations of one row and of many, rows with more matches than a warp
takes, two joined relations, several rules, a log that has to grow, the iteration limit."""
import numpy as np
import pytest

from oracle import oracle as O
from xlog_b200 import _abi as A
from xlog_b200 import programs, workloads
from xlog_b200.executor import run_program
from xlog_b200.lib import XlbError
from xlog_b200.plan import CompiledRule, ExecutionPlan, Join, Project, Scan, Scc
from xlog_b200.provider import KernelProvider

pytestmark = pytest.mark.gpu
U2 = (A.U32, A.U32)


def both(plan, inputs, out, monkeypatch, **kw):
    res = []
    for off in (False, True):
        if off:
            monkeypatch.setenv("XLB_NO_DELTA_LOOP", "1")
        else:
            monkeypatch.delenv("XLB_NO_DELTA_LOOP", raising=False)
        p = KernelProvider(device=0, **kw)
        got, stats = run_program(p, plan, inputs, [out])
        p.close()
        res.append((got[out], stats["iterations"], stats["candidate_tuples"]))
    for a, b in zip(res[0][0], res[1][0]):
        assert np.array_equal(a, b)
    assert res[0][1:] == res[1][1:]
    return res[0]


def star(hub, leaves):
    """hub -> leaves -> hub' -> leaves': rows with `leaves` matches."""
    l0 = np.arange(10, 10 + leaves, dtype=np.uint32)
    return [np.concatenate([np.full(leaves, hub), l0]).astype(np.uint32), np.concatenate([l0, np.full(leaves, hub + 1)]).astype(np.uint32)]


def chain(n):
    return [np.arange(n - 1, dtype=np.uint32), np.arange(1, n, dtype=np.uint32)]


@pytest.mark.parametrize("edge", [chain(2), chain(3), chain(300), star(1, 511), star(1, 513), star(1, 40000)], ids=["one", "two", "chain", "row511", "row513", "row40000"])
@pytest.mark.parametrize("program", [programs.transitive_closure, programs.transitive_closure_left_linear, programs.transitive_closure_swapped_head])
def test_closure(edge, program, monkeypatch):
    got, _, _ = both(program(), {"edge": edge}, "reach", monkeypatch)
    want, _ = O.run_program(program(), {"edge": edge}, ["reach"])
    for g, w in zip(got, want["reach"]):
        assert np.array_equal(g, w)


def paths(tail):
    """A path of 33 to 70 edges that ends in nothing, in a loop back, in a branch that closes again (and a second path
    behind it), in a value with 40 matches: what a row that is followed as a path can run into."""
    a, b = list(range(70)), list(range(1, 71))
    if tail == "loop":
        a, b = a + [70], b + [3]
    elif tail == "itself":
        a, b = a + [70], b + [70]
    elif tail == "branch":
        a, b = a + [70, 70, 71, 72] + list(range(73, 140)), b + [71, 72, 73, 73] + list(range(74, 141))
    elif tail == "fan":
        a, b = a + [70] * 40, b + list(range(71, 111))
    return np.array(a, np.uint32), np.array(b, np.uint32)


# (ids up to 2^11 and 2^14: every value has an entry in a row's queue; up to 2^15: it has not)
@pytest.mark.parametrize("top", [200, 2047, (1 << 14) - 1, (1 << 15) - 1])
@pytest.mark.parametrize("tail", ["end", "loop", "itself", "branch", "fan"])
def test_rows_that_follow_a_path(tail, top, monkeypatch):
    edge = [np.where(x == 0, top, x).astype(np.uint32) for x in paths(tail)]
    both(programs.transitive_closure(), {"edge": edge}, "reach", monkeypatch)


# Followed for 32 levels and more (a level for 96 values: 85 of 13 bits, 170 of 14), walked, cut short by a twig, later tried again
@pytest.mark.parametrize("top", [1000, 8191, (1 << 14) - 1])
@pytest.mark.parametrize("every", [33, 40, 72, 73, 200, 500])
@pytest.mark.parametrize("back", [None, 0, 590, 600])
def test_rows_that_are_walked(top, every, back, monkeypatch):
    n = 600
    twigs = np.arange(every // 2, n, every)
    src = [np.arange(n), twigs, [top]] + ([] if back is None else [[n]])
    dst = [np.arange(1, n + 1), n + 1 + np.arange(len(twigs)), [0]] + ([] if back is None else [[back]])
    both(programs.transitive_closure(), {"edge": [np.concatenate(c).astype(np.uint32) for c in (src, dst)]}, "reach", monkeypatch)


@pytest.mark.parametrize("limit", [31, 32, 33, 34, 69, 70])
def test_iteration_limit_on_a_path(limit):
    p = KernelProvider(device=0, max_iterations=limit)
    if limit == 70:  # 71 nodes
        got, stats = run_program(p, programs.transitive_closure(), {"edge": list(paths("end"))}, ["reach"])
        assert len(got["reach"][0]) == 71 * 70 // 2 and stats["iterations"] == 70 and stats["candidate_tuples"] == 71 * 70 // 2
    else:
        with pytest.raises(XlbError) as e:
            run_program(p, programs.transitive_closure(), {"edge": list(paths("end"))}, ["reach"])
        assert e.value.status == A.ERR_ITER_LIMIT
    p.close()


# values with as many matches as a row of the head has words (1, 2, 16, 32, 64; 128 are too many), and fewer; some edges twice
@pytest.mark.parametrize("nodes,degree", [(20, 8), (60, 4), (500, 40), (500, 12), (1000, 40), (1500, 70), (3000, 130)])
def test_dense_closures(nodes, degree, monkeypatch):
    rng = np.random.default_rng(nodes)
    hubs = rng.integers(0, nodes // 2, nodes * degree)  # a part of the nodes has no successor
    e = [np.append(hubs, nodes - 1).astype(np.uint32), np.append(rng.integers(0, nodes, nodes * degree), 0).astype(np.uint32)]
    e = [np.concatenate([c, c[:50]]) for c in e]
    both(programs.transitive_closure(), {"edge": e}, "reach", monkeypatch)
    # a path of such blocks: a level for each
    b = nodes // 10 + 1
    k = 10 * b
    src = np.repeat(np.arange(k - b), 2)
    dst = (src // b + 1) * b + rng.integers(0, b, len(src))
    dense = [np.concatenate([src, np.repeat(np.arange(b), 9 * b)]).astype(np.uint32), np.concatenate([dst, np.tile(np.arange(b, k), b)]).astype(np.uint32)]
    both(programs.transitive_closure(), {"edge": dense}, "reach", monkeypatch)


# Dense, with rows that are done at once (no successor, or the last of a band) beside rows that are not
@pytest.mark.parametrize("kind", ["band", "skewed", "bipartite", "bipartite and back"])
@pytest.mark.parametrize("nodes,degree", [(128, 70), (600, 40), (2000, 70)])
def test_dense_closures_of_uneven_rows(kind, nodes, degree, monkeypatch):
    rng = np.random.default_rng(nodes)
    n = nodes * degree
    if kind == "band":
        u = rng.integers(0, nodes, n)
        v = np.minimum(u + rng.integers(1, 40, n), nodes - 1)
    elif kind == "skewed":
        u, v = (np.minimum((rng.random(n) ** 6 * nodes).astype(int), nodes - 1) for _ in range(2))
    else:
        u, v = rng.integers(0, nodes // 20 + 1, n), rng.integers(nodes // 20 + 1, nodes, n)
        if kind != "bipartite":
            u, v = np.append(u, rng.integers(0, nodes, 50)), np.append(v, rng.integers(0, nodes, 50))
    both(programs.transitive_closure(), {"edge": [np.append(u, 0).astype(np.uint32), np.append(v, nodes - 1).astype(np.uint32)]}, "reach", monkeypatch)


def test_many_long_rows(monkeypatch):
    # 70 sources with 1100 matches each twice over: the list of long rows is used by many warps at once
    src = np.repeat(np.arange(70, dtype=np.uint32), 1100)
    mid = np.tile(np.arange(100, 1200, dtype=np.uint32), 70)
    back = [np.arange(100, 1200, dtype=np.uint32), np.arange(1100, dtype=np.uint32) % 70]
    both(programs.transitive_closure(), {"edge": [np.concatenate([src, back[0]]), np.concatenate([mid, back[1]])]}, "reach", monkeypatch)


@pytest.mark.parametrize("nodes", [40, 701])
def test_same_generation(nodes, monkeypatch):
    c0, c1, _ = workloads.tree_dag(nodes, 0.05)
    got, _, _ = both(programs.same_generation(), {"edge": [c0, c1]}, "sg", monkeypatch)
    want, _ = O.run_program(programs.same_generation(), {"edge": [c0, c1]}, ["sg"])
    for g, w in zip(got, want["sg"]):
        assert np.array_equal(g, w)


def sides(kinds):
    """p(X,Y) :- s(X,Y), then one rule per kind: both columns led on, the first, the second."""
    ids = {"s": 0, "a": 1, "b": 2, "p": 3}
    rules = [CompiledRule("p", Scan(0), U2)]
    for k in kinds:
        if k == "both":    # p(X,Y) :- a(P,X), p(P,Q), b(Q,Y)
            rules.append(CompiledRule("p", Project(Join(Join(Scan(1), Scan(3), [0], [0]), Scan(2), [3], [0]), [1, 5]), U2))
        elif k == "first":  # p(X,Y) :- a(P,X), p(P,Y)
            rules.append(CompiledRule("p", Project(Join(Scan(1), Scan(3), [0], [0]), [1, 3]), U2))
        else:              # p(X,Y) :- p(X,Q), b(Q,Y)
            rules.append(CompiledRule("p", Project(Join(Scan(3), Scan(2), [1], [0]), [0, 3]), U2))
    return ExecutionPlan([Scc(0, True, rules)], ids)


# heads of 4 to 14 bits a column: too few in all for bit rows, a row of two words, of one per lane, of eight, too long
@pytest.mark.parametrize("kinds", [("both",), ("first",), ("both", "second"), ("first", "second", "both")], ids="-".join)
@pytest.mark.parametrize("hi,lo,rows", [(10, 40, 60), (8191, 100, 9000), (8000, 63, 9000), (130, 8191, 3000), (1000, 1023, 1500), (1500, 1500, 2000), (8000, 8191, 9000), (300, 16000, 9000)])
def test_columns_led_on_apart(hi, lo, rows, kinds, monkeypatch):
    rng = np.random.default_rng(hi * lo)
    pairs = lambda n, x, y: [rng.integers(0, x, n).astype(np.uint32), rng.integers(0, y, n).astype(np.uint32)]  # noqa: E731
    s = pairs(40, hi, lo)
    s[0][0], s[1][0] = hi - 1, lo - 1
    both(sides(kinds), {"s": s, "a": pairs(rows, hi, hi), "b": pairs(rows, lo, lo)}, "p", monkeypatch)


@pytest.mark.parametrize("fan", [16, 17, 1024, 1025])
def test_columns_led_on_to_many(fan, monkeypatch):
    # lists about as long as what a lane takes alone (second column) and as a row is allowed to lead to (first)
    hub = [np.full(fan, 3, np.uint32), np.arange(10, 10 + fan, dtype=np.uint32)]
    back = [np.arange(10, 10 + fan, dtype=np.uint32), np.full(fan, 3, np.uint32)]
    e = [np.concatenate([hub[0], back[0][:9], [2000]]).astype(np.uint32), np.concatenate([hub[1], back[1][:9], [2000]]).astype(np.uint32)]
    both(sides(("both",)), {"s": [np.array([3, 3], np.uint32), np.array([3, 11], np.uint32)], "a": e, "b": e}, "p", monkeypatch)


@pytest.mark.parametrize("n,burst", [(20, 0), (25, 0), (26, 0), (200, 0), (2000, 0), (26, 200), (60, 200)])
def test_columns_led_on_along_a_path(n, burst, monkeypatch):
    # one tuple an iteration: after some of them the loop goes on; at the end of the path burst^2 of them at once
    a = list(chain(n + 1))
    a = [np.concatenate([a[0], np.full(burst, n), [2000]]).astype(np.uint32), np.concatenate([a[1], np.arange(n + 1, n + 1 + burst), [2000]]).astype(np.uint32)]
    plan, rels = sides(("both",)), {"s": [np.array([0], np.uint32)] * 2, "a": a, "b": [a[0], a[1]]}
    both(plan, rels, "p", monkeypatch)
    for limit in (n - 1, n, n + 1):
        res = []
        for off in (False, True):
            if off:
                monkeypatch.setenv("XLB_NO_DELTA_LOOP", "1")
            else:
                monkeypatch.delenv("XLB_NO_DELTA_LOOP", raising=False)
            p = KernelProvider(device=0, max_iterations=limit)
            try:
                got, stats = run_program(p, plan, rels, ["p"])
                res.append((len(got["p"][0]), stats["iterations"]))
            except XlbError as e:
                res.append(e.status)
            p.close()
        assert res[0] == res[1]


def crowd(rels, rows):
    """Seeds given so often that bit rows are begun: one and a half for every row of the head, whatever they lead to."""
    n = -(-3 * (1 << (rows - 1).bit_length()) // (2 * len(rels["s"][0])))
    return {**rels, "s": [np.tile(c, n) for c in rels["s"]]}


# As above, begun as bit rows; (2000, 2000, 20000) more rows of a relation than are looked through for rows led to once
@pytest.mark.parametrize("kinds", [("both",), ("first",), ("both", "second"), ("first", "second", "both")], ids="-".join)
@pytest.mark.parametrize("hi,lo,rows", [(8191, 100, 9000), (8000, 130, 9000), (130, 8191, 3000), (1000, 1023, 1500), (1500, 1500, 2000), (8000, 8191, 9000), (2000, 2000, 20000)])
def test_columns_led_on_apart_by_bit_rows(hi, lo, rows, kinds, monkeypatch):
    rng = np.random.default_rng(hi * lo)
    pairs = lambda n, x, y: [rng.integers(0, x, n).astype(np.uint32), rng.integers(0, y, n).astype(np.uint32)]  # noqa: E731
    s = pairs(40, hi, lo)
    s[0][0], s[1][0] = hi - 1, lo - 1
    both(sides(kinds), crowd({"s": s, "a": pairs(rows, hi, hi), "b": pairs(rows, lo, lo)}, hi), "p", monkeypatch)


@pytest.mark.parametrize("fan", [16, 17, 1024, 1025])
def test_columns_led_on_to_many_by_bit_rows(fan, monkeypatch):
    hub = [np.full(fan, 3, np.uint32), np.arange(10, 10 + fan, dtype=np.uint32)]
    back = [np.arange(10, 10 + fan, dtype=np.uint32), np.full(fan, 3, np.uint32)]
    e = [np.concatenate([hub[0], back[0][:9], [2000]]).astype(np.uint32), np.concatenate([hub[1], back[1][:9], [2000]]).astype(np.uint32)]
    both(sides(("both",)), crowd({"s": [np.array([3, 3], np.uint32), np.array([3, 11], np.uint32)], "a": e, "b": e}, 2001), "p", monkeypatch)


# Handed to the loop after 32 small iterations, as `rows` rows or `rows` tuples of one row; at the end of the path each of them meets `burst` values at once
@pytest.mark.parametrize("n,rows,burst", [(30, 1, 0), (31, 1, 0), (32, 1, 0), (33, 1, 0), (32, 1, 200), (60, 1, 200), (300, 40, 0), (300, 1500, 0), (40, 1500, 60)])
@pytest.mark.parametrize("turned", [False, True])
def test_bit_rows_left_for_the_loop(n, rows, burst, turned, monkeypatch):
    path = list(chain(n + 1))
    path = [np.concatenate([path[0], np.full(burst, n), [2000]]).astype(np.uint32), np.concatenate([path[1], np.arange(n + 1, n + 1 + burst), [2000]]).astype(np.uint32)]
    still = [np.append(np.arange(rows), 2000).astype(np.uint32)] * 2
    s = [np.zeros(rows, np.uint32), np.arange(rows, dtype=np.uint32)]
    rels = {"s": s[::-1] if turned else s, "a": still if turned else path, "b": path if turned else still}
    rels = crowd(rels, 2001)
    both(sides(("both",)), rels, "p", monkeypatch)
    for limit, fits in ((n - 1, False), (n + 1 + (burst > 0), True)):
        p = KernelProvider(device=0, max_iterations=limit)
        try:
            run_program(p, sides(("both",)), rels, ["p"])
            assert fits
        except XlbError as e:
            assert not fits and e.status == A.ERR_ITER_LIMIT
        p.close()


def test_two_recursive_rules_and_wide_domain(monkeypatch):
    # p(X,Y) :- e(X,Y).  p(X,Z) :- p(X,Y), e(Y,Z).  p(X,Z) :- f(X,Y), p(Y,Z).  ids up to 2^15: 30 bits
    ids = {"e": 0, "f": 1, "p": 2}
    plan = ExecutionPlan([Scc(0, True, [
        CompiledRule("p", Scan(0), U2),
        CompiledRule("p", Project(Join(Scan(2), Scan(0), [1], [0]), [0, 3]), U2),
        CompiledRule("p", Project(Join(Scan(1), Scan(2), [1], [0]), [0, 3]), U2)])], ids)
    rng = np.random.default_rng(3)
    e = [rng.integers(0, 1 << 15, 3000).astype(np.uint32) for _ in range(2)]
    f = [rng.integers(0, 1 << 15, 3000).astype(np.uint32), e[0][rng.integers(0, 3000, 3000)]]
    both(plan, {"e": e, "f": f}, "p", monkeypatch)


def test_log_grows(monkeypatch):
    # 2000 nodes in one cycle-rich component: 3.9 M tuples, more than the first log holds under a small budget
    c = workloads.uniform_digraph()
    got, _, _ = both(programs.transitive_closure(), {"edge": list(c)}, "reach", monkeypatch, memory_budget_bytes=200 << 20)
    assert len(got[0]) > 1 << 21


def test_iteration_limit():
    for n, fits in [(6, True), (7, False)]:  # a chain of n nodes takes n - 1 iterations, the last of which finds nothing
        p = KernelProvider(device=0, max_iterations=5)
        if fits:
            got, stats = run_program(p, programs.transitive_closure(), {"edge": chain(n)}, ["reach"])
            assert len(got["reach"][0]) == n * (n - 1) // 2 and stats["iterations"] == 5
        else:
            with pytest.raises(XlbError) as e:
                run_program(p, programs.transitive_closure(), {"edge": chain(n)}, ["reach"])
            assert e.value.status == A.ERR_ITER_LIMIT
        p.close()


def test_one_column_head_after_the_frontier_loop(monkeypatch):
    # a path longer than the frontier loop follows: the rest of it runs in the delta loop
    got, it, _ = both(programs.reach_from_source(0), {"edge": chain(500)}, "r", monkeypatch)
    assert len(got[0]) == 499 and it == 499


@pytest.mark.parametrize("nodes,edges", [(2, 1), (31, 60), (33, 70), (500, 900), (4000, 4200)])
def test_two_recursive_atoms(nodes, edges, monkeypatch):
    c = workloads.uniform_digraph(nodes, edges, 5)
    both(programs.transitive_closure_nonlinear(), {"edge": list(c)}, "reach", monkeypatch)


@pytest.mark.parametrize("scale", [0.00001, 0.0001, 0.0004])
def test_points_to(scale, monkeypatch):
    rels = {k: list(v) for k, v in workloads.andersen_program(scale, 11).items()}
    # stored values no derived tuple ever has: beyond the head's domain
    rels["store"] = [np.append(rels["store"][0], 3).astype(np.uint32), np.append(rels["store"][1], 1 << 20).astype(np.uint32)]
    got, _, _ = both(programs.andersen(), rels, "pt", monkeypatch)
    want, _ = O.run_program(programs.andersen(), rels, ["pt"])
    for g, w in zip(got, want["pt"]):
        assert np.array_equal(g, w)


def by_rows(kinds):
    """p(X,Y) :- s(X,Y), then one rule per kind, each with the stored relation's columns either way round."""
    ids = {"s": 0, "e": 1, "f": 2, "p": 3}
    join = lambda l, r, a, b: Join(l, r, [a], [b])  # noqa: E731
    rules = {
        "copy": Project(join(Scan(1), Scan(3), 0, 0), [1, 3]),                          # p(X,Y) :- e(P,X), p(P,Y)
        "copy2": Project(join(Scan(2), Scan(3), 1, 0), [0, 3]),                         # p(X,Y) :- f(X,P), p(P,Y)
        "step": Project(join(Scan(3), Scan(3), 1, 0), [0, 3]),                          # p(P,Y) :- p(P,Q), p(Q,Y)
        "steps": Project(join(join(Scan(1), Scan(3), 0, 0), Scan(3), 3, 0), [1, 5]),    # p(X,Y) :- e(P,X), p(P,Q), p(Q,Y)
        "steps2": Project(join(join(Scan(2), Scan(3), 1, 0), Scan(3), 3, 0), [0, 5]),   # p(X,Y) :- f(X,P), p(P,Q), p(Q,Y)
        "across": Project(join(join(Scan(1), Scan(3), 0, 0), Scan(3), 1, 0), [3, 5]),   # p(Q,Y) :- e(P,W), p(P,Q), p(W,Y)
        "across2": Project(join(join(Scan(2), Scan(3), 1, 0), Scan(3), 0, 0), [3, 5]),  # p(Q,Y) :- f(W,P), p(P,Q), p(W,Y)
    }
    return ExecutionPlan([Scc(0, True, [CompiledRule("p", Scan(0), U2)] + [CompiledRule("p", rules[k], U2) for k in kinds])], ids)


# values of 6 bits (a row of two words) to 13, and of 14, which are too many
@pytest.mark.parametrize("kinds", [("steps",), ("across",), ("copy", "steps"), ("copy2", "steps2", "across2"), ("copy", "steps", "across", "step")], ids="-".join)
@pytest.mark.parametrize("top,rows", [(3, 4), (63, 60), (64, 90), (700, 500), (2047, 900), (8191, 2500), (8192, 2500)])
def test_rules_by_rows(kinds, top, rows, monkeypatch):
    rng = np.random.default_rng(top)
    pairs = lambda n: [rng.integers(0, top, n, endpoint=True).astype(np.uint32) for _ in range(2)]  # noqa: E731
    rels = {"s": pairs(rows), "e": pairs(rows // 3 + 1), "f": pairs(rows // 3 + 1)}
    rels["s"][0][0] = top
    got, it, _ = both(by_rows(kinds), rels, "p", monkeypatch)
    if top <= 700:
        want, _ = O.run_program(by_rows(kinds), rels, ["p"])
        for g, w in zip(got, want["p"]):
            assert np.array_equal(g, w)
    if it > 1:
        for limit, fits in ((it, True), (it - 1, False)):
            p = KernelProvider(device=0, max_iterations=limit)
            try:
                run_program(p, by_rows(kinds), rels, ["p"])
                assert fits
            except XlbError as e:
                assert not fits and e.status == A.ERR_ITER_LIMIT
            p.close()


# From 12 bits on (ACROSS alone: 11) rows are taken where the lists are long or many: `hubs` values with 60 of them each, one row
# for every fourth value (few: the loop), or for every one and the other way round
@pytest.mark.parametrize("kinds", [("across",), ("steps",), ("copy", "steps"), ("copy2", "steps2", "across2")], ids="-".join)
@pytest.mark.parametrize("top", [2047, 4095, 8191])
@pytest.mark.parametrize("hubs", [0, 2, 60])
def test_rules_by_rows_where_they_pay(kinds, top, hubs, monkeypatch):
    rng = np.random.default_rng(top + hubs)
    pairs = lambda n: [rng.integers(0, top, n, endpoint=True).astype(np.uint32) for _ in range(2)]  # noqa: E731
    lists = lambda way: [np.concatenate(c).astype(np.uint32) for c in zip(pairs(top // 4), [np.repeat(np.arange(hubs) * 30, 60), rng.integers(0, top, 60 * hubs)][::way])]  # noqa: E731
    rels = {"s": pairs(top // 3), "e": lists(1), "f": lists(-1)}
    rels["s"][0][0] = top
    got, it, cand = both(by_rows(kinds), rels, "p", monkeypatch)
    monkeypatch.delenv("XLB_NO_DELTA_LOOP")
    p = KernelProvider(device=0)
    p.profile_enable("list_squares")
    again, _ = run_program(p, by_rows(kinds), rels, ["p"])
    asked = "list_squares" in p.profile_read()
    p.close()
    if hubs < 60:  # (rows enough decide by their number)
        assert asked == (top > 2047 or kinds == ("across",))
    for a, b in zip(again["p"], got):
        assert np.array_equal(a, b)


def test_transposed_partner_and_composed_relation(monkeypatch):
    # p(X,Z) :- p(X,Y), p(Z,Y), g(X,Z)-free: the partner by its second column; q-shaped: p(Z,Y) :- g(Z,X), p(X,W), p(W,Y)
    ids = {"e": 0, "g": 1, "p": 2}
    plan = ExecutionPlan([Scc(0, True, [
        CompiledRule("p", Scan(0), U2),
        CompiledRule("p", Project(Join(Scan(2), Scan(2), [1], [1]), [0, 2]), U2),
        CompiledRule("p", Project(Join(Join(Scan(1), Scan(2), [1], [0]), Scan(2), [3], [0]), [0, 5]), U2)])], ids)
    rng = np.random.default_rng(9)
    e = [rng.integers(0, 300, 200).astype(np.uint32) for _ in range(2)]
    g = [rng.integers(0, 300, 150).astype(np.uint32) for _ in range(2)]
    got, _, _ = both(plan, {"e": e, "g": g}, "p", monkeypatch)
    want, _ = O.run_program(plan, {"e": e, "g": g}, ["p"])
    for a, w in zip(got, want["p"]):
        assert np.array_equal(a, w)


@pytest.mark.parametrize("bits", [17, 24, 28, 29, 32])
@pytest.mark.parametrize("values", [2, 500, 65536, 65537])
def test_thinly_spread_values(bits, values, monkeypatch):
    # ids of `bits` bits, `values` different ones: run on ranks (and on hash sets where there are too many)
    if values >= 1 << bits:
        return
    rng = np.random.default_rng(bits)
    ids = np.unique(np.concatenate([rng.integers(0, 1 << bits, 2 * values, dtype=np.uint64), [0, (1 << bits) - 1]]).astype(np.uint32))
    ids = np.sort(np.concatenate([ids[[0, -1]], rng.permutation(ids[1:-1])[: values - 2]]))
    assert len(ids) == values
    n = min(values, 3000)
    some = rng.permutation(ids)[:n]
    u, v = rng.integers(0, n, n), rng.integers(0, n, n)
    # the rest of the ids in pairs, so that every one of them is there
    edge = [np.concatenate([some[u], ids[:-1:2]]), np.concatenate([some[v], ids[1::2]])]
    if values % 2:
        edge = [np.append(edge[0], ids[-1]), np.append(edge[1], ids[0])]
    both(programs.transitive_closure(), {"edge": edge}, "reach", monkeypatch)


@pytest.mark.parametrize("bits", [14, 15, 16])
@pytest.mark.parametrize("values", [64, 4096, 8191, 8193])
def test_thinly_spread_values_of_16_bits(bits, values, monkeypatch):
    test_thinly_spread_values(bits, values, monkeypatch)


def _rows_graph(kind):
    rng = np.random.default_rng(3)
    if kind.startswith("values"):  # bits of the second column: a word, two words, 16 and 17 bits
        n = int(kind[6:])
        m = min(2 * n, 3000)
        return [rng.integers(0, n, m, dtype=np.uint32), np.concatenate([rng.integers(0, n, m - 1, dtype=np.uint32), [n - 1]]).astype(np.uint32)]
    if kind.startswith("front"):  # chains that run into a node with so many successors, which come together again
        k = int(kind[5:])
        leaves = np.arange(400, 400 + k, dtype=np.uint32)
        a = [np.arange(50), np.full(k, 50), leaves, np.arange(100, 399)]
        b = [np.arange(1, 51), leaves, np.full(k, 60), np.arange(101, 400)]
        return [np.concatenate(x).astype(np.uint32) for x in (a, b)]
    if kind == "all_wide":  # every row outgrows its queue
        leaves = np.arange(4000, 20600, dtype=np.uint32)
        src = np.arange(1500, dtype=np.uint32)
        return [np.concatenate([src, np.full(16600, 3500)]).astype(np.uint32), np.concatenate([np.full(1500, 3500), leaves]).astype(np.uint32)]
    n = 300  # every node next to every other: long rows
    return [np.repeat(np.arange(n, dtype=np.uint32), n), np.tile(np.arange(n, dtype=np.uint32), n)]


@pytest.mark.parametrize("kind", ["values31", "values32", "values33", "values65536", "values65537", "front16383", "front16384", "front16385", "all_wide", "dense"])
def test_rows_apart(kind, monkeypatch):
    edge = _rows_graph(kind)
    got, _, _ = both(programs.transitive_closure(), {"edge": edge}, "reach", monkeypatch)
    if kind not in ("dense", "all_wide"):
        want, _ = O.run_program(programs.transitive_closure(), {"edge": edge}, ["reach"])
        for g, w in zip(got, want["reach"]):
            assert np.array_equal(g, w)


@pytest.mark.parametrize("nodes", [40, 1500])
def test_rows_apart_two_rules(nodes, monkeypatch):
    # p(X,Z) :- p(X,Y), a(Y,Z).  p(X,Z) :- p(X,Y), b(Y,Z).
    ids = {"a": 0, "b": 1, "p": 2}
    rules = [CompiledRule("p", Scan(0), U2)] + [CompiledRule("p", Project(Join(Scan(2), Scan(r), [1], [0]), [0, 3]), U2) for r in (0, 1)]
    rng = np.random.default_rng(nodes)
    pairs = lambda m: [rng.integers(0, nodes, m, dtype=np.uint32), rng.integers(0, nodes, m, dtype=np.uint32)]  # noqa: E731
    both(ExecutionPlan([Scc(0, True, rules)], ids), {"a": pairs(nodes), "b": pairs(nodes // 2)}, "p", monkeypatch)


def test_log_grows_left_linear(monkeypatch):
    got, _, _ = both(programs.transitive_closure_left_linear(), {"edge": list(workloads.uniform_digraph())}, "reach", monkeypatch, memory_budget_bytes=200 << 20)
    assert len(got[0]) > 1 << 21
