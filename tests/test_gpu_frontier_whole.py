"""Frontier fixpoints in one launch against the oracle: row counts around the limits of the three
kernels, paths longer than the latter follows, values at the edge of the domains,
no seed at all, the iteration limit, both join columns."""
import numpy as np
import pytest

from oracle import oracle as O
from xlog_b200 import _abi as A
from xlog_b200 import programs
from xlog_b200.executor import run_program
from xlog_b200.lib import XlbError
from xlog_b200.plan import CompiledRule, ExecutionPlan, Filter, Join, Project, Scan, Scc
from xlog_b200.provider import KernelProvider

pytestmark = pytest.mark.gpu
LARGE = (1 << 21) + 101  # rows: the kernel that keeps lists of the rows still of use


def check(plan, edge, out="r"):
    p = KernelProvider(device=0)
    got, stats = run_program(p, plan, {"edge": edge}, [out])
    p.close()
    want, ex = O.run_program(plan, {"edge": edge}, [out])
    assert np.array_equal(got[out][0], want[out][0])
    assert stats["iterations"] == ex.iterations and stats["candidate_tuples"] == ex.candidates
    return stats


@pytest.mark.parametrize("n", [1, 2, 1023, 32767, 32768, 32769, 100003, (1 << 21), (1 << 21) + 1])
def test_row_counts(n):
    rng = np.random.default_rng(n)
    nodes = max(n // 3, 2)
    check(programs.reach_from_source(0), [rng.integers(0, nodes, n).astype(np.uint32), rng.integers(0, nodes, n).astype(np.uint32)])


@pytest.mark.parametrize("n,rows", [(2000, 2000), (47, 40000), (49, 40000), (400, 40000), (47, LARGE), (60, LARGE)])
def test_paths(n, rows):
    # a path of n nodes, and unrelated rows to make up the number
    edge = [np.arange(n - 1, dtype=np.uint32), np.arange(1, n, dtype=np.uint32)]
    fill = np.arange(rows - n + 1, dtype=np.uint32) % (1 << 19) + n
    assert check(programs.reach_from_source(0), [np.append(edge[0], fill), np.append(edge[1], fill)])["iterations"] == n - 1


@pytest.mark.parametrize("top", [(1 << 18) - 1, (1 << 19) - 1, 1 << 19, (1 << 20) - 1, 1 << 20, (1 << 32) - 1])
@pytest.mark.parametrize("rows", [100, 40000, LARGE])
def test_large_values(top, rows):
    rng = np.random.default_rng(rows)
    a, b = rng.integers(0, 500, rows).astype(np.uint32), rng.integers(0, 500, rows).astype(np.uint32)
    a[:3], b[:3] = [0, 17, top], [17, top, 3]
    check(programs.reach_from_source(0), [a, b])


def test_no_seed_other_column_and_two_seeds():
    rng = np.random.default_rng(1)
    edge = [rng.integers(1, 3000, 9000).astype(np.uint32), rng.integers(1, 3000, 9000).astype(np.uint32)]
    check(programs.reach_from_source(0), edge)
    # backwards from 5 and forwards from 9's row itself: r(X) :- edge(X,5). r(X) :- edge(X,9). r(X) :- r(Y), edge(X,Y).
    ids = {"edge": 0, "r": 1}
    u = (A.U32,)
    plan = ExecutionPlan([Scc(0, True, [
        CompiledRule("r", Project(Filter(Scan(0), A.EQ, 1, 5, True), [0]), u),
        CompiledRule("r", Project(Filter(Scan(0), A.EQ, 0, 9, True), [0]), u),
        CompiledRule("r", Project(Join(Scan(1), Scan(0), [0], [1]), [1]), u)])], ids)
    for n in (9000, 40000, LARGE):
        check(plan, [rng.integers(1, 3000, n).astype(np.uint32), rng.integers(1, 3000, n).astype(np.uint32)])


@pytest.mark.parametrize("rows", [10, 40000, LARGE])
def test_iteration_limit(rows):
    n = 10
    fill = np.arange(rows - n + 1, dtype=np.uint32) % (1 << 19) + n
    edge = [np.append(np.arange(n - 1, dtype=np.uint32), fill), np.append(np.arange(1, n, dtype=np.uint32), fill)]
    for limit, ok in ((n - 1, True), (n - 2, False)):
        p = KernelProvider(device=0, max_iterations=limit)
        if ok:
            assert len(run_program(p, programs.reach_from_source(0), {"edge": edge}, ["r"])[0]["r"][0]) == n - 1
        else:
            with pytest.raises(XlbError) as e:
                run_program(p, programs.reach_from_source(0), {"edge": edge}, ["r"])
            assert e.value.status == A.ERR_ITER_LIMIT
        p.close()
