"""Operations whose result fits a memory budget that their quickest route does not: they take the other one."""
import numpy as np
import pytest

from oracle import oracle as O
from xlog_b200 import _abi as A
from xlog_b200 import programs, workloads
from xlog_b200.executor import run_program
from xlog_b200.provider import KernelProvider

pytestmark = pytest.mark.gpu

N = 8192  # rows, the most one block takes
REST = 16 << 10  # bytes a column may hold beyond its rows


def with_spare(cols, spare):
    """A provider with these relations and `spare` more bytes."""
    p = KernelProvider(device=0, memory_budget_bytes=sum(c.nbytes for r in cols for c in r) + spare)
    return p, [p.create_buffer_from_slices(r) for r in cols]


@pytest.mark.parametrize("kind", [A.JOIN_SEMI, A.JOIN_ANTI, A.JOIN_INNER])
def test_small_joins(kind):
    key = np.arange(N, dtype=np.uint64)
    left = [key] + [key + np.uint64(k) for k in range(1, 6)]  # 393 KB
    right = [np.append(key[:3], key[5:] if kind == A.JOIN_ANTI else key[:0])[:4096]]
    left = [c[:4096] for c in left] if kind == A.JOIN_ANTI else left
    want = [c[np.isin(left[0], right[0]) != (kind == A.JOIN_ANTI)] for c in left] + ([right[0]] if kind == A.JOIN_INNER else [])
    assert len(want[0]) < 10
    # (the inner join's row lists: 8 + 4 bytes a probe row)
    p, (lb, rb) = with_spare([left, right], 160 << 10)
    for g, w in zip(p.download(p.hash_join_v2(lb, rb, [0], [0], kind)), want):
        assert np.array_equal(g, w)
    p.close()


def test_small_groups():
    key = np.arange(N, dtype=np.uint32) % np.uint32(3)
    v = np.arange(N, dtype=np.uint64)
    p, (b,) = with_spare([[key, v]], 32 << 10)
    got = p.download(p.groupby_multi_agg(b, [0], [(1, op) for op in (A.AGG_SUM, A.AGG_MIN, A.AGG_MAX, A.AGG_COUNT, A.AGG_SUM)]))  # 360 KB for all rows
    groups = [v[key == k] for k in range(3)]
    for g, f in zip(got[1:], (np.sum, np.min, np.max, len, np.sum)):
        assert g.tolist() == [f(x) for x in groups]
    p.close()


def test_large_sets_come_back():
    # the first column as runs needs a few KB on the device: without them all columns are copied
    n, budget = 2_200_000, 256 << 20
    cols = [np.repeat(np.arange(n // 1000, dtype=np.uint32), 1000), np.arange(n, dtype=np.uint32)]
    p = KernelProvider(device=0, memory_budget_bytes=budget)
    rel = p.dedup(p.create_buffer_from_slices(cols))
    assert rel.is_canonical()
    for full in (False, True):
        if full:
            filler = p.create_buffer_from_slices([np.zeros((budget - p.memory_stats()[0] - 256) // 8, dtype=np.uint64)])
            assert budget - p.memory_stats()[0] < 512
        for g, c in zip(p.download(rel), cols):
            assert np.array_equal(g, c)
    del filler
    p.close()


@pytest.mark.parametrize("rows", [0, 1, 130, 4096])
def test_small_results_keep_what_they_need(rows):
    probe = [np.arange(N, dtype=np.uint32), np.arange(N, dtype=np.uint64), np.zeros(N, dtype=np.float32)]
    build = [np.arange(N - rows, 2 * N - rows, dtype=np.uint32)[:4096], np.arange(4096, dtype=np.uint32)]
    p = KernelProvider(device=0)
    lb, rb = p.create_buffer_from_slices(probe), p.create_buffer_from_slices(build)
    for kind, width in ((A.JOIN_SEMI, 16), (A.JOIN_ANTI, 16), (A.JOIN_INNER, 24)):
        before = p.memory_stats()[0]
        out = p.hash_join_v2(lb, rb, [0], [0], kind)
        assert out.num_rows() == (N - rows if kind == A.JOIN_ANTI else rows)
        assert width * out.num_rows() <= p.memory_stats()[0] - before <= width * out.num_rows() + 5 * REST
        again = p.hash_join_v2(lb, rb, [0], [0], kind)  # (in what the first did not keep)
        for g, w in zip(p.download(out), p.download(again)):
            assert np.array_equal(g, w)
        del out, again
    before = p.memory_stats()[0]
    g = p.create_buffer_from_slices([np.arange(N, dtype=np.uint32) % np.uint32(max(rows, 1)), probe[1]])
    own = p.memory_stats()[0] - before
    out = p.groupby_multi_agg(g, [0], [(1, A.AGG_SUM)])
    assert out.num_rows() == max(rows, 1) and 0 <= p.memory_stats()[0] - before - own - 12 * out.num_rows() <= 2 * REST
    p.close()


def test_rules_by_rows_without_a_log():
    # values of 9 bits: a bitmap of 32 KB, where a log of all there could be takes 2 MB
    rels = {k: list(v) for k, v in workloads.andersen_program(0.0001, 5).items()}
    want, _ = O.run_program(programs.andersen(), rels, ["pt"])
    assert max(int(c.max()) for c in want["pt"]) < 512
    launches = []
    for budget in (1 << 30, 1536 << 10):
        p = KernelProvider(device=0, memory_budget_bytes=budget)
        got, stats = run_program(p, programs.andersen(), rels, ["pt"])
        launches.append(stats["kernel_launches"])
        assert p.memory_stats()[1] < 1536 << 10
        p.close()
        for g, w in zip(got["pt"], want["pt"]):
            assert np.array_equal(g, w)
    assert launches[0] == launches[1] < 40  # (iteration by iteration several hundred)
