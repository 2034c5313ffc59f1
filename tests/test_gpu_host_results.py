"""Results fetched into staged and into page-locked memory: sizes around the limit of the staging
buffer, columns of every width, results that outlive their context, blocks used again."""
import gc
import glob
import os
import threading

import numpy as np
import pytest

from xlog_b200 import _abi as A
from xlog_b200 import programs
from xlog_b200.executor import run_program
from xlog_b200.plan import CompiledRule, ExecutionPlan, Scan, Scc
from xlog_b200.provider import KernelProvider

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 3, 13107, 13108, 32767, 32768, 32769, 600001])
def test_columns_come_back_as_they_went_in(n):
    rng = np.random.default_rng(n)
    cols = [rng.integers(0, 1 << 32, n, dtype=np.uint32), rng.integers(0, 1 << 63, n, dtype=np.uint64),
            rng.integers(0, 2, n).astype(np.bool_), rng.standard_normal(n).astype(np.float32)]
    p = KernelProvider(device=0)
    got = p.download(p.create_buffer_from_slices(cols))
    assert [g.dtype for g in got] == [np.uint32, np.uint64, np.uint8, np.float32]
    for g, c in zip(got, cols):
        assert np.array_equal(g, c)
        assert g.flags.writeable
    for k in (1, 2):  # packed relations
        d = p.dedup(p.create_buffer_from_slices(cols[:1] * k))
        u = np.unique(cols[0])
        for g in p.download(d):
            assert np.array_equal(g, u)
    p.close()


def test_results_are_independent_and_outlive_the_context():
    p = KernelProvider(device=0)
    held, want = [], []
    for k in range(6):
        c = np.arange(k, k + 300000, dtype=np.uint64)
        held.append(p.download(p.create_buffer_from_slices([c]))[0])
        want.append(c)
        if k == 3:
            del held[1], want[1]
            gc.collect()
    p.close()
    for h, w in zip(held, want):
        assert np.array_equal(h, w)


def expect(p, rel, cols):
    for g, c in zip(p.download(rel), cols):
        assert np.array_equal(g, c)


CORES = min([len(os.sched_getaffinity(0))] + [int(q[0]) // int(q[1]) for q in [open(f).read().split() for f in glob.glob("/sys/fs/cgroup/cpu.max")] if q[0] != "max"])


def went_as_runs(p, fetch):
    """Whether `fetch` brought a first column as runs: two kernels, of which plain copies have none."""
    p.profile_enable("to_host")
    fetch()
    launches = p.profile_read().get("to_host", {"launches": 0})["launches"]
    p.profile_enable(None)
    assert launches in (0, 2)
    return launches == 2


def rows_from(starts, n):
    starts = np.unique(starts)
    return np.diff(np.append(starts, n))


# First columns of sets, of 6 MB and more and of few values, go as runs: tiles are 4096 rows, a warp's 512, what a
# thread fills 65536 (4 bytes) or 32768 (8 bytes) rows, and the staging holds 32766 or 16383 runs.
@pytest.mark.parametrize("runs", ["one", "last", "edges", "even", "most", "many"])
@pytest.mark.parametrize("n", [(3 << 19) - 1, 3 << 19, (3 << 19) + 4097, (1 << 21) - 1, 1 << 21, 2222222])
def test_first_columns_of_long_runs(runs, n):
    starts = {"one": [0], "last": [0, n - 1], "edges": [x + d for x in (0, 512, 4096, 32768, 65536, 131072, n - 4096) for d in (-1, 0, 1) if 0 <= x + d < n],
              "even": np.arange(0, n, 1000), "most": np.linspace(0, n - 1, 1 << 14).astype(np.int64), "many": np.arange(0, n, 9)}[runs]
    first = np.repeat(np.arange(len(np.unique(starts)), dtype=np.uint32), rows_from(starts, n))
    cols = [first, np.arange(n, dtype=np.uint32)]
    p = KernelProvider(device=0)
    rel = p.dedup(p.create_buffer_from_slices([c[::-1] for c in cols]))
    assert rel.is_canonical()
    assert went_as_runs(p, lambda: expect(p, rel, cols)) == (CORES >= 4 and n >= 3 << 19 and 400 << len(bin(int(first[-1]))) - 2 <= 4 * n)
    assert not went_as_runs(p, lambda: expect(p, p.create_buffer_from_slices(cols), cols))  # (not known to be in order)
    p.close()


@pytest.mark.parametrize("dtype", [np.uint64, np.int64, np.float32, np.int32])
def test_first_columns_of_wide_results(dtype):
    # of a plan over typed columns: a set of decoded ranks
    code = {np.uint64: A.U64, np.int64: A.I64, np.float32: A.F32, np.int32: A.I32}[dtype]
    rng = np.random.default_rng(5)
    per = rng.integers(1, 4000, 1000)
    per[::7] = 1
    values = np.unique(rng.integers(-(1 << 30), 1 << 30, 5000)).astype(dtype)[:4000]
    if dtype == np.float32:
        values = np.sort(values)
    values = np.unique(values) if dtype != np.uint64 else np.unique(np.abs(values.astype(np.int64)).astype(np.uint64))
    n = len(values)
    first = np.repeat(values[:1000], np.minimum(per, n))
    second = np.concatenate([values[: min(k, n)] for k in per])
    plan = ExecutionPlan([Scc(0, False, [CompiledRule("h", Scan(0), (code, code))])], {"s": 0, "h": 1})
    order = rng.permutation(len(first))
    p = KernelProvider(device=0)
    res = []
    assert went_as_runs(p, lambda: res.append(run_program(p, plan, {"s": [first[order], second[order]]}, ["h"])[0])) == (CORES >= 4)
    assert len(first) * first.itemsize >= 6 << 20
    got = res[0]
    for g, w in zip(got["h"], (first, second)):
        assert np.array_equal(g, w)
    p.close()


# 4-byte runs are worth their while from 100 rows on, 8-byte ones from 50
@pytest.mark.parametrize("dtype,runs,rows", [(np.uint32, 16384, 99), (np.uint32, 16384, 100), (np.uint64, 16000, 50), (np.uint64, 8000, 99)])
def test_short_runs(dtype, runs, rows):
    ids = np.arange(runs, dtype=dtype) * dtype(1 if dtype == np.uint32 else 1 << 33)
    first, second = np.repeat(ids, rows), np.tile(ids[:rows], runs)
    code = A.U32 if dtype == np.uint32 else A.U64
    plan = ExecutionPlan([Scc(0, False, [CompiledRule("h", Scan(0), (code, code))])], {"s": 0, "h": 1})
    p = KernelProvider(device=0)
    res = []
    assert went_as_runs(p, lambda: res.append(run_program(p, plan, {"s": [first, second]}, ["h"])[0])) == (CORES >= 4 and rows * first.itemsize >= 400)
    for g, w in zip(res[0]["h"], (first, second)):
        assert np.array_equal(g, w)
    p.close()


def cycle_of_blocks(ids, blocks):
    """Every value of a block leads to every one of the next: the closure is all pairs."""
    b = np.array_split(ids, blocks)
    return [np.concatenate([np.repeat(x, len(y)) for x, y in zip(b, b[1:] + b[:1])]), np.concatenate([np.tile(y, len(x)) for x, y in zip(b, b[1:] + b[:1])])]


def test_first_columns_of_decoded_ranks():
    # ids of 30 bits, which a plan runs over as ranks: the result's first values are as many as there are ranks
    rng = np.random.default_rng(3)
    ids = np.sort(rng.choice(1 << 30, 1400, replace=False)).astype(np.uint32)
    p = KernelProvider(device=0)
    res = []
    assert went_as_runs(p, lambda: res.append(run_program(p, programs.transitive_closure(), {"edge": cycle_of_blocks(ids, 10)}, ["reach"])[0])) == (CORES >= 4)
    got = res[0]
    assert 4 * len(got["reach"][0]) >= 6 << 20
    assert np.array_equal(got["reach"][0], np.repeat(ids, len(ids))) and np.array_equal(got["reach"][1], np.tile(ids, len(ids)))
    p.close()


def test_two_contexts_fetch_at_once():
    n, wrong = 2_200_000, []

    def work(seed):
        try:
            p = KernelProvider(device=0)
            cols = [np.repeat(np.arange(n // 1000, dtype=np.uint32) * np.uint32(3 + seed), 1000), np.arange(n, dtype=np.uint32) * np.uint32(7)]
            rel = p.dedup(p.create_buffer_from_slices([c[::-1] for c in cols]))
            assert rel.is_canonical()
            cols[1] = cols[1].reshape(-1, 1000)
            cols[1] = np.sort(cols[1], axis=1).reshape(-1)
            for _ in range(25):
                expect(p, rel, cols)
            p.close()
        except BaseException as e:  # noqa: BLE001
            wrong.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("offset", [None, 0, 4, 36])
def test_long_runs_into_memory_of_the_callers(offset):
    # The C interface takes any memory: what is not page-locked is copied as before, what is need not begin at a
    # cache line.
    import ctypes as C

    total = 2200000
    first, second = np.repeat(np.arange(total // 1000, dtype=np.uint32), 1000), np.arange(total, dtype=np.uint32)
    p = KernelProvider(device=0)
    buf = p.dedup(p.create_buffer_from_slices([first, second]))
    assert buf.is_canonical()
    for m in (total, total - 49999):  # all rows, and as many as the caller has room for
        if offset is None:
            out = [np.zeros(m, dtype=np.uint32) for _ in range(2)]
        else:
            block = C.c_void_p()
            p._check(p._lib.xlb_host_alloc(C.c_uint64(8 * m + 256), C.byref(block)))
            all_of_it = np.ctypeslib.as_array((C.c_uint32 * (2 * m + 64)).from_address(block.value))
            all_of_it[:] = 0xABABABAB
            at = offset // 4
            out = [all_of_it[at:at + m], all_of_it[at + m + 1:at + 2 * m + 1]]
        rows = C.c_uint64()
        fetch = lambda: p._check(p._lib.xlb_rel_to_host(p._ctx, buf._h, (C.c_void_p * 2)(*[o.ctypes.data for o in out]), m, C.byref(rows)))  # noqa: E731, B023
        assert went_as_runs(p, fetch) == (offset is not None and CORES >= 4)
        assert rows.value == total and np.array_equal(out[0], first[:m]) and np.array_equal(out[1], second[:m])
        if offset is not None:
            assert np.all(all_of_it[:at] == 0xABABABAB) and all_of_it[at + m] == 0xABABABAB and np.all(all_of_it[at + 2 * m + 1:] == 0xABABABAB)
            p._lib.xlb_host_free(block)
    p.close()
