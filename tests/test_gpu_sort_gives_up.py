"""A sort whose bounded wait runs out leaves incomplete lists and row numbers.  Whatever is built on a
sort reports the failure, stays inside its buffers, and the context goes on working."""
import numpy as np
import pytest

from xlog_b200 import _abi as A
from xlog_b200.lib import XlbError
from xlog_b200.provider import KernelProvider

pytestmark = pytest.mark.gpu
N = 100_003


@pytest.fixture()
def p():
    prov = KernelProvider(device=0)
    yield prov
    prov.close()


def wide(rng, n):
    return rng.integers(0, 1 << 64, n, dtype=np.uint64)


def sort_two_words(p, b):
    return p.sort(b["three"], [0, 1])


def dedup_rows(p, b):
    return p.dedup(b["three"])


def dedup_by_key(p, b):
    return p.dedup(b["three"], [0])


def difference(p, b):
    return p.diff_gpu(b["one"], b["other"])


def union(p, b):
    return p.union_gpu(b["one"], b["other"])


def groups(p, b):
    return p.groupby_multi_agg(b["three"], [0], [(1, A.AGG_SUM), (2, A.AGG_MAX)])


def join_with_hub(p, b):
    return p.hash_join_v2(b["one"], b["hub"], [0], [0])


@pytest.mark.parametrize("op", [sort_two_words, dedup_rows, dedup_by_key, difference, union, groups, join_with_hub])
def test_failure_is_reported_and_contained(p, op):
    rng = np.random.default_rng(5)
    key = wide(rng, N // 2)[rng.integers(0, N // 2, N)]
    cols = {"three": [key, wide(rng, N), rng.integers(0, 1 << 32, N, dtype=np.uint64).astype(np.uint32)], "one": [key], "other": [wide(rng, N)],
            "hub": [np.concatenate([key[: N - 70], np.full(70, key[0])]), np.arange(N, dtype=np.uint32)]}
    b = {k: p.create_buffer_from_slices(v) for k, v in cols.items()}
    want = p.download(op(p, b))
    guard = [p.create_buffer_from_slices([np.full(5000, k, dtype=np.uint64)]) for k in range(40)]  # buffers all around
    p._check(p._lib.xlb_test_set_lookback(p._ctx, 4000, 1))
    for _ in range(2):
        with pytest.raises(XlbError) as e:
            op(p, b)
        assert e.value.status == A.ERR_TIMEOUT
    p._check(p._lib.xlb_test_set_lookback(p._ctx, 0, 0))
    for k, g in enumerate(guard):
        assert np.all(p.download(g)[0] == k)
    for k, v in cols.items():
        for g, w in zip(p.download(b[k]), v):
            assert np.array_equal(g, w)
    for g, w in zip(p.download(op(p, b)), want):
        assert np.array_equal(g, w)
