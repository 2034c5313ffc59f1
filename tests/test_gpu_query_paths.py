"""Joins and aggregations at the sizes where their routes change hands: keys with one, a few and very
many build rows, domains around the table limits, hub groups, row counts around tiles; and sorts
around the sizes one block takes."""
import numpy as np
import pytest

from xlog_b200 import _abi as A
from xlog_b200.provider import KernelProvider

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def p():
    prov = KernelProvider(device=0)
    yield prov
    prov.close()


def inner(lk, rk):
    """(left row, right row) pairs by left row, then right row."""
    order = np.argsort(rk, kind="stable")
    s = rk[order]
    lo, hi = np.searchsorted(s, lk, "left"), np.searchsorted(s, lk, "right")
    n = hi - lo
    left = np.repeat(np.arange(len(lk)), n)
    first = np.cumsum(n) - n
    right = order[np.repeat(lo, n) + np.arange(len(left)) - np.repeat(first, n)]
    return left, right


@pytest.mark.parametrize("nl,nr,keys", [(1, 1, 1), (1, 64, 1), (3, 65, 1), (2047, 2049, 700), (2048, 513, 40), (2049, 100000, 60000), (70000, 3000, 1 << 31), (5000, 8192, 100)])
@pytest.mark.parametrize("dtype", [np.uint32, np.uint64, "pair"])
def test_joins(p, nl, nr, keys, dtype):
    rng = np.random.default_rng(nl + nr)
    draw = lambda n: rng.integers(0, keys, n)  # noqa: E731
    if dtype == "pair":
        lkc, rkc = [draw(nl).astype(np.uint32), (draw(nl) % 2).astype(np.uint32)], [draw(nr).astype(np.uint32), (draw(nr) % 2).astype(np.uint32)]
        lk, rk = [(c[0].astype(np.uint64) << np.uint64(32)) | c[1] for c in (lkc, rkc)]
    else:
        scale = np.uint64(0x9E3779B97F4A7C15 if dtype is np.uint64 else 1)
        with np.errstate(over="ignore"):
            lkc, rkc = [(draw(nl).astype(np.uint64) * scale).astype(dtype)], [(draw(nr).astype(np.uint64) * scale).astype(dtype)]
        lk, rk = lkc[0], rkc[0]
    lv, rv = rng.integers(0, 1 << 60, nl, dtype=np.uint64), rng.integers(0, 255, nr).astype(np.float32)
    L, R = p.create_buffer_from_slices(lkc + [lv]), p.create_buffer_from_slices([rv] + rkc)
    nk = len(lkc)
    got = p.download(p.hash_join_v2(L, R, list(range(nk)), list(range(1, nk + 1))))
    left, right = inner(lk, rk)
    want = [c[left] for c in lkc + [lv]] + [c[right] for c in [rv] + rkc]
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
    has = np.isin(lk, rk)
    for kind, keep in ((A.JOIN_SEMI, has), (A.JOIN_ANTI, ~has)):
        for g, w in zip(p.download(p.hash_join_v2(L, R, list(range(nk)), list(range(1, nk + 1)), kind)), lkc + [lv]):
            assert np.array_equal(g, w[keep])


@pytest.mark.parametrize("n,groups,hub", [(1, 1, 0), (2048, 65536, 0), (2049, 65537, 0), (16385, 65537, 0), (100001, 30000, 50000), (200000, 10, 0), (200000, 3, 150000), (70001, 1 << 31, 0)])
@pytest.mark.parametrize("nk", [1, 2])
def test_groupby(p, n, groups, hub, nk):
    rng = np.random.default_rng(n)
    g = rng.integers(0, groups, n)
    g[:hub] = groups - 1
    g = rng.permutation(g).astype(np.uint32)
    cols = [g, rng.integers(0, 3, n).astype(np.uint32)][:nk] + [rng.integers(0, 1 << 63, n, dtype=np.uint64), rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)]
    b = p.create_buffer_from_slices(cols)
    got = p.download(p.groupby_multi_agg(b, list(range(nk)), [(nk, A.AGG_SUM), (nk + 1, A.AGG_MIN), (nk, A.AGG_MAX), (0, A.AGG_COUNT), (nk + 1, A.AGG_SUM)]))
    key = cols[0].astype(np.uint64) if nk == 1 else (cols[0].astype(np.uint64) << np.uint64(32)) | cols[1]
    order = np.argsort(key, kind="stable")
    u, at = np.unique(key[order], return_index=True)
    v, w = cols[nk][order], cols[nk + 1][order]
    want = ([u.astype(np.uint32)] if nk == 1 else [(u >> np.uint64(32)).astype(np.uint32), u.astype(np.uint32)]) + [
        np.add.reduceat(v, at), np.minimum.reduceat(w, at), np.maximum.reduceat(v, at), np.diff(np.append(at, n)).astype(np.uint64), np.add.reduceat(w.astype(np.uint64), at)]
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and np.array_equal(a, b)


@pytest.mark.parametrize("n", [2, 31, 1023, 1024, 1025, 2048, 2049, 4097, 8191, 8192, 8193])
def test_small_sorts(p, n):
    rng = np.random.default_rng(n)
    for cols in ([rng.integers(0, 1 << 63, n, dtype=np.uint64)], [rng.integers(0, 5, n).astype(np.uint32), rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)],
                 [np.full(n, (1 << 64) - 1, np.uint64)]):
        b = p.create_buffer_from_slices(cols + [np.arange(n, dtype=np.uint32)])
        keys = list(range(len(cols)))
        order = np.lexsort([c for c in reversed(cols)])
        for g, c in zip(p.download(p.sort(b, keys)), cols + [np.arange(n, dtype=np.uint32)]):
            assert np.array_equal(g, c[order])


def joined(left, right, lk, rk):
    """Matches of the rows of `left`, in their order and each in the order of `right`."""
    rows = {}
    for i, k in enumerate(zip(*(right[c].tolist() for c in rk))):
        rows.setdefault(k, []).append(i)
    pairs = [(i, j) for i, k in enumerate(zip(*(left[c].tolist() for c in lk))) for j in rows.get(k, [])]
    l, r = (np.array(x, dtype=np.int64) for x in (zip(*pairs) if pairs else ((), ())))
    return [c[l] for c in left] + [c[r] for c in right]


# groups of up to 64 rows; up to four outputs a build row go out from the chains, more from lists.  Keys of 0 and of all ones.
@pytest.mark.parametrize("kind", ["u32", "u64", "two"])
@pytest.mark.parametrize("sizes", [[1], [1, 2, 3, 4], [4, 5, 6], [1, 31, 32, 33, 63, 64], [64]], ids=str)
@pytest.mark.parametrize("probes", [1, 31, 900, 5000])
def test_joins_from_chains_and_from_lists(kind, sizes, probes):
    rng = np.random.default_rng(len(sizes) * probes)
    sizes = np.resize(sizes, 90)
    top = (1 << 64) - 1 if kind == "u64" else (1 << 32) - 1
    dtype = np.uint64 if kind == "u64" else np.uint32
    names = np.concatenate([np.array([0, top], dtype=dtype), (rng.choice(1 << 31, 98, replace=False) + 1).astype(dtype)])
    key = rng.permutation(np.repeat(names[:90], sizes))  # (ten names have no rows)
    ask = names[rng.integers(0, 100, probes)]
    left, right = [ask, np.arange(probes, dtype=np.uint32)], [np.arange(len(key), dtype=np.uint64), key]
    lk, rk = [0], [1]
    if kind == "two":
        left, right = left + [ask % dtype(3)], right + [key % dtype(3)]
        lk, rk = [0, 2], [1, 2]
    p = KernelProvider(device=0)
    lb, rb = p.create_buffer_from_slices(left), p.create_buffer_from_slices(right)
    for g, w in zip(p.download(p.hash_join_v2(lb, rb, lk, rk)), joined(left, right, lk, rk)):
        assert np.array_equal(g, w)
    there = np.isin(ask, key)
    for how, keep in ((A.JOIN_SEMI, there), (A.JOIN_ANTI, ~there)):
        for g, w in zip(p.download(p.hash_join_v2(lb, rb, lk, rk, how)), left):
            assert np.array_equal(g, w[keep])
    p.close()


# What one block takes: 4096 build rows, 8192 probe rows, four outputs a probe row and 1024 (2 keys: half of all pairs)
@pytest.mark.parametrize("nl,nr,keys", [(8191, 4095, 3000), (8192, 4096, 3000), (8193, 4096, 3000), (8192, 4097, 3000), (1, 4096, 4096), (8192, 1, 2), (100, 12, 2), (100, 28, 2),
                                        (1025, 64, 1), (1024, 65, 1)])
def test_joins_of_one_block(p, nl, nr, keys):
    rng = np.random.default_rng(nl * nr)
    left = [rng.integers(0, keys, nl).astype(np.uint32), np.arange(nl, dtype=np.uint64)]
    right = [np.arange(nr, dtype=np.float32), (rng.permutation(nr) % keys).astype(np.uint32)]
    lb, rb = p.create_buffer_from_slices(left), p.create_buffer_from_slices(right)
    l, r = inner(left[0], right[1])
    for g, w in zip(p.download(p.hash_join_v2(lb, rb, [0], [1])), [c[l] for c in left] + [c[r] for c in right]):
        assert np.array_equal(g, w)
    has = np.isin(left[0], right[1])
    for kind, keep in ((A.JOIN_SEMI, has), (A.JOIN_ANTI, ~has)):
        for g, w in zip(p.download(p.hash_join_v2(lb, rb, [0], [1], kind)), left):
            assert np.array_equal(g, w[keep])


# ... and groups whose tables are at most 160 KB (2 tables of 8 bytes and the counts: 2^13 keys)
@pytest.mark.parametrize("n", [1, 1023, 1025, 8192, 8193])
@pytest.mark.parametrize("top", [0, 1, 1023, 8191, 8192, 1 << 31])
@pytest.mark.parametrize("nk", [1, 2])
def test_groups_of_one_block(p, n, top, nk):
    rng = np.random.default_rng(n + top)
    key = rng.integers(0, top, n, endpoint=True).astype(np.uint32)
    key[0] = top
    cols = [key, (key >> np.uint32(3)) % np.uint32(5)][:nk] + [rng.integers(0, 1 << 32, n, dtype=np.uint32), rng.integers(0, 1 << 40, n, dtype=np.uint64)]
    got = p.download(p.groupby_multi_agg(p.create_buffer_from_slices(cols), list(range(nk)), [(nk, A.AGG_COUNT), (nk, A.AGG_SUM), (nk + 1, A.AGG_MIN)]))
    order = np.lexsort(cols[:nk][::-1])
    s = [c[order] for c in cols]
    first = np.flatnonzero(np.concatenate([[True], np.any([k[1:] != k[:-1] for k in s[:nk]], axis=0)])) if n > 1 else np.array([0])
    want = [k[first] for k in s[:nk]] + [np.diff(np.append(first, n)), np.add.reduceat(s[nk].astype(np.uint64), first), np.minimum.reduceat(s[nk + 1], first)]
    for g, w in zip(got, want):
        assert np.array_equal(g.astype(np.uint64), w.astype(np.uint64))


# rows of one key next to each other in a warp, alone in it, all of them, in a warp that is not full
@pytest.mark.parametrize("n", [1, 3, 31, 33, 1000, 1025, 8191, 8192])
@pytest.mark.parametrize("kind", ["one", "two", "ten", "hub", "runs", "all", "late"])
def test_few_groups_of_one_block(p, n, kind):
    rng = np.random.default_rng(n)
    i = np.arange(n)
    key = {"one": i * 0, "two": rng.integers(0, 2, n), "ten": rng.integers(0, 10, n), "hub": np.where(rng.integers(0, 10, n), 777, rng.integers(0, 4096, n)), "runs": i // 5, "all": i,
           "late": np.where(i % 32 > 27, 5, i % 32)}[kind].astype(np.uint32)
    cols = [key, rng.integers(0, 1 << 32, n, dtype=np.uint32), rng.integers(1 << 63, 1 << 64, n, dtype=np.uint64, endpoint=False)]
    got = p.download(p.groupby_multi_agg(p.create_buffer_from_slices(cols), [0], [(1, A.AGG_SUM), (2, A.AGG_MAX), (1, A.AGG_COUNT), (2, A.AGG_MIN), (2, A.AGG_SUM)][: 5 if kind != "all" else 2]))
    order = np.argsort(key, kind="stable")
    u, at = np.unique(key[order], return_index=True)
    v, w = cols[1][order].astype(np.uint64), cols[2][order]
    want = [u, np.add.reduceat(v, at), np.maximum.reduceat(w, at), np.diff(np.append(at, n)).astype(np.uint64), np.minimum.reduceat(w, at), np.add.reduceat(w, at)]
    for g, x in zip(got, want):
        assert np.array_equal(g.astype(np.uint64), x.astype(np.uint64))


# Groups of a key and outputs beyond the room that one block's columns have, up to and past the longest group; key 0 among them
@pytest.mark.parametrize("npr,nb,keys", [(100, 100, 2), (300, 300, 10), (1025, 64, 1), (1100, 4096, 64), (8192, 4096, 64), (8192, 4000, 400), (8192, 64, 1), (18, 4096, 64), (8191, 129, 2), (8191, 130, 2), (1, 4096, 1), (100, 256, 1), (100, 257, 1), (500, 4096, 300), (500, 3600, 300), (500, 3900, 300), (8192, 3840, 15)])
@pytest.mark.parametrize("dtype", [np.uint32, np.uint64])
def test_more_outputs_than_one_block_has_room_for(p, npr, nb, keys, dtype):
    rng = np.random.default_rng(npr + nb)
    left = [rng.integers(0, keys + 1, npr).astype(dtype), np.arange(npr, dtype=np.uint64)]
    right = [np.arange(nb, dtype=np.float32), (rng.permutation(nb) % keys).astype(dtype)]
    lb, rb = p.create_buffer_from_slices(left), p.create_buffer_from_slices(right)
    l, r = inner(left[0], right[1])
    for _ in range(2):
        for g, w in zip(p.download(p.hash_join_v2(lb, rb, [0], [1])), [c[l] for c in left] + [c[r] for c in right]):
            assert np.array_equal(g, w)


# Many build rows: groups of 9 to 16 go out from lists where they go out often
@pytest.mark.parametrize("group,ratio", [(8, 8), (9, 5), (9, 6), (13, 4), (16, 3), (16, 4), (17, 1)])
def test_joins_of_many_rows_from_chains_and_from_lists(p, group, ratio):
    rng = np.random.default_rng(group)
    n = (1 << 18) + 5000
    key = rng.permutation(np.arange(n, dtype=np.uint64) // np.uint64(group) * np.uint64(977) + np.uint64(1))
    ask = key[rng.integers(0, n, n * ratio // group)]
    left, right = [ask, np.arange(len(ask), dtype=np.uint32)], [np.arange(n, dtype=np.uint32), key]
    l, r = inner(ask, key)
    for g, w in zip(p.download(p.hash_join_v2(p.create_buffer_from_slices(left), p.create_buffer_from_slices(right), [0], [1])), [c[l] for c in left] + [c[r] for c in right]):
        assert np.array_equal(g, w)


# Rows of a key next to each other in the build side: a warp's lanes claim one slot, count and link on it at once
@pytest.mark.parametrize("group", [2, 3, 8, 15, 16, 17, 31, 32, 64])
@pytest.mark.parametrize("apart", [1, 32, 256, 5000])
def test_rows_of_one_key_side_by_side(p, group, apart):
    n = 60_000
    i = np.arange(n, dtype=np.uint64)
    key = (i // np.uint64(apart * group) * np.uint64(apart) + i % np.uint64(apart)) * np.uint64(3)  # (`group` rows each, `apart` rows from one to the next)
    rng = np.random.default_rng(group)
    left, right = [rng.integers(0, int(key.max()) + 1, 9000, dtype=np.uint64), np.arange(9000, dtype=np.uint32)], [i.astype(np.uint32), key]
    l, r = inner(left[0], key)
    lb, rb = p.create_buffer_from_slices(left), p.create_buffer_from_slices(right)
    for _ in range(5):
        for g, w in zip(p.download(p.hash_join_v2(lb, rb, [0], [1])), [c[l] for c in left] + [c[r] for c in right]):
            assert np.array_equal(g, w)
