"""Rows ordered by key columns: words of the varying bits, row numbers beside them, columns decoded."""
import numpy as np
import pytest

from xlog_b200 import _abi as A
from xlog_b200.provider import KernelProvider

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def prov():
    return KernelProvider(device=0)


def _image(col):
    """Unsigned integers that order as the column's type does."""
    if col.dtype.kind == "f":
        u = col.view(np.uint32 if col.dtype.itemsize == 4 else np.uint64)
        sign = u.dtype.type(1) << u.dtype.type(8 * col.dtype.itemsize - 1)
        return np.where(u & sign, ~u, u | sign)
    if col.dtype.kind == "i":
        return (col.astype(np.int64).view(np.uint64)) ^ np.uint64(1 << 63)
    return col


def _column(rng, kind, n):
    if kind == "id":
        return rng.integers(0, max(n // 8, 2), n, dtype=np.uint32)
    if kind == "u32":
        return rng.integers(0, 1 << 32, n, dtype=np.uint32)
    if kind == "const":
        return np.full(n, 7, np.uint32)
    if kind == "u64":
        return rng.integers(0, 1 << 63, n, dtype=np.uint64) * np.uint64(2)
    if kind == "time":
        return rng.integers(-(1 << 39), 1 << 39, n, dtype=np.int64)
    if kind == "i32":
        return rng.integers(-5, 5, n, dtype=np.int32)
    if kind == "bool":
        return rng.integers(0, 2, n).astype(bool)
    c = rng.standard_normal(n).astype(np.float32 if kind == "f32" else np.float64)
    c[:: 7] = np.nan
    c[3:: 11] = -0.0
    return c


@pytest.mark.parametrize("n", [0, 1, 2, 1023, 1025, 8192, 8193, 30000, 200003])
@pytest.mark.parametrize("kinds,keys", [
    ("id id", [0, 1]),                # every column in the word: no row numbers
    ("id id u32", [0, 1]),            # row numbers beside the keys
    ("id time f32", [0, 1]),          # a word without room for them
    ("u64 f64 i32 bool", [0, 1, 2]),  # several words
    ("f32 bool i32 id", [3, 1, 0]),
    ("const u32 const", [0, 2]),      # nothing to sort by
    ("i32 f64", [0, 0]),              # a key named twice
])
def test_sort_rows(prov, n, kinds, keys):
    rng = np.random.default_rng(n + len(kinds))
    cols = [_column(rng, k, n) for k in kinds.split()]
    got = prov.download(prov.sort(prov.create_buffer_from_slices(cols), keys))
    order = np.lexsort([_image(cols[k]) for k in reversed(keys)]) if n else np.zeros(0, np.int64)
    for g, c in zip(got, cols):
        assert g.tobytes() == c[order].tobytes()


@pytest.mark.parametrize("n", [8193, 65536, 65537, 300007])
@pytest.mark.parametrize("kind", ["spread", "run33", "run34", "run_of_equal", "few"])
def test_rows_of_one_prefix(prov, n, kind):
    """Sorted by the highest bits, the rest put in order afterwards: prefixes of a few rows, of as many as
    that is done for, of more, and values that are too few for it."""
    rng = np.random.default_rng(n)
    key = rng.integers(0, 1 << 56, n, dtype=np.uint64)
    k = {"run33": 33, "run34": 34, "run_of_equal": 500}.get(kind, 0)
    if k:  # so many rows next to each other in the order, below the bits sorted by
        key[rng.choice(n, k, replace=False)] = np.uint64(123 << 40) + (np.zeros(k, np.uint64) if kind == "run_of_equal" else rng.integers(0, 1 << 10, k, dtype=np.uint64))
    if kind == "few":
        key = key[rng.integers(0, 50, n)]
    cols = [key, np.arange(n, dtype=np.uint32)]
    got = prov.download(prov.sort(prov.create_buffer_from_slices(cols), [0]))
    order = np.argsort(key, kind="stable")
    for g, c in zip(got, cols):
        assert np.array_equal(g, c[order])


@pytest.mark.parametrize("bits", [(1, 1), (7, 9), (12, 12), (13, 20), (32, 3), (3, 32), (32, 32)])
@pytest.mark.parametrize("n", [8192, 8193, 100001])
def test_digits_across_the_halves_of_a_pair(prov, bits, n):
    rng = np.random.default_rng(n + bits[0])
    a = rng.integers(0, 1 << bits[0], n, dtype=np.uint64).astype(np.uint32)
    b = rng.integers(0, 1 << bits[1], n, dtype=np.uint64).astype(np.uint32)
    want = np.unique((a.astype(np.uint64) << np.uint64(32)) | b)
    got = prov.download(prov.dedup_full_row(prov.create_buffer_from_slices([a, b], [A.U32, A.U32])))
    assert np.array_equal(got[0], (want >> np.uint64(32)).astype(np.uint32))
    assert np.array_equal(got[1], (want & np.uint64(0xFFFFFFFF)).astype(np.uint32))
