"""Routes that give up in favour of another one: around the sizes at which they do, and with what makes
them notice early or late."""
import numpy as np
import pytest

from xlog_b200 import programs
from xlog_b200.executor import run_program
from xlog_b200.provider import KernelProvider

from test_gpu_query_paths import inner

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def p():
    prov = KernelProvider(device=0)
    yield prov
    prov.close()


# (the build side is sampled from 65536 rows on; a key of half of them is met there, one of 65 only when counted)
@pytest.mark.parametrize("nr,longest", [(64, 64), (65, 65), (2049, 1025), (65_535, 65_535), (65_536, 64), (65_536, 65), (65_536, 65_536), (65_537, 32_769), (300_000, 64), (300_000, 65), (300_000, 4000), (300_000, 150_000), (300_000, 300_000)])
@pytest.mark.parametrize("dtype", [np.uint32, np.uint64])
def test_join_with_one_long_key(p, nr, longest, dtype):
    rng = np.random.default_rng(nr + longest)
    rk = rng.permutation(np.concatenate([np.full(longest, 7), 100 + rng.permutation(nr - longest)])).astype(dtype)
    lk = np.concatenate([rng.integers(100, 100 + 2 * nr, 5000), np.full(3, 7)]).astype(dtype)
    lv, rv = np.arange(len(lk), dtype=np.uint32), rng.integers(0, 1 << 60, nr, dtype=np.uint64)
    got = p.download(p.hash_join_v2(p.create_buffer_from_slices([lk, lv]), p.create_buffer_from_slices([rv, rk]), [0], [1]))
    left, right = inner(lk, rk)
    for g, w in zip(got, [lk[left], lv[left], rv[right], rk[right]]):
        assert np.array_equal(g, w)


@pytest.mark.parametrize("bits", [28, 29, 31, 32])
@pytest.mark.parametrize("rows,values", [(65_537, 2), (65_537, 65_536), (65_537, 65_537), (200_000, 65_536), (200_000, 65_537), (200_000, 200_000), (3_000_000, 40_000), (3_000_000, 1_000_000)])
def test_closure_over_few_or_many_spread_values(bits, rows, values):
    # a loop at every value (over and over where rows are many) and a star: what is there is the closure
    rng = np.random.default_rng(rows + values + bits)
    ids = np.unique(np.concatenate([rng.integers(1, (1 << bits) - 1, 2 * values, dtype=np.uint64), [0, (1 << bits) - 1]]).astype(np.uint32))
    ids = np.concatenate([ids[[0, -1]], rng.permutation(ids[1:-1])[: values - 2]])
    assert len(np.unique(ids)) == values
    ids = rng.permutation(ids)
    loops = rng.permutation(np.resize(ids[1:], max(rows, values - 1)))
    tips = ids[1:1001]
    edge = [np.concatenate([np.full(len(tips), ids[0]), loops]), np.concatenate([tips, loops])]
    prov = KernelProvider(device=0)
    got, _ = run_program(prov, programs.transitive_closure(), {"edge": edge}, ["reach"])
    prov.close()
    pack = lambda c: (c[0].astype(np.uint64) << np.uint64(32)) | c[1]  # noqa: E731
    assert np.array_equal(pack(got["reach"]), np.unique(pack(edge)))
