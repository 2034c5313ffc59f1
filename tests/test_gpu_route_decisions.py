"""Routes that give up in favour of another one: around the sizes at which they do, and with what makes
them notice early or late."""
import numpy as np
import pytest

from xlog_b200 import _abi as A
from xlog_b200.provider import KernelProvider

from test_gpu_query_paths import inner

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def p():
    prov = KernelProvider(device=0)
    yield prov
    prov.close()


# (the build side is sampled from 2048 rows on; a key of half of them is met there, one of 65 only when counted)
@pytest.mark.parametrize("nr,longest", [(64, 64), (65, 65), (2047, 2047), (2048, 64), (2048, 65), (2048, 2048), (2049, 1025), (300_000, 64), (300_000, 65), (300_000, 4000), (300_000, 150_000), (300_000, 300_000)])
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
