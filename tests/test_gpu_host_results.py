"""Results fetched into staged and into page-locked memory: sizes around the limit of the staging
buffer, columns of every width, results that outlive their context, blocks used again."""
import gc

import numpy as np
import pytest

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
