"""Set operations over small domains (a bitmap of the domain) and larger ones (sorted, merged)."""
import numpy as np
import pytest

from xlog_b200.provider import KernelProvider

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def prov():
    return KernelProvider(device=0)


def _pairs(rng, n, bits):
    return [rng.integers(0, 1 << b, n, dtype=np.uint64).astype(np.uint32) for b in bits]


def _words(cols):
    w = np.zeros(len(cols[0]), np.uint64)
    for c in cols:
        w = (w << np.uint64(32)) | c
    return w


# n rows against 2**sum(bits) possible ones: on both sides of the line, and around a tile of a selection
@pytest.mark.parametrize("n,bits", [
    (1, (1, 1)), (5, (3, 0)), (2048, (9, 9)), (2049, (9, 9)), (2047, (10, 9)), (4096, (12,)), (70001, (12, 12)),
    (70001, (3, 20)), (70001, (13, 20)), (70001, (32,)), (300007, (11, 17)),
])
def test_dedup_difference_union(prov, n, bits):
    rng = np.random.default_rng(n + sum(bits))
    a, b, d = _pairs(rng, n, bits), _pairs(rng, n // 3 + 1, bits), _pairs(rng, n // 2, bits)
    wa, wb, wd = (np.unique(_words(x)) for x in (a, b, d))
    ra, rb, rd = (prov.create_buffer_from_slices(x) for x in (a, b, d))

    def same(buf, want):
        assert buf.is_canonical()
        assert np.array_equal(_words(prov.download(buf)), want)

    ca, cb = prov.dedup_full_row(ra), prov.dedup_full_row(rb)
    same(ca, wa)
    same(prov.diff_gpu(ca, cb), np.setdiff1d(wa, wb))
    same(prov.diff_gpu(ra, rb), np.setdiff1d(wa, wb))
    same(prov.union_gpu(ca, cb), np.union1d(wa, wb))
    same(prov.union_many_gpu([ra, cb, rd]), np.union1d(np.union1d(wa, wb), wd))
    assert np.array_equal(_words(prov.download(ra)), _words(a))  # the inputs are as they were
