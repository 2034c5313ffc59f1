"""Threads that write a column of runs out: every row, whatever the runs, and no core while there is nothing to do."""
import ctypes as C
import time

import numpy as np
import pytest

from test_cuda_errors_cpu import build


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return build(str(tmp_path_factory.mktemp("fill")), """
extern "C" Filler<uint32_t>* begin(unsigned threads) { return new Filler<uint32_t>(threads); }
extern "C" void end(Filler<uint32_t>* f) { delete f; }
extern "C" void fill(Filler<uint32_t>* f, uint32_t* to, const Run<uint32_t>* runs, uint64_t n_runs, uint64_t n) { f->fill(to, runs, n_runs, n); }
""", "xlb_fill.h")


def begin(lib, threads):
    lib.begin.restype = C.c_void_p
    return C.c_void_p(lib.begin(threads))


def test_waiting_threads_sleep(lib):
    for told in (False, True):
        f = begin(lib, 4)
        t = time.process_time()
        time.sleep(0.5)
        assert time.process_time() - t < 0.1  # (spinning, each of three took 0.5)
        if told:
            out, runs = np.zeros(1 << 20, np.uint32), np.array([[0, 7]], np.uint32)
            lib.fill(f, C.c_void_p(out.ctypes.data), C.c_void_p(runs.ctypes.data), C.c_uint64(1), C.c_uint64(len(out)))
        lib.end(f)
        assert not told or np.all(out == 7)


@pytest.mark.parametrize("threads", [1, 4])
@pytest.mark.parametrize("n,starts", [(1, [0]), (65535, [0, 1, 65534]), (65537, [0, 65536]), (300_001, list(range(0, 300_001, 17))), (300_001, [0, 65535, 65536, 131072, 300_000])])
def test_every_row_is_written(lib, n, starts, threads):
    runs = np.stack([starts, np.arange(len(starts)) * 3 + 1], axis=1).astype(np.uint32)
    want = np.repeat(runs[:, 1], np.diff(np.append(starts, n)))
    for off in (0, 1, 15):
        out = np.zeros(n + 32, np.uint32)
        f = begin(lib, threads)
        lib.fill(f, C.c_void_p(out.ctypes.data + 4 * off), C.c_void_p(runs.ctypes.data), C.c_uint64(len(runs)), C.c_uint64(n))
        lib.end(f)
        assert np.array_equal(out[off:off + n], want) and not out[:off].any() and not out[off + n:].any()
