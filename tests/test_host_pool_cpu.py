"""The pool of page-locked result memory with several devices, ranks and threads, over a stand-in for
the CUDA runtime."""
import ctypes as C
import os
import random
import threading
import time

import pytest

from test_cuda_errors_cpu import build

OK, EXHAUSTED = 0, 3
MB = 1 << 20


@pytest.fixture()
def pool(tmp_path):
    lib = build(str(tmp_path), """
extern "C" void opened(int d) { host_pool_context_opened(d); }
extern "C" void closed(int d) { host_pool_context_closed(d); }
extern "C" int last_device() { return fake.last_device; }
extern "C" int touched_devices() { return fake.touched_devices.exchange(0); }
extern "C" int registered() { return fake.registered; }
extern "C" int device_here() { return fake_device; }
extern "C" void device_is(int d) { fake_device = d; }
extern "C" void registration_takes(int ms) { fake.register_ms = ms; }
extern "C" uint64_t most() { return host_pool_most(); }
extern "C" unsigned cores() { return host_pool_cores(); }
extern "C" unsigned quota(const char* groups, const char* mount) { return host_cores_quota(groups, mount); }
extern "C" void ranks(unsigned n) { host_pool_ranks(n); }
extern "C" void fail(int r, int u) { fake.fail_register = r; fake.fail_unregister = u; }
""", "xlb_host.cu")
    lib.xlb_host_alloc.argtypes = [C.c_uint64, C.POINTER(C.c_void_p)]
    lib.xlb_host_free.argtypes = [C.c_void_p]
    lib.most.restype = C.c_uint64
    return lib


def alloc(lib, size, status=OK):
    p = C.c_void_p()
    assert lib.xlb_host_alloc(size, C.byref(p)) == status
    return p.value


def in_thread(f):
    got = []
    t = threading.Thread(target=lambda: got.append(f()))
    t.start()
    t.join()
    return got[0]


def test_a_fresh_thread_uses_the_device_of_the_open_context(pool):
    pool.device_is(5)
    pool.opened(5)
    a = alloc(pool, MB)                       # the rank's own thread
    assert pool.last_device() == 5
    b = in_thread(lambda: alloc(pool, MB))    # one that never chose a device
    assert pool.last_device() == 5
    for p in (a, b):
        in_thread(lambda: pool.xlb_host_free(p))
    in_thread(lambda: pool.closed(5))         # the last context: what is kept is given back
    assert pool.last_device() == 5 and pool.registered() == 0
    assert pool.touched_devices() == 1 << 5   # device 0 is nobody's here
    assert in_thread(pool.device_here) == 0 and pool.device_here() == 5


@pytest.mark.parametrize("said", [None, "8", "0", "many"])
def test_ranks_share_the_bound(pool, said, monkeypatch):
    memory = os.sysconf("SC_PHYS_PAGES") * os.sysconf("SC_PAGE_SIZE")
    share = lambda ranks: min(16 << 30, memory // 8 // ranks)  # noqa: E731
    monkeypatch.delenv("LOCAL_WORLD_SIZE", raising=False)
    assert pool.most() == share(1)
    if said is not None:
        monkeypatch.setenv("LOCAL_WORLD_SIZE", said)
    assert pool.most() == share(8 if said == "8" else 1)
    pool.ranks(4)  # a communicator
    assert pool.most() == share(8 if said == "8" else 4)
    monkeypatch.setenv("LOCAL_WORLD_SIZE", str(memory // (64 * MB)))  # a share of 8 MB
    alloc(pool, 6 * MB)
    alloc(pool, 4 * MB, EXHAUSTED)
    alloc(pool, 1 << 63, EXHAUSTED)
    alloc(pool, (1 << 64) - 1, EXHAUSTED)


def test_others_do_not_wait_while_a_block_is_made(pool):
    pool.opened(0)
    kept, held = alloc(pool, 4 * MB), alloc(pool, 16 * MB)
    pool.xlb_host_free(kept)
    pool.registration_takes(1500)
    maker = threading.Thread(target=lambda: alloc(pool, 64 * MB))
    maker.start()
    time.sleep(0.3)
    t = time.perf_counter()
    pool.xlb_host_free(held)
    assert alloc(pool, 4 * MB) == kept
    assert time.perf_counter() - t < 0.5 and maker.is_alive()
    maker.join()
    assert pool.registered() == 3


def test_many_threads(pool, monkeypatch):
    # blocks of all sizes under a bound that they reach: nobody shares one, and all come back
    monkeypatch.setenv("LOCAL_WORLD_SIZE", str(os.sysconf("SC_PHYS_PAGES") * os.sysconf("SC_PAGE_SIZE") // 8 // (48 * MB)))
    pool.opened(0)
    owned, lock, wrong = set(), threading.Lock(), []

    def work(seed):
        rng = random.Random(seed)
        for _ in range(60):
            p = C.c_void_p()
            st = pool.xlb_host_alloc(rng.randint(1, 12 * MB), C.byref(p))
            if st == EXHAUSTED:
                continue
            with lock:
                if st != OK or p.value in owned:
                    wrong.append((st, p.value))
                owned.add(p.value)
            with lock:
                owned.discard(p.value)
            pool.xlb_host_free(p)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    pool.closed(0)
    assert pool.registered() == 0


def test_without_a_context_the_thread_decides(pool):
    pool.device_is(3)
    p = alloc(pool, MB)
    assert pool.last_device() == 3
    pool.xlb_host_free(p)
    assert pool.registered() == 0 and pool.touched_devices() == 1 << 3


@pytest.mark.parametrize("groups,files,cores", [
    ("0::/\n", {}, 0),
    ("0::/\n", {"cpu.max": "max 100000"}, 0),
    ("0::/\n", {"cpu.max": "350000 100000"}, 3),
    ("0::/\n", {"cpu.max": "50000 100000"}, 1),
    ("0::/a/b\n", {"a/b/cpu.max": "max 100000", "a/cpu.max": "200000 100000", "cpu.max": "900000 100000"}, 2),
    ("3:cpuset:/x\n2:cpuacct,cpu:/x\n1:memory:/x\n", {"cpu/x/cpu.cfs_quota_us": "400000", "cpu/x/cpu.cfs_period_us": "100000"}, 4),
    ("2:cpu:/x\n0::/\n", {"cpu/x/cpu.cfs_quota_us": "-1", "cpu/x/cpu.cfs_period_us": "100000", "cpu/cpu.cfs_quota_us": "-1"}, 0),
    ("nonsense\n\n4:\n0::\n", {"cpu.max": "oops"}, 0),
])
def test_cores_under_a_quota(pool, tmp_path, groups, files, cores):
    (tmp_path / "cgroup").write_text(groups)
    for name, text in files.items():
        f = tmp_path / "mount" / name
        f.parent.mkdir(parents=True, exist_ok=True)
        f.write_text(text + "\n")
    assert pool.quota(str(tmp_path / "cgroup").encode(), str(tmp_path / "mount").encode()) == cores
    assert pool.quota(b"/nowhere", b"/nowhere") == 0


def test_cores_of_this_process(pool, monkeypatch):
    cores = pool.cores()
    assert 1 <= cores <= len(os.sched_getaffinity(0))
    monkeypatch.setenv("LOCAL_WORLD_SIZE", "2")
    assert pool.cores() == cores // 2
