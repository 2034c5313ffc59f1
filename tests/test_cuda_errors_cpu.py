"""Calls of the CUDA runtime: a failure is reported where it happens and never left on the thread for
the next launch to find.  The host-only sources run here against a stand-in for the runtime."""
import ctypes as C
import glob
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "xlog_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def build(tmp, body, *sources):
    """A library of `body` and host-only sources of the library, over the stand-in runtime."""
    src, out = os.path.join(tmp, "t.cpp"), os.path.join(tmp, "t.so")
    with open(src, "w") as f:
        f.write('#include "%s/tests/fake_cudart.h"\n' % ROOT + "".join('#include "%s/%s"\n' % (CSRC, s) for s in sources) + body)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-pthread", "-I", os.path.join(CUDA, "include"), "-o", out, src])
    return C.CDLL(out)


def test_every_runtime_call_is_checked():
    free = {"cudaGetLastError", "cudaPeekAtLastError", "cudaGetErrorString"}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*")) + glob.glob(os.path.join(CSRC, "*.h"))):
        for i, line in enumerate(open(path), 1):
            for m in re.finditer(r"\b(cuda[A-Z]\w*)\(", line.split("//")[0]):
                before = line[:m.start()].rstrip()
                checked = re.search(r"(CUDA_OK|CUDA_QUIET|cuda_take)\(\(?$", before)
                passed_on = before.endswith("return")  # to callers that check it
                if m.group(1) not in free and line[:m.start()].count('"') % 2 == 0:
                    assert checked or passed_on, f"{os.path.basename(path)}:{i}: {line.strip()}"


def test_a_reported_failure_is_taken_off_the_thread(tmp_path):
    lib = build(str(tmp_path), """
extern "C" int status_of_failing_call() {
    fake.fail_register = 1;
    try {
        CUDA_OK(cudaHostRegister(nullptr, 0, 0));
    } catch (const XlbError& e) {
        return e.st;
    }
    return -1;
}
extern "C" int left() { return cudaPeekAtLastError(); }
""", "xlb_error.h")
    assert lib.status_of_failing_call() == 3  # XLB_ERR_RESOURCE_EXHAUSTED
    assert lib.left() == 0


def test_the_pool_leaves_no_error_behind(tmp_path):
    lib = build(str(tmp_path), """
extern "C" int left() { return cudaPeekAtLastError(); }
extern "C" void fail(int r, int u) { fake.fail_register = r; fake.fail_unregister = u; }
extern "C" int registered() { return fake.registered; }
""", "xlb_host.cu")
    p = C.c_void_p()
    lib.fail(1, 0)
    assert lib.xlb_host_alloc(C.c_uint64(1 << 20), C.byref(p)) == 3 and lib.left() == 0
    lib.fail(0, 1)
    assert lib.xlb_host_alloc(C.c_uint64(1 << 20), C.byref(p)) == 0
    lib.xlb_host_free(p)  # no context is open: given back at once
    assert lib.registered() == 0 and lib.left() == 0
