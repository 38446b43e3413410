"""Host classes of the native library under threads, a second device and little memory, without a GPU."""
import os
import resource
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ftlm_extended_hubbard_b200", "csrc")
CUDA = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))


def _run_program(tmp_path, name, *sources):
    """Compiles tests/<name>.cpp against the pretended runtime of tests/fake_runtime.hpp and runs it."""
    exe = str(tmp_path / name)
    cmd = ["g++", "-std=c++17", "-O1", "-pthread", "-I", HERE, "-I", CSRC, "-I", os.path.join(CUDA, "include"),
           os.path.join(HERE, name + ".cpp"), *sources, "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("name,sources", [("host_lazy_stream", []), ("host_pool", ["pool.cpp"]), ("host_workers", [])])
def test_host_classes(tmp_path, name, sources):
    _run_program(tmp_path, name, *(os.path.join(CSRC, s) for s in sources))


_NO_THREADS = '''
import ctypes as C
import resource
import ftlm_extended_hubbard_b200 as F
from ftlm_extended_hubbard_b200 import _lib
hops, pairs = F.build_hubbard_geometry(F.HubbardParams(4, 4, 1.0, -0.25, 8.0, 1.0, 0.1, 0.0))
ch, cp = F.api._c_hops(hops), F.api._c_pairs(pairs)


def create(grow=None):
    h = C.c_void_p()
    old = resource.getrlimit(resource.RLIMIT_AS)
    if grow is not None:
        resource.setrlimit(resource.RLIMIT_AS, (size() + grow, old[1]))
    rc = _lib.lib().ftlm_gpu_sector_create_host(16, 7, 7, 8.0, 1.0, ch, len(hops), cp, len(pairs), C.byref(h))
    resource.setrlimit(resource.RLIMIT_AS, old)
    return rc, h


def entries(h):
    n, ng, nt, ok = C.c_longlong(), C.c_longlong(), C.c_int(), C.c_int()
    args = (h, C.byref(ok), C.byref(ng), C.byref(n), C.byref(nt), None)
    _lib.call("ftlm_gpu_sector_down_table_gauge", *args, None, None, None)
    ent = (C.c_uint32 * n.value)()
    _lib.call("ftlm_gpu_sector_down_table_gauge", *args, ent, None, None)
    return bytes(ent)


def size():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[0]) * resource.getpagesize()


want = entries(create()[1])
assert want
rc, h = create(220 << 20)
assert rc == 0 and entries(h) == want
'''


def test_plan_without_a_further_thread():
    """Where no worker thread can be started (256 MB of stack for each, 220 MB left) the plan of a 4x4 (7,7) sector, 11,440
    strings a species, is built without, and is the same."""
    def stack():
        resource.setrlimit(resource.RLIMIT_STACK, (256 << 20, 256 << 20))

    r = subprocess.run([sys.executable, "-c", _NO_THREADS], capture_output=True, text=True, timeout=300, preexec_fn=stack,
                       cwd=os.path.dirname(HERE))
    assert r.returncode == 0, r.stderr


_NO_MEMORY = '''
import resource
import numpy as np
from ftlm_extended_hubbard_b200 import _lib
n = 40000  # the n x n matrices take 13 GB
a, lam, z = np.ones(n), np.empty(n), np.empty(1)
with open("/proc/self/statm") as f:
    size = int(f.read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (size + (1 << 30),) * 2)
p = [v.ctypes.data for v in (a, a, lam, z)]
L = _lib.lib()
assert L.ftlm_gpu_duhamel_weights(p[0], p[1], n, 1.0, p[2], p[2], p[2]) == 3
assert b"allocation" in L.ftlm_gpu_last_error()
'''


def test_no_exception_crosses_the_c_interface():
    """Host memory that does not suffice is an error code (3)."""
    r = subprocess.run([sys.executable, "-c", _NO_MEMORY], capture_output=True, text=True, timeout=300, cwd=os.path.dirname(HERE))
    assert r.returncode == 0, r.stderr
