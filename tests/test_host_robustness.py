"""Host classes of the native library under threads, a second device and little memory, without a GPU."""
import os
import shutil
import subprocess

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


@pytest.mark.parametrize("name,sources", [("host_lazy_stream", []), ("host_pool", ["pool.cpp"])])
def test_host_classes(tmp_path, name, sources):
    _run_program(tmp_path, name, *(os.path.join(CSRC, s) for s in sources))
