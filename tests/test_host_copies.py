"""CPU test of the host copies (csrc/host_copy.h) against a stand-in for CUDA's copies:
every byte arrives at chunk edges, in both directions, and VFEM_HOST_COPY_THREADS
bounds the threads that take part."""
import os
import subprocess

import pytest

from tests.conftest import ROOT


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    from vulkanfem_gb300 import build
    exe = str(tmp_path_factory.mktemp("copies") / "host_copy_check")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", build.CSRC, "-I", cuda, "-o", exe,
                        os.path.join(ROOT, "tests", "host_copy_check.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("setting,threads", [("1", 1), ("2", 2), ("", 8), ("many", 8), ("-5", 1)])
def test_copies_and_thread_bound(program, setting, threads):
    env = dict(os.environ, VFEM_HOST_COPY_THREADS=setting)
    r = subprocess.run([program], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert 1 <= int(r.stdout) <= 1 + min(threads, os.cpu_count())


@pytest.mark.parametrize("allocations", [0, 1, 2, 3, 5, 60])
def test_without_memory_for_threads(program, allocations):
    """No exception leaves the copies, which are called from C entries."""
    r = subprocess.run([program, str(allocations)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
