"""The library's host code against a fake CUDA runtime (tests/cpp/
fake_cudart.h): failures and lifetimes that need no GPU."""
import os
import subprocess

import pytest

from broxy_gb300 import _lib as L

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("tu", ["test_launch_status.cpp", "test_batch_graph.cpp", "test_batch_alloc.cpp", "test_frame_field_alloc.cpp", "test_stale_error.cpp"])
def test_host_code(tmp_path, tu):
    from __graft_entry__ import build
    build()
    libdir, exe = os.path.dirname(L.LIB_PATH), str(tmp_path / "host_code")
    # (-rdynamic: the library takes the executable's runtime functions)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-rdynamic", "-I", os.path.join(ROOT, "broxy_gb300", "csrc"),
                        "-I", os.path.join(ROOT, "include"), "-I/usr/local/cuda/include",
                        os.path.join(ROOT, "tests", "cpp", tu), "-o", exe,
                        "-L", libdir, "-lgmorpho_gb300", "-Wl,-rpath," + libdir,
                        "-L/usr/local/cuda/lib64", "-lcudart"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([exe], env=dict(os.environ, CUDA_VISIBLE_DEVICES=""), capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
