"""Device code of prender_gb300/csrc compiled for the host (tests/host), where
a fault may be shown that must not run on a GPU: accesses of shared memory
between the lanes of a warp that no fence orders."""
import os
import shutil
import subprocess

import pytest

HOST = os.path.join(os.path.dirname(os.path.abspath(__file__)), "host")


def _cuda_include():
    from prender_gb300 import build
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")


def _run(tmp_path, name, flags=(), timeout=300):
    exe = str(tmp_path / name)
    subprocess.run([shutil.which("g++"), "-std=c++17", "-O1", "-g", "-w", "-ffp-contract=off", "-pthread",
                    "-isystem", _cuda_include(), *flags, "-o", exe, os.path.join(HOST, name + ".cpp")], check=True)
    return subprocess.run([exe], capture_output=True, text=True, timeout=timeout,
                          env=dict(os.environ, TSAN_OPTIONS="exitcode=66 halt_on_error=1"))


@pytest.mark.parametrize("sanitizer", [False, True])
def test_warp_triangles_is_each_lanes_own_loop_and_free_of_races(tmp_path, sanitizer):
    r = _run(tmp_path, "warp_triangles", ["-fsanitize=thread"] if sanitizer else [])
    if "FATAL: ThreadSanitizer" in r.stderr:  # this kernel's address layout is not one the sanitizer knows
        pytest.skip("the thread sanitizer does not start here")
    assert r.returncode == 0, r.stdout + r.stderr[-3000:]
