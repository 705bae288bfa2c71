"""Device code of prender_gb300/csrc compiled for the host (tests/host), where
a fault may be shown that must not run on a GPU: accesses of shared memory
between the lanes of a warp that no fence orders, loops that only their caps
end."""
import os
import shutil
import subprocess

import pytest

HOST = os.path.join(os.path.dirname(os.path.abspath(__file__)), "host")


def _cuda_include():
    from prender_gb300 import build
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")


def _run(tmp_path, name, flags=(), args=(), timeout=300):
    exe = str(tmp_path / name)
    subprocess.run([shutil.which("g++"), "-std=c++17", "-O1", "-g", "-w", "-ffp-contract=off", "-pthread",
                    "-isystem", _cuda_include(), *flags, "-o", exe, os.path.join(HOST, name + ".cpp")], check=True)
    return subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=timeout,
                          env=dict(os.environ, TSAN_OPTIONS="exitcode=66 halt_on_error=1"))


@pytest.mark.parametrize("sanitizer", [False, True])
def test_warp_triangles_is_each_lanes_own_loop_and_free_of_races(tmp_path, sanitizer):
    r = _run(tmp_path, "warp_triangles", ["-fsanitize=thread"] if sanitizer else [])
    if "FATAL: ThreadSanitizer" in r.stderr:  # this kernel's address layout is not one the sanitizer knows
        pytest.skip("the thread sanitizer does not start here")
    assert r.returncode == 0, r.stdout + r.stderr[-3000:]


@pytest.mark.parametrize("kind,hit,err,nodes", [(0, 1, 0, 1), (1, 0, 2, 1 << 24), (2, 0, 1, 22)])
def test_exact_traversal_of_a_malformed_tree_ends(tmp_path, kind, hit, err, nodes):
    """err: PR_DEV_LOOP_CAP after 2^24 visits, PR_DEV_STACK_OVERFLOW where 64
    entries, three more per visit, are full"""
    r = _run(tmp_path, "exact_tree", ["-O2"], [kind], timeout=60)
    got = [int(x) for x in r.stdout.split()]
    assert got[0] == hit and got[2] == err and got[3] == nodes


@pytest.mark.parametrize("length", [1.0, 1.0 + 4e-7, 1.0 - 4e-7, 1.0 + 3e-6, 0.5, 0.9, 2.0, 10.0])
def test_segments_left_out_have_no_hit(tmp_path, length):
    """the sphere test takes directions for unit vectors: with others it has
    roots where the line meets nothing"""
    r = _run(tmp_path, "segment_tests", ["-O2"], [length])
    assert r.returncode == 0, r.stdout + r.stderr[-3000:]


@pytest.mark.parametrize("length", [1.0, 0.7, 3.0])
@pytest.mark.parametrize("scene", ["walls", "nested", "hemispheres", "many"])
def test_sphere_runs_are_the_fp64_tests_of_every_sphere(tmp_path, scene, length):
    r = _run(tmp_path, "sphere_runs", ["-O2"], [scene, length])
    assert r.returncode == 0, r.stdout + r.stderr[-3000:]


def test_wavefront_pool_sizes(tmp_path):
    r = _run(tmp_path, "wavefront_pool")
    assert r.returncode == 0, r.stdout + r.stderr[-3000:]
