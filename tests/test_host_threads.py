"""Host threads that share the copy of a result table, or the sets of a batched
join, when memory or threads are refused (csrc/host_threads.h)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_refused_memory_and_threads(tmp_path):
    exe = tmp_path / "host_threads_check"
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-pthread",
                           "-I", os.path.join(ROOT, "hybrid_k_nearest_neighbor_self_join_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "host_threads_check.cpp"), "-o", str(exe), "-ldl"])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "cases=144 bad=0" in out.stdout
