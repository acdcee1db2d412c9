"""Kernel launches of the counting sort that fail are reported by the call they
belong to, also when an earlier error is pending, and nothing is launched on
what they left undone: the entry points' own objects, linked against a CUDA
runtime that fails the k-th launch (tests/cpp/sort_launch_errors.cpp)."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.parametrize("known_context", [0, 1])  # scratch of the default pool, of the library's own
def test_failed_launches_are_reported(tmp_path, known_context):
    from lustrine_gb300 import _lib, build
    _lib.load()  # builds the objects if needed
    exe = tmp_path / "sort_launch_errors"
    objs = [os.path.join(build.BUILD, f"pbf_sort{u}.o") for u in ("", "_api", "_noalloc")]
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-w", f"-DKNOWN_CONTEXT={known_context}",
                        os.path.join(ROOT, "tests", "cpp", "sort_launch_errors.cpp"), *objs, "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout[-2000:]
