"""Every field of a launch shape changes the launches of the PBF list build and
passes that it names, for every list format and on both sides of the sizes up to
which a list build of 256 threads takes four lanes a particle (the launchers over
a runtime that records, tests/cpp/launch_shapes.cu)."""
import os
import subprocess
from collections import defaultdict

from conftest import ROOT


def test_shape_fields_reach_the_launches(tmp_path):
    from lustrine_gb300 import _lib, build
    _lib.load()  # builds the objects if needed
    cpp, exe = os.path.join(ROOT, "tests", "cpp"), tmp_path / "launch_shapes"
    objs = [os.path.join(build.BUILD, f"pbf_{u}.o") for u in ("solver", "compact", "sort")]
    r = subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, "-cudart", "none", "-Xcompiler", "-w",
                        os.path.join(cpp, "launch_shapes.cu"), os.path.join(cpp, "launch_shapes_runtime.cpp"),
                        *objs, "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr[-2000:]
    passes, lists = defaultdict(dict), {}
    for line in r.stdout.splitlines():
        name, n, kind, list_block, block, unroll, grid, threads, kernel, count = line.split()
        n, list_block, block, unroll, grid, threads = map(int, (n, list_block, block, unroll, grid, threads))
        assert count == "1"
        if name == "lists":
            per = {"16": 11_000, "column": 20_000, "frame": 20_000}.get(kind, 0)
            lanes = 4 if list_block == 256 and n <= per else 1
            assert (threads, grid) == (list_block, -(-n * lanes // list_block)), line
            lists.setdefault((n, kind, list_block), kernel)
            assert lists[n, kind, list_block] == kernel
        else:
            assert (threads, grid) == (block, -(-n // block)), line
            passes[name, n, kind][block, unroll] = kernel
    assert len(lists) == 4 * 5 * 3 and len(passes) == 3 * 4 * 5
    for key, kernels in passes.items():
        assert len(kernels) == len(set(kernels.values())) == 12, key
