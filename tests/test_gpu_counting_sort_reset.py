"""The counting sort's kept scratch after a reset of the device, in a process of
its own: the next call takes new scratch and reads its own status word."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C, glob, os, sys
import numpy as np
for name in ("libcudart.so.13", "/usr/local/cuda/lib64/libcudart.so"):
    try:
        rt = C.CDLL(name)
        break
    except OSError:
        rt = None
if rt is None:
    print("no cudart")
    sys.exit(0)
lib = C.CDLL(sys.argv[1])
def sort(n, cells, bad):
    k = np.random.default_rng(n).integers(0, cells, n).astype(np.int32)
    if bad:
        k[n // 2] = cells
    p = [C.c_void_p() for _ in range(3)]
    for q, m in zip(p, (n, cells + 1, n)):
        assert rt.cudaMalloc(C.byref(q), C.c_size_t(4 * m)) == 0
    assert rt.cudaMemcpy(p[0], k.ctypes.data_as(C.c_void_p), C.c_size_t(4 * n), 1) == 0
    rc = lib.lustrine_counting_sort(p[1], p[0], C.c_size_t(n), C.c_size_t(cells), p[2], None)
    out = np.zeros(n, np.int32)
    assert rt.cudaMemcpy(out.ctypes.data_as(C.c_void_p), p[2], C.c_size_t(4 * n), 2) == 0
    return rc != 0 if bad else rc == 0 and np.array_equal(out, np.argsort(k, kind="stable"))
for _ in range(3):
    assert lib.lustrine_release_scratch() == 0
    assert sort(1000, 100, False) and sort(1000, 100, True) and sort(70000, 5000, False)
    assert lib.lustrine_release_scratch() == 0
    assert sort(70000, 5000, False)
    assert rt.cudaDeviceReset() == 0
print("sorted")
"""


def test_sort_after_device_reset():
    from lustrine_gb300 import _lib, build
    _lib.load()
    r = subprocess.run([sys.executable, "-c", CHILD, str(build.LIB)], capture_output=True, text=True, timeout=300)
    if "no cudart" in r.stdout:
        pytest.skip("no shared CUDA runtime to reset the device with")
    assert r.returncode == 0 and "sorted" in r.stdout, (r.returncode, r.stderr[-500:])
