"""The two forms of the pair terms' reciprocal distance (inv_r_of: rsqrtf in
per-cell mixed passes, its flush-to-zero form elsewhere) give the same bits for
every float r2 >= 0: paths that must agree bit for bit use either."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.gpu
def test_both_forms_give_the_same_bits(tmp_path):
    from lustrine_gb300 import build
    exe = tmp_path / "inv_r"
    r = subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, os.path.join(ROOT, "tests", "cpp", "inv_r.cu"),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "no error" in r.stdout, r.stdout
