"""The default launch shape gives way where many contexts share the device: the
rule on the CPU (tests/cpp/default_shape.cu), and on the GPU contexts in a crowd
against the same contexts alone, bit for bit."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def test_rule(tmp_path):
    from lustrine_gb300 import build
    cpp, exe = os.path.join(ROOT, "tests", "cpp"), tmp_path / "default_shape"
    r = subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, "-cudart", "none", "-Xcompiler", "-w",
                        os.path.join(cpp, "default_shape.cu"), os.path.join(cpp, "launch_shapes_runtime.cpp"),
                        "-lpthread", "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout[-2000:]


@pytest.mark.gpu
@pytest.mark.parametrize("precision,solids", [(0, 0), (0, 60), (1, 60), (2, 0)])
def test_bits_in_a_crowd(precision, solids):
    from lustrine_gb300 import PbfSim, pbf_params
    sizes = [700, 5_000, 9_000, 18_000, 60_000, 300_000]  # more than two waves

    def scene(n):
        rng = np.random.default_rng(n)
        a = int(np.ceil(n ** (1 / 3)))
        i = np.arange(n)
        x = np.stack([i // a % a, i // (a * a), i % a], 1) * 0.9 + 1.5 + rng.uniform(-0.2, 0.2, (n, 3))
        s = rng.uniform(1, 0.9 * a, (solids, 3)).astype(np.float32) if solids else None
        return x.astype(np.float32), s, a + 3

    def make(n):
        x, s, side = scene(n)
        sim = PbfSim(pbf_params(side, side, side, iterations=2, precision=precision), n, solids)
        sim.upload(x, None, s)
        return sim

    def steps(sim):
        for _ in range(4):  # launched, captured and replayed
            sim.step(1 / 60)
        assert sim.status() == 0
        return sim.download(lambdas=True, density=True)

    alone = []
    for n in sizes:
        with make(n) as sim:
            alone.append(steps(sim))
    crowd = [make(n) for n in sizes]
    for sim, want in zip(crowd, alone):
        for u, w in zip(steps(sim), want):
            np.testing.assert_array_equal(u, w)
    for sim in crowd[:-1]:
        sim.close()
    x, s, _ = scene(sizes[-1])  # alone again, with the shape it captured
    crowd[-1].upload(x, None, s)
    for u, w in zip(steps(crowd[-1]), alone[-1]):
        np.testing.assert_array_equal(u, w)
    crowd[-1].close()
