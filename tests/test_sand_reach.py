"""The sand contacts' squared reach (sand_reach.h) for every kind of diameter:
the search ends and gives the bound it promises.  On the GPU: sand steps at
diameters from negative to all neighbours in contact against the oracle's
restatement of simulate_sand (Simulate.cpp:156-325), bit for bit."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, phys_params


def test_contact_reach(tmp_path):
    exe = tmp_path / "sand_reach"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "lustrine_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "sand_reach.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout[-2000:]


@pytest.mark.gpu
@pytest.mark.parametrize("diameter", [-1.0, 0.0, 1e-20, 0.7, 3.0])
def test_sand_steps_at_diameters(orc, diameter):
    from lustrine_gb300 import PbfSim, sand_params
    n, domain = 500, (14, 14, 14)
    rng = np.random.default_rng(7)
    i = np.arange(n)
    x = (np.stack([i // 8 % 8, i // 64, i % 8], 1) * 0.9 + rng.uniform(2.8, 3.2, (n, 3))).astype(np.float32)
    x[1] = x[0]  # coincident particles
    v = rng.normal(0, 0.5, x.shape).astype(np.float32)
    q, p = sand_params(*domain), phys_params(orc.reference_params(*domain, 0.5, 2.0))
    if diameter < 0:  # the diameter that a context starts with is twice its particles' radius
        q.particle_radius = p.particle_radius = diameter / 2
    with PbfSim(q, n) as sim:
        if diameter >= 0:
            sim.set_sand_controls(diameter=diameter)
        sim.upload(x, v, None)
        a = np.zeros(n, np.int32)
        for _ in range(2):
            o = orc.sand_step(p, orc.sand_controls(diameter=diameter), np.float32(1 / 60), x, v, a, cap=512)
            sim.step(1 / 60)
            gx, gv, _, _ = sim.download()
            x, v, a = o["x"], o["v"], o["attracted"]
            np.testing.assert_array_equal(gx, x)
            np.testing.assert_array_equal(gv, v)
