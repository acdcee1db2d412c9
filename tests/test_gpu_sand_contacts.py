"""The sand step where its list build and contact collection change path:
lists within and past the staged entries, more contacts than are collected at
once, list capacities below and above the staging, particles with and without
static particles nearby, block remainders.  Everything bit for bit against the
oracle's restatement of simulate_sand (Simulate.cpp:156-325)."""
import numpy as np
import pytest

from conftest import phys_params

pytestmark = pytest.mark.gpu


def _cloud(rng, n, spacing, domain, solids):
    """n particles on a jittered lattice of the given spacing; `solids` static
    ones scattered through the lower half of the box."""
    a = int(np.ceil(n ** (1 / 3)))
    i = np.arange(n)
    x = np.stack([i // a % a, i // (a * a), i % a], 1) * spacing + 1.0
    x = (x + rng.uniform(-0.3, 0.3, x.shape) * spacing).astype(np.float32)
    s = rng.uniform(0.6, 1.0, (solids, 3)) * (np.asarray(domain) * [1, 0.5, 1] - 1.2)
    return x, s.astype(np.float32)


@pytest.mark.parametrize("n,spacing,solids,scale,cap", [
    (1, 1.0, 0, 3.1, 96),
    (129, 1.0, 0, 3.1, 96),       # lists of some 18 entries: all staged
    (1000, 0.62, 0, 3.1, 128),    # some 60 entries, a dozen and more contacts
    (1500, 0.45, 0, 2.0, 200),    # more contacts than a thread collects at once
    (777, 0.9, 600, 3.1, 128),    # static particles in most cells
    (777, 0.9, 40, 2.0, 96),      # in few: both walks in a warp
    (640, 0.8, 100, 3.1, 8),      # cut at a capacity below the staged entries
    (640, 0.62, 0, 3.1, 30),      # and above them
])
def test_sand_lists_and_contacts_match_oracle(orc, n, spacing, solids, scale, cap):
    from lustrine_gb300 import PbfSim, sand_params
    rng = np.random.default_rng(n + solids + cap)
    domain = (16, 14, 15)
    x, s = _cloud(rng, n, spacing, domain, solids)
    v = rng.normal(0, 0.5, x.shape).astype(np.float32)
    sim = PbfSim(sand_params(*domain, kernel_radius_scale=scale, max_neighbors=cap), n, solids)
    sim.upload(x, v, s if solids else None)
    p = phys_params(orc.reference_params(*domain, 0.5, scale))
    ao = np.zeros(n, np.int32)
    xo, vo = x.copy(), v.copy()
    for step in range(2):
        ctl = orc.sand_controls(prev_attract=False, diameter=1.0)
        o = orc.sand_step(p, ctl, np.float32(1.0 / 60.0), xo, vo, ao, solid=s, cap=512)
        sim.step(1.0 / 60.0)
        cnt, idx = sim.neighbors(cap=512)
        full = [r[:c][r[:c] != k] for k, (c, r) in enumerate(zip(o["nbr_count"], o["nbr_idx"]))]
        longest = max(len(r) for r in full)
        for k in range(n):
            assert np.array_equal(idx[k, :cnt[k]], full[k][:cap]), f"step {step}: list {k}"
        if longest > cap:  # a cut list changes the contacts: only the lists compare
            assert sim.status() == 4
            break
        gx, gv, _, _ = sim.download()
        xo, vo, ao = o["x"], o["v"], o["attracted"]
        assert np.array_equal(gx, xo) and np.array_equal(gv, vo), f"step {step}"
        assert sim.status() == 0
    sim.close()
