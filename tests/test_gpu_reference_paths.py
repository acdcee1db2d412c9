"""The reference-semantics fluid step where its kernels change path: lists
within and past the staged entries, rows with and without solids, both halves
of the cubic kernel, s_corr exponents with and without the fp32 power, kernel
radii with and without the known-divisor quotient.  Neighbour lists equal in
order and lambdas bitwise (no power in them); positions and velocities within
the contract's 1e-5 of the oracle's Jacobi step (glibc's powf misrounds
0.07 % of the powers, so they are not always bitwise)."""
import numpy as np
import pytest

from conftest import phys_params

pytestmark = pytest.mark.gpu

REL = 1e-5


@pytest.mark.parametrize("n,spacing,solids,scale,factor,exponent", [
    (1, 1.0, 0, 2.0, 0.5, 4.0),
    (257, 1.0, 0, 3.1, 0.5, 4.0),     # lists of some 27 entries
    (900, 0.7, 0, 3.1, 0.5, 4.0),     # past the staged entries
    (700, 1.0, 500, 3.1, 0.5, 4.0),   # solids in most rows
    (700, 1.0, 30, 2.0, 0.5, 4.0),    # in few
    (500, 0.9, 0, 2.3, 1.0, 4.0),     # the kernel's outer half
    (500, 0.9, 0, 2.3, 0.5, 3.0),     # an exponent that takes the double power
    (500, 0.9, 20, 2.0, 0.8, 2.5),    # and one that takes powf
])
def test_reference_step_matches_oracle(orc, n, spacing, solids, scale, factor, exponent):
    from lustrine_gb300 import PbfSim, reference_params
    rng = np.random.default_rng(n + solids)
    domain = (18, 16, 17)
    a = int(np.ceil(n ** (1 / 3)))
    i = np.arange(n)
    x = np.stack([i // a % a, i // (a * a), i % a], 1) * spacing + 2.0
    x = (x + rng.uniform(-0.2, 0.2, x.shape) * spacing).astype(np.float32)
    v = rng.normal(0, 0.5, x.shape).astype(np.float32)
    s = (rng.uniform(0.1, 0.9, (solids, 3)) * domain).astype(np.float32)
    g, o = phys_params(reference_params(*domain, 0.5, scale)), phys_params(orc.reference_params(*domain, 0.5, scale))
    for p in (g, o):
        p.kernel_factor, p.s_corr_n, p.s_corr_dq = factor, exponent, 0.3
    o.jacobi = 1
    sim = PbfSim(g, n, solids)
    sim.upload(x, v, s if solids else None)
    sim.step(0.01)
    ref = orc.compat_step(o, 0.01, x, v, solid=s, cap=512)
    cnt, idx = sim.neighbors(cap=512)
    assert np.array_equal(cnt, ref["nbr_count"])
    assert all(np.array_equal(idx[k, :cnt[k]], ref["nbr_idx"][k, :cnt[k]]) for k in range(n))
    gx, gv, lam, _ = sim.download(lambdas=True)
    assert sim.status() == 0
    sim.close()
    assert np.array_equal(lam, ref["lambdas"][:n])
    assert np.abs(gx - ref["x"]).max() <= REL * np.abs(ref["x"]).max()
    assert np.abs(gv - ref["v"]).max() <= REL * np.abs(ref["x"]).max() / 0.01
