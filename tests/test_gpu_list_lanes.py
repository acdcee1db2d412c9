"""List builds by four lanes a particle (a list block of 256 up to a size, which
the default shape takes there) against one lane (a list block of 64), the same
context otherwise: lists, lambdas, densities and states bit for bit.  fp32 and
the scene frame, compact and column lists, with and without static particles, sizes
at the lines and block remainders, lists past a lane's part, past the staged
entries and past the capacity."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spacing,cap", [(1, 1.0, 64), (63, 0.5, 96), (11_000, 0.9, 64), (11_001, 0.9, 64),
                                           (20_000, 0.8, 64), (333, 0.5, 9), (1_111, 0.3, 250), (1_111, 0.3, 61)])
@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("lists", ["compact", "column", "solids"])
def test_four_lanes_give_the_bits_of_one(lists, precision, n, spacing, cap):
    from lustrine_gb300 import PbfSim, pbf_params
    rng = np.random.default_rng(n)
    a = int(np.ceil(n ** (1 / 3)))
    i = np.arange(n)
    x = np.stack([i // a % a, i // (a * a), i % a], 1) * spacing + 2.0
    x = (x + rng.uniform(-0.3, 0.3, x.shape) * spacing).astype(np.float32)
    side = int(np.ceil(a * spacing)) + 5
    s = np.unique(rng.integers(1, side - 1, (max(n // 20, 40), 3)), axis=0).astype(np.float32) + 0.5
    s = s if lists == "solids" else None
    got = []
    for list_block in (64, 256, None):
        p = pbf_params(side, side, side, iterations=2, precision=precision, max_neighbors=cap)
        with PbfSim(p, n, 0 if s is None else len(s)) as sim:
            if list_block:
                sim.set_tuning(128, 2, list_block, 4, list_format=int(lists != "column"))
            sim.upload(x, None, s)
            for _ in range(2):
                sim.step(1 / 60)
                got.append(sim.download(lambdas=True, density=True) + sim.neighbors(cap=cap + 1) + (sim.status(),))  # + itself
            if list_block:
                assert sim.list_format() == ("compact" if lists == "compact" else "column")
    if cap in (9, 61):
        assert got[0][6] == 4
    if spacing == 0.3 and cap == 250:
        assert got[0][4].max() > 49
    for other in (2, 4):
        for step in range(2):
            for u, w in zip(got[step], got[other + step]):
                np.testing.assert_array_equal(u, w)
