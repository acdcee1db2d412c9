"""A context whose launch shape was not set takes one by list format and size:
the bits of an explicitly set shape, on both sides of the sizes where the rule
changes; get_tuning reports the library's default until one is set."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ONE_WAVE = 152 * 9 * 128


@pytest.mark.parametrize("n,precision,solids", [(300, 0, 0), (300, 0, 50), (300, 1, 50), (300, 2, 0),
                                                (ONE_WAVE, 1, 0), (ONE_WAVE + 1, 1, 0), (ONE_WAVE + 1, 0, 5),
                                                (250_000, 0, 0), (250_001, 0, 0)])
def test_default_shape_gives_the_bits_of_a_set_one(n, precision, solids):
    from lustrine_gb300 import PbfSim, pbf_params
    rng = np.random.default_rng(n + solids)
    a = int(np.ceil(n ** (1 / 3)))
    i = np.arange(n)
    x = (np.stack([i // a % a, i // (a * a), i % a], 1) + 1.0 + rng.uniform(-0.1, 0.1, (n, 3))).astype(np.float32)
    s = rng.uniform(1, a, (solids, 3)).astype(np.float32)
    res = []
    for set_shape in (False, True):
        with PbfSim(pbf_params(a + 3, a + 3, a + 3, iterations=2, precision=precision), n, solids) as sim:
            sim.upload(x, None, s if solids else None)
            if set_shape:
                sim.set_tuning(128, 2, 128, 8)
            t = sim.get_tuning()
            assert (t["block"], t["unroll"], t["list_block"], t["xsph_unroll"]) == (128, 2, 128, 8)
            sim.step(1 / 60, 2)
            assert sim.status() == 0
            res.append(sim.download(lambdas=True, density=True))
    for u, w in zip(*res):
        np.testing.assert_array_equal(u, w)
