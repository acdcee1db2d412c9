"""Hashed grids of the smallest table (1,024 buckets), where the lines of cells
share buckets and run over the table's end: clumps in a wide box, and in a box
longer than the table, against the dense grid of the same scene.  The first
step visits the same particles in the same order, so it agrees bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solids", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("domain", [(48, 40, 56), (6, 6, 3000)])
def test_small_table(domain, precision, solids):
    from lustrine_gb300 import PbfSim, pbf_params
    from lustrine_gb300._lib import GRID_DENSE, GRID_HASHED
    for seed in range(12):
        rng = np.random.default_rng(seed)
        at = np.asarray(domain) * 0.9
        c = rng.uniform(0.05, 1.0, (10, 3)) * at
        x = (c[:, None] + rng.uniform(-1.3, 1.3, (10, 19 + seed % 2, 3))).reshape(-1, 3)
        x = np.clip(x, 0.6, np.asarray(domain) - 0.6).astype(np.float32)
        s = np.floor(rng.uniform(-1.3, 1.3, (50, 3)) + c[rng.integers(0, 10, 50)]) + 0.5
        s = np.clip(s, 0.5, np.asarray(domain) - 0.5).astype(np.float32) if solids else np.zeros((0, 3), np.float32)
        got = []
        for grid in (GRID_DENSE, GRID_HASHED):
            p = pbf_params(*domain, iterations=2, precision=precision, grid_mode=grid, max_neighbors=64)
            with PbfSim(p, len(x), len(s)) as sim:
                sim.upload(x, None, s if solids else None)
                sim.step(1 / 60)
                assert sim.status() == 0
                got.append(sim.download(lambdas=True, density=True) + sim.neighbors(cap=64))
        dense, hashed = got
        assert dense[4].max() > 4
        for a, b in zip(dense, hashed):
            np.testing.assert_array_equal(a, b)
