"""The scan's per-tile totals counted by the predictions: blocks whose keys lie
in one tile of 4,096 cells, in two, in many, and blocks that are not full.
Wrong totals shift whole tiles of the cell table, so the neighbour counts of
every step are compared with brute force over its predicted positions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("n,box,order", [(1, (40, 40, 40), "random"), (33, (8, 8, 8), "sorted"),
                                         (255, (40, 40, 40), "random"), (257, (40, 40, 40), "sorted"),
                                         (1025, (64, 17, 30), "random"), (4000, (40, 40, 40), "sorted")])
def test_neighbour_counts_along_steps(n, box, order, precision):
    from lustrine_gb300 import PRECISION_FP32, PRECISION_MIXED, PbfSim, pbf_params
    rng = np.random.default_rng(n)
    x = (rng.uniform(0.5, 1.0, (n, 3)) * (np.asarray(box) - 1.0)).astype(np.float32)
    if order == "sorted":
        c = np.floor(x).astype(int)
        x = x[np.lexsort((c[:, 2], c[:, 0], c[:, 1]))]
    v = rng.normal(0, 20.0, x.shape).astype(np.float32)  # particles change cells and tiles every step
    dt, g = np.float32(1.0 / 60.0), np.float32(-9.81)
    p = pbf_params(*box, iterations=1, precision=PRECISION_MIXED if precision == "mixed" else PRECISION_FP32)
    hi = np.asarray(box, np.float64) - 0.5
    with PbfSim(p, n) as sim:
        sim.upload(x, v)
        for _ in range(3):
            x0, v0, _, _ = sim.download()
            sim.step(float(dt))
            cnt, _ = sim.neighbors()
            v0 = v0.astype(np.float64)
            v0[:, 1] += float(g) * float(dt)
            pred = np.clip(x0 + v0 * float(dt), 0.5, hi)
            d2 = ((pred[:, None, :] - pred[None, :, :]) ** 2).sum(-1)
            near = np.abs(d2 - 1.0) < 1e-4  # pairs that rounding decides
            assert (cnt >= (d2 <= 1.0 - 1e-4).sum(1)).all() and (cnt <= (d2 <= 1.0).sum(1) + near.sum(1)).all()
        assert sim.status() == 0
