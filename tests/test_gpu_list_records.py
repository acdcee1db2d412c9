"""Wide compact records of 24-bit slots (contexts below 2^24 particles) and of
32-bit ones (a context reserved for more) against the column lists: lists that
end in the first record, in the second, in its last entry and in the overflow
rows, cut at a capacity, with every number of gathers in flight; and column
lists with static particles, which only warps that have some among their
entries test for, against two particles per thread (which test always) and
brute force.  Everything bit for bit but the brute-force counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _block(spacing, n, seed):
    """n particles of a jittered lattice in a box that takes the dense grid."""
    rng = np.random.default_rng(seed)
    a = int(np.ceil(n ** (1 / 3)))
    i = np.arange(n)
    x = np.stack([i // a % a, i // (a * a), i % a], 1) * spacing + 1.0
    return (x + rng.uniform(-0.2, 0.2, x.shape) * spacing).astype(np.float32), int(np.ceil(a * spacing)) + 3


def _run(x, box, lists, unroll=2, reserve=0, cap=64, steps=2):
    from lustrine_gb300 import PbfSim, pbf_params
    sim = PbfSim(pbf_params(box, box, box, iterations=3, max_neighbors=cap), len(x))
    if reserve:
        sim.reserve(reserve)
    sim.upload(x)
    sim.set_tuning(128, unroll, 128, unroll, 1, list_format=lists)
    sim.step(1 / 60, steps)
    out = (*sim.download(lambdas=True, density=True), *sim.neighbors(cap=cap + 1))
    res = out, sim.list_format(), sim.status()
    sim.close()
    return res


@pytest.mark.parametrize("spacing,cap", [(1.0, 64), (0.8, 64), (0.6, 64), (0.7, 4), (0.7, 5), (0.6, 10), (0.6, 13)])
@pytest.mark.parametrize("reserve", [0, (1 << 24) + 5])
def test_wide_records_equal_column_lists(spacing, cap, reserve):
    from lustrine_gb300 import LISTS_COLUMN, LISTS_COMPACT
    x, box = _block(spacing, 66_001, 7)
    want, fmt, status = _run(x, box, LISTS_COLUMN, cap=cap)
    assert fmt == "column"
    for unroll in ((1, 2, 4, 8) if not reserve else (2,)):
        got, fmt, st = _run(x, box, LISTS_COMPACT, unroll, reserve, cap)
        assert fmt == "compact_wide" and st == status
        for a, b in zip(want, got):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("n,solids,spacing,cap", [(33, 3, 1.0, 64), (700, 40, 0.9, 64), (2000, 900, 0.9, 64),
                                                  (2000, 900, 0.7, 6), (129, 0, 0.9, 64)])
def test_column_lists_with_static_particles(n, solids, spacing, cap, precision):
    from lustrine_gb300 import LISTS_COLUMN, PbfSim, pbf_params
    x, box = _block(spacing, n, 11)
    rng = np.random.default_rng(12)
    s = rng.uniform(0.6, box - 0.6, (solids, 3)).astype(np.float32)
    res = []
    # the scene frame has one particle per thread only
    for unroll, ppt in ((1, 1), (2, 1), (4, 1), (8, 1)) + (((2, 2),) if precision < 2 else ()):
        with PbfSim(pbf_params(box, box, box, iterations=3, precision=precision, max_neighbors=cap), n, solids) as sim:
            sim.upload(x, None, s if solids else None)
            sim.set_tuning(128, unroll, 128, unroll, ppt, list_format=LISTS_COLUMN)
            sim.step(1 / 60, 2)
            res.append((*sim.download(lambdas=True, density=True), *sim.neighbors(cap=cap + 1)))
    for r in res[1:]:
        for a, b in zip(res[0], r):
            np.testing.assert_array_equal(a, b)
    # the first step's lists hold every pair the predicted positions put in reach
    with PbfSim(pbf_params(box, box, box, iterations=3, precision=precision, max_neighbors=64), n, solids) as sim:
        sim.upload(x, None, s if solids else None)
        sim.step(1 / 60)
        cnt, idx = sim.neighbors()
    pred = np.clip(x.astype(np.float64) + [0, -9.81 / 3600, 0], 0.5, box - 0.5)
    both = np.concatenate([pred, s.astype(np.float64)])
    d2 = ((pred[:, None, :] - both[None, :, :]) ** 2).sum(-1)
    near = (np.abs(d2 - 1.0) < 1e-4).sum(1)
    assert (np.abs(cnt - (d2 <= 1.0).sum(1)) <= near).all()
    for k in range(n):
        assert (d2[k, idx[k, :cnt[k]]] <= 1.0 + 1e-4).all() and len(set(idx[k, :cnt[k]])) == cnt[k]
