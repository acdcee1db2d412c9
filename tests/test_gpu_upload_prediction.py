"""upload_state_async from page-locked buffers predicts the next step for the
last step's dt.  Whatever comes between the upload and the step (nothing,
another upload, another dt, other parameters, a profiled step, the end of the
context's tuning), the step gives the bits of a context that was just created
with that state, and what reads the state before the step sees it as uploaded."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def _pinned(a):
    import torch
    t = torch.empty(a.shape, dtype=torch.float32, pin_memory=True)
    t.numpy()[...] = a
    return t


def _states(rng, counts):
    out = []
    for n in counts:
        a = int(np.ceil(n ** (1 / 3)))
        i = np.arange(n)
        x = np.stack([i // a % a, i // (a * a), i % a], 1) * 0.9 + 1.0 + rng.uniform(-0.1, 0.1, (n, 3))
        out.append(x.astype(np.float32))
    return out


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("counts", [(1,), (1025,), (700, 33, 1200)])
@pytest.mark.parametrize("between", ["nothing", "upload", "dt", "params", "profile", "tuning", "no_velocity"])
def test_step_after_upload_equals_a_fresh_context(counts, precision, between):
    from lustrine_gb300 import PbfSim, pbf_params
    rng = np.random.default_rng(sum(counts) + precision)
    x = np.concatenate(_states(rng, counts))
    v = rng.normal(0, 1, x.shape).astype(np.float32)
    y, u = (x + rng.uniform(-0.2, 0.2, x.shape)).astype(np.float32), rng.normal(0, 1, x.shape).astype(np.float32)
    boxes = [(16, 15, 17)] * len(counts)

    def make(**kw):
        p = pbf_params(16, 15, 17, iterations=2, precision=precision, **kw)
        return PbfSim.batch(p, boxes, counts) if len(counts) > 1 else PbfSim(p, len(x)), p

    dt = DT / 2 if between == "dt" else DT
    xsph = 0.05 if between == "params" else 0.01
    vel = None if between == "no_velocity" else u
    fresh, _ = make(c_xsph=xsph)
    fresh.upload(y, vel)
    fresh.step(dt, 2)
    want = fresh.download(lambdas=True, density=True)
    fresh.close()

    sim, p = make()
    sim.upload(x, v)
    sim.step(DT, 3)  # a dt is known from here on
    py, pu = _pinned(y), _pinned(u)
    if between == "upload":
        px, pv = _pinned(x), _pinned(v)
        sim.upload_state_async(px.data_ptr(), pv.data_ptr())
    sim.upload_state_async(py.data_ptr(), None if vel is None else pu.data_ptr())
    gx, gv, _, _ = sim.download()  # the state as uploaded (mixed: up to its rounding)
    assert np.abs(gx - y).max() <= 2e-6 and np.array_equal(gv, np.zeros_like(u) if vel is None else u)
    if between == "params":
        p.c_xsph = xsph
        sim.set_params(p)
    if between == "tuning":
        sim.set_tuning(256, 1, 64, 1)
    if between == "profile":
        sim.profile_step(DT)
        sim.step(dt)
    else:
        sim.step(dt, 2)
    got = sim.download(lambdas=True, density=True)
    assert sim.status() == 0
    sim.close()
    for a, b in zip(want, got):
        np.testing.assert_array_equal(a, b)
