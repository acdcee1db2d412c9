"""The work a program has this library do, as measurable cases.

A case is one pass through the public entry points:

  rollout  from a state the program holds in page-locked memory: upload,
           `steps` steps, download of positions and velocities, wait (a
           simulation advanced between two reads of its state; steps = 1 is
           one frame of a game);
  frames   `steps` frames of a host that owns the particle arrays: each frame
           is one step_host call on them (upload, step, download, wait);
  sort     one counting sort of device keys.

The three step semantics (the PBF step in its three position
representations, the reference's fluid step, the sand step), one scene or a
batch, boundary voxels, dense and hashed grids and ragged sizes are fields of
the case.  `spacing` and `jitter` set the state: 1.0 / 0.05 is the lattice the
dam breaks start from (about 4 neighbours a particle), smaller spacings with
larger jitter what they are in after some fifty steps (6-8 neighbours).
"""
import math

import numpy as np
import torch

import lustrine_gb300 as L
from lustrine_gb300.sorting import counting_sort

F32 = np.float32


def _case(name, entry="rollout", mode="pbf", n=0, scenes=1, smallest=0, largest=0, spacing=1.0, jitter=0.05,
          solids=False, blobs=0, precision="fp32", iterations=4, steps=1, hz=60, kernel_scale=2.0, tuned=False,
          cells=0, shuffled=False):
    c = dict(name=name, entry=entry, mode=mode, n=n, scenes=scenes, smallest=smallest, largest=largest,
             spacing=spacing, jitter=jitter, solids=solids, blobs=blobs, precision=precision, iterations=iterations,
             steps=steps, hz=hz, kernel_scale=kernel_scale, tuned=tuned, cells=cells, shuffled=shuffled)
    if name is None:
        del c["name"]
    return c


def listed():
    return [
        # one frame of the 10,000-particle dam break: launches and latency count
        _case("pbf_frame_10k", n=10_000),
        # a game host that owns the arrays: frames of a ragged block lying on voxel terrain
        _case("pbf_host_frames_solids_77k", entry="frames", n=77_777, solids=True, spacing=0.85, jitter=0.15, steps=4),
        # the 64^3 block with some 50k boundary voxels, mid-run
        _case("pbf_solids_262k", n=262_144, solids=True, spacing=0.85, jitter=0.15, steps=4),
        # cell-relative positions with boundary voxels, ragged
        _case("pbf_mixed_solids_150k", n=150_001, solids=True, precision="mixed", spacing=0.9, jitter=0.12, steps=4),
        # the large dam break, 6 iterations
        _case("pbf_2m", n=2_097_152, iterations=6, hz=120, steps=6),
        # 16 blobs far apart in a 4096 x 256 x 4096 box: hashed grid, cell-relative positions, 8 iterations
        _case("pbf_hashed_mixed_4m", n=4_194_304, blobs=16, precision="mixed", iterations=8, steps=6),
        # 512 independent scenes of 1,024 to 65,536 particles, the benchmark's launch shape
        _case("batch_512_scene_frame", scenes=512, smallest=1024, largest=65_536, precision="scene", tuned=True,
              steps=6),
        # a few dozen small scenes, mid-run, the library's default shape
        _case("batch_37_fp32", scenes=37, smallest=500, largest=20_000, spacing=0.85, jitter=0.15, steps=4),
        # the wrapper's default step: sand on voxel terrain, init_simulation's kernel radius
        _case("sand_solids_262k", mode="sand", n=262_144, solids=True, spacing=0.98, jitter=0.1, kernel_scale=3.1,
              steps=8),
        # one frame of a small sand heap
        _case("sand_frame_20k", mode="sand", n=20_011, solids=True, spacing=0.98, jitter=0.1),
        # the reference's own fluid step (long lists: kernel radius 3.1 r)
        _case("reference_fluid_100k", mode="reference", n=100_000, spacing=1.0, jitter=0.1, kernel_scale=3.1,
              hz=100, steps=2),
        # the counting sort by itself: cell keys of a million particles
        _case("sort_1m", entry="sort", mode="sort", n=1_000_003, cells=1_250_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pbf", "pbf", "pbf", "solids", "solids", "hashed", "batch", "batch", "sand", "sand",
                       "reference", "sort"])
    spacing = round(rng.uniform(0.82, 1.0), 3)
    state = dict(spacing=spacing, jitter=round(0.05 + (1.0 - spacing) * 0.6, 3))
    steps = rng.choice([1, 2, 3, 4, 6, 8] if spacing > 0.96 else [1, 2, 3, 4])
    if kind == "pbf":
        return _case(None, n=_log_int(rng, 2_000, 2_000_000), precision=rng.choice(["fp32", "fp32", "scene", "mixed"]),
                     iterations=rng.randint(2, 6), steps=steps, **state)
    if kind == "solids":
        return _case(None, entry=rng.choice(["rollout", "frames"]), n=_log_int(rng, 5_000, 500_000), solids=True,
                     precision=rng.choice(["fp32", "fp32", "mixed", "scene"]), iterations=rng.randint(2, 6),
                     steps=steps, **state)
    if kind == "hashed":
        return _case(None, n=_log_int(rng, 100_000, 3_000_000), blobs=16, precision=rng.choice(["fp32", "mixed"]),
                     iterations=rng.randint(4, 8), steps=min(steps, 4), **state)
    if kind == "batch":
        return _case(None, scenes=_log_int(rng, 8, 300), smallest=rng.randint(300, 2_000),
                     largest=rng.randint(8_000, 65_536), precision=rng.choice(["fp32", "scene"]),
                     tuned=rng.random() < 0.5, steps=steps, **state)
    if kind == "sand":
        return _case(None, mode="sand", n=_log_int(rng, 5_000, 400_000), solids=rng.random() < 0.7,
                     spacing=round(rng.uniform(0.95, 1.0), 3), jitter=0.1, kernel_scale=rng.choice([2.0, 3.1]),
                     steps=steps)
    if kind == "reference":
        return _case(None, mode="reference", n=_log_int(rng, 5_000, 250_000), solids=rng.random() < 0.5,
                     spacing=1.0, jitter=round(rng.uniform(0.05, 0.12), 3), kernel_scale=rng.choice([2.0, 3.1]),
                     hz=100, steps=min(steps, 2))
    n = _log_int(rng, 10_000, 3_000_000)
    return _case(None, entry="sort", mode="sort", n=n, cells=int(n * rng.uniform(0.5, 5.0)), shuffled=rng.random() < 0.5)


# ------------------------------------------------------------------- scenes --

def _counts(case):
    """Particles of every scene (a property of the case, not of the seed)."""
    if case["scenes"] == 1:
        return np.array([case["n"]], np.int64)
    rng = np.random.default_rng(case["scenes"])
    return np.round(np.exp(rng.uniform(math.log(case["smallest"]), math.log(case["largest"]),
                                       case["scenes"]))).astype(np.int64)


def _total(case):
    return int(_counts(case).sum())


TERRAIN = 4  # highest column of the voxel terrain


def _boxes(case):
    if case["blobs"]:
        return [(4096, 256, 4096)]
    out = []
    for n in _counts(case):
        a = math.ceil(round(int(n) ** (1 / 3), 9))
        side = max(8, 2 * a)
        out.append((side, a + 2 + (TERRAIN + 1 if case["solids"] else 0), side))
    return out


def _scene(case, seed):
    """x, v, solid: float32 cuda tensors (n, 3), (n, 3), (ns, 3)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    dev, s = "cuda", case["spacing"]
    counts = torch.as_tensor(_counts(case), device=dev)
    n = int(counts.sum())
    if case["blobs"]:  # a block per blob, the last ones one particle smaller
        b = case["blobs"]
        counts = torch.tensor([n // b + (k < n % b) for k in range(b)], device=dev)
    side = torch.as_tensor([math.ceil(round(int(c) ** (1 / 3), 9)) for c in counts.tolist()], device=dev)
    block = torch.repeat_interleave(torch.arange(len(counts), device=dev), counts)
    m = torch.arange(n, device=dev) - (torch.cumsum(counts, 0) - counts)[block]
    a = side[block]
    site = torch.stack([(m // a) % a, m // (a * a), m % a], 1)  # filled layer by layer from the floor
    x = (site.float() + 0.5) * s + (torch.rand((n, 3), generator=g, device=dev) * 2 - 1) * case["jitter"]
    solid = torch.zeros((0, 3), device=dev)
    if case["solids"]:
        w = _boxes(case)[0][0]
        ph = torch.rand(6, generator=g, device=dev) * (2 * math.pi)
        u = torch.arange(w, device=dev).float()
        hx = torch.sin(u * 0.21 + ph[0]) + torch.sin(u * 0.07 + ph[1]) + torch.sin(u * 0.5 + ph[2])
        hz = torch.sin(u * 0.19 + ph[3]) + torch.sin(u * 0.08 + ph[4]) + torch.sin(u * 0.45 + ph[5])
        h = (1 + (TERRAIN - 1) * (hx[:, None] + hz[None, :] + 6) / 12).round().long()
        col = torch.arange(w * w, device=dev)
        col = torch.repeat_interleave(col, h.reshape(-1))
        first = torch.cumsum(h.reshape(-1), 0) - h.reshape(-1)
        y = torch.arange(len(col), device=dev) - first[col]
        solid = torch.stack([col // w, y, col % w], 1).float() + 0.5
        foot = (site[:, ::2].float() * s).long().clamp(max=w - 1)
        x[:, 1] += h[foot[:, 0], foot[:, 1]].float()
    if case["blobs"]:
        k = torch.arange(case["blobs"], device=dev)
        at = torch.rand((case["blobs"], 3), generator=g, device=dev)
        x += torch.stack([80 + 1000.0 * (k % 4) + 800 * at[:, 0], 4 + 150 * at[:, 1],
                          80 + 1000.0 * (k // 4) + 800 * at[:, 2]], 1)[block]
    else:
        box = torch.as_tensor(_boxes(case), device=dev).float()
        x = torch.minimum(x.clamp(min=0.5), box[block if case["scenes"] > 1 else torch.zeros_like(block)] - 0.5)
    v = torch.randn((n, 3), generator=g, device=dev) * 0.5
    return x.contiguous(), v.contiguous(), solid.contiguous()


def _params(case):
    box = _boxes(case)[0]
    if case["mode"] == "reference":
        return L.reference_params(*box, kernel_radius_scale=case["kernel_scale"])
    if case["mode"] == "sand":
        return L.sand_params(*box, kernel_radius_scale=case["kernel_scale"])
    return L.pbf_params(*box, iterations=case["iterations"],
                        precision={"fp32": L.PRECISION_FP32, "mixed": L.PRECISION_MIXED,
                                   "scene": L.PRECISION_MIXED_SCENE}[case["precision"]])


# --------------------------------------------------------------------- pass --

def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def _keys(case, seed):
    """Cell keys of particles that lie in cell order but for what they moved in the last step."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    at = torch.rand(case["n"], generator=g, device="cuda", dtype=torch.float64) * case["cells"]
    if not case["shuffled"]:
        at = at.sort().values + torch.randn(case["n"], generator=g, device="cuda", dtype=torch.float64)
    return at.floor().clamp(0, case["cells"] - 1).int()


def prepare(case, seed):
    if case["entry"] == "sort":
        return dict(case=case, keys=_keys(case, seed),
                    counts=torch.empty(case["cells"] + 1, dtype=torch.int32, device="cuda"),
                    order=torch.empty(case["n"], dtype=torch.int32, device="cuda"))
    x, v, solid = _scene(case, seed)
    p = _params(case)
    if case["scenes"] > 1:
        sim = L.PbfSim.batch(p, _boxes(case), _counts(case))
    else:
        sim = L.PbfSim(p, len(x), len(solid))
    if case["tuned"]:
        sim.set_tuning(256, 1, 128, 1)
    torch.cuda.synchronize()
    sim.upload_device(x.data_ptr(), v.data_ptr(), solid.data_ptr() if len(solid) else None)
    return dict(case=case, sim=sim, dt=1.0 / case["hz"], x0=_pinned(x), v0=_pinned(v),
                x=torch.empty(x.shape, pin_memory=True), v=torch.empty(v.shape, pin_memory=True))


def run(state):
    case = state["case"]
    if case["entry"] == "sort":
        counting_sort(state["counts"], state["keys"], case["cells"], state["order"])
        return {"counts": state["counts"], "order": state["order"]}
    sim, x, v = state["sim"], state["x"], state["v"]
    if case["entry"] == "frames":
        x.copy_(state["x0"])
        v.copy_(state["v0"])
        for _ in range(case["steps"]):
            sim.step_host(state["dt"], x.data_ptr(), v.data_ptr())
        return {"x": x, "v": v}
    sim.upload_state_async(state["x0"].data_ptr(), state["v0"].data_ptr())
    sim.step(state["dt"], case["steps"])
    sim.download_state_async(x.data_ptr(), v.data_ptr())
    sim.synchronize()
    return {"x": x, "v": v}


def _neighbours(case):
    """Pairs a particle takes part in, about: the number density times the kernel's ball."""
    h = 1.0 if case["mode"] == "pbf" else case["kernel_scale"] * 0.5
    return 4.19 * (h / case["spacing"]) ** 3


def work(case):
    n, steps = _total(case), case["steps"]
    if case["entry"] == "sort":
        return {"bytes": 4 * (2 * n + case["cells"] + 1), "flops": 0}
    nb = _neighbours(case)
    # per step: x, v in and out; per pass over the neighbours: positions (and
    # lambdas) in, what it computes out
    if case["mode"] == "sand":
        return {"bytes": n * steps * (48 + 4 * 24), "flops": n * nb * steps * 4 * 60}
    iters = case["iterations"] if case["mode"] == "pbf" else 1
    return {"bytes": n * steps * (48 + iters * 44), "flops": n * nb * steps * iters * 60}


# -------------------------------------------------------------- in 64 bits --

class _Pairs:
    """Pairs (i, j) within h of each other, i fluid, j fluid (index < n) or a
    static particle (n + its index), in the order cell by cell (y, x, z
    outermost first), fluid before static particles, by index in a cell."""

    def __init__(self, x, solid, cell_of, cell_of_solid, grid, group, h):
        n, dev = len(x), x.device
        gx, gy, gz = grid
        key = lambda c, s: ((s * gy + c[:, 1]) * gx + c[:, 0]) * gz + c[:, 2]  # noqa: E731
        tables = [(x, key(cell_of, group), 0)]
        if len(solid):
            tables.append((solid, key(cell_of_solid, torch.zeros_like(cell_of_solid[:, 0])), n))
        tables = [(q, *torch.sort(k, stable=True), off) for q, k, off in tables]
        ii, jj = [], []
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                for dz in (-1, 0, 1):
                    c = cell_of + torch.tensor([dx, dy, dz], device=dev)
                    inside = ((c >= 0) & (c < torch.tensor([gx, gy, gz], device=dev))).all(1).nonzero()[:, 0]
                    k = key(c[inside], group[inside])
                    for q, sorted_k, perm, off in tables:
                        a = torch.searchsorted(sorted_k, k)
                        m = torch.searchsorted(sorted_k, k, right=True) - a
                        i = torch.repeat_interleave(inside, m)
                        t = torch.arange(len(i), device=dev) - torch.repeat_interleave(torch.cumsum(m, 0) - m - a, m)
                        j = perm[t]
                        near = ((x[i] - q[j]) ** 2).sum(1) <= h * h
                        ii.append(i[near])
                        jj.append(j[near] + off)
        self.i, self.j, self.n = torch.cat(ii), torch.cat(jj), n
        order = torch.sort(self.i, stable=True).indices
        self.i, self.j = self.i[order], self.j[order]

    def sum(self, value):
        out = torch.zeros((self.n,) + value.shape[1:], dtype=value.dtype, device=value.device)
        return out.index_add_(0, self.i, value)


def _box_tensors(case, group):
    return torch.as_tensor(_boxes(case), device="cuda").double()[group]


def _exact_pbf(case, x, v, solid):
    h, rho0, r, dt, g = 1.0, 1.0, 0.5, float(F32(1.0 / case["hz"])), float(F32(-9.81))
    m = float(F32(64 * math.pi / 315))
    eps, sk, dq, cx, contact = 10.0, float(F32(0.1)), float(F32(0.2)), float(F32(0.01)), 1.0
    k6, ks = 315 / (64 * math.pi), 45 / math.pi
    n = len(x)
    counts = torch.as_tensor(_counts(case), device="cuda")
    group = torch.repeat_interleave(torch.arange(len(counts), device="cuda"), counts)
    box = _box_tensors(case, group)
    grid = [int(max(b[a] for b in _boxes(case))) + 1 for a in range(3)]
    for _ in range(case["steps"]):
        pv = v.clone()
        pv[:, 1] += g * dt
        xs = torch.minimum((x + pv * dt).clamp(min=r), box - r)
        P = _Pairs(xs, solid, xs.floor().long(), solid.floor().long(), grid, group, h)
        keep = P.i != P.j
        P.i, P.j = P.i[keep], P.j[keep]
        sol = P.j >= n
        for _ in range(case["iterations"]):
            allx = torch.cat([xs, solid])
            d = xs[P.i] - allx[P.j]
            r2 = (d * d).sum(1)
            rr = r2.sqrt()
            hd = (h * h - r2).clamp(min=0)
            gr = torch.where((rr > 0)[:, None], (-ks * (h - rr).clamp(min=0) ** 2 / rr.clamp(min=1e-300))[:, None] * d,
                             torch.zeros_like(d)) * (m / rho0)
            rho = m * k6 + P.sum(m * k6 * hd ** 3)
            gi = P.sum(gr)
            S = P.sum(torch.where(sol, torch.zeros_like(r2), (gr * gr).sum(1))) + (gi * gi).sum(1)
            lam = -(rho / rho0 - 1) / (S + eps)
            lj = torch.where(sol, lam[P.i], lam[P.j.clamp(max=n - 1)])
            sc = -sk * (hd / (h * h - dq * dq)) ** 12
            dp = P.sum((lam[P.i] + lj + sc)[:, None] * gr)
            if len(solid):
                hit = sol & (rr < contact) & (rr > 0)
                push = P.sum(torch.where(hit[:, None], ((contact - rr) / rr.clamp(min=1e-300))[:, None] * d,
                                         torch.zeros_like(d)))
                dp = dp + push / P.sum(hit.double()).clamp(min=1)[:, None]
            xs = torch.minimum((xs + dp).clamp(min=r), box - r)
        nv = (xs - x) / dt
        fl = ~sol
        i, j = P.i[fl], P.j[fl]
        w = k6 * (h * h - ((xs[i] - xs[j]) ** 2).sum(1)).clamp(min=0) ** 3
        x, v = xs, nv + cx * torch.zeros_like(nv).index_add_(0, i, (nv[j] - nv[i]) * w[:, None])
    return x, v


def _cells_truncated(a, cell, grid):
    """The reference's cell of fp32 positions: truncating fp32 division, clamped."""
    c = torch.from_numpy((a.cpu().numpy().astype(F32) / F32(cell)).astype(np.int64)).cuda()
    return torch.minimum(c.clamp(min=0), torch.tensor(grid, device="cuda") - 1)


def _exact_reference(case, x, v, solid):
    h, r = float(F32(case["kernel_scale"]) * F32(0.5)), 0.5
    dt = float(F32(min(max(1.0 / case["hz"], 0.001), 0.01)))
    rho0, m, eps, sk, dq = 24.0, 5.0, 10.0, 1.0, 0.5
    ck, cl = 8 / (math.pi * h ** 3), 48 / (math.pi * h ** 3)
    box = torch.tensor(_boxes(case)[0], device="cuda").double()
    grid = [int(b / F32(h)) + 1 for b in _boxes(case)[0]]
    n = len(x)

    def W(rad):
        q = rad * 0.5 / h
        return torch.where(q <= 0.5, ck * (6 * q ** 3 - 6 * q ** 2 + 1),
                           torch.where(q <= 1, ck * 2 * (1 - q) ** 3, torch.zeros_like(q)))

    zero = torch.zeros(1, device="cuda", dtype=torch.float64)
    for _ in range(case["steps"]):
        pv = v.clone()
        pv[:, 1] += -10.0 * m * dt
        xs = x + pv * dt
        P = _Pairs(xs, solid, _cells_truncated(xs, h, grid), _cells_truncated(solid, h, grid), grid,
                   torch.zeros(n, dtype=torch.long, device="cuda"), h)
        d = xs[P.i] - torch.cat([xs, solid])[P.j]
        rr = (d * d).sum(1).sqrt()
        rl = rr * 0.5
        q = rl / h
        c = torch.where(q <= 0.5, cl * q * (3 * q - 2), cl * -(1 - q) ** 2) / (rl * h).clamp(min=1e-300)
        gr = torch.where(((rl > 1e-5) & (q <= 1))[:, None], c[:, None] * d, torch.zeros_like(d))
        rho = P.sum(m * W(rr)) + m * W(zero)
        gj = -(m / rho0) * gr
        gi = P.sum(gj)
        S = P.sum((gj * gj).sum(1)) + (gi * gi).sum(1)
        lam = torch.where(S > 0, -(rho / rho0 - 1) / (S + eps), torch.zeros_like(S))
        # the reference reads the neighbour's lambda at the neighbour's place in the list
        first = torch.searchsorted(P.i, torch.arange(n, device="cuda"))
        place = torch.arange(len(P.i), device="cuda") - first[P.i]
        sc = -sk * (W(rr) / W(zero + dq)) ** 4
        dp = P.sum((lam[P.i] + lam[place] + sc)[:, None] * gr) / rho0
        y = xs + dp
        hi = box - r
        y = torch.where(y <= r, torch.full_like(y, float(F32(0.01))), torch.where(y > hi, hi - float(F32(0.01)), y))
        x, v = y, (y - x) / dt
    return x, v


def _exact_sand(case, x32, v32, solid):
    """One step.  The step re-orders the particles by the cell of their fp32
    prediction; that order is formed in fp32, everything after it in 64 bits."""
    h, r, dia, mass = float(F32(case["kernel_scale"]) * F32(0.5)), 0.5, 1.0, 1.0
    dt32, g32 = F32(1.0 / case["hz"]), F32(-9.81)
    grid = [int(b / F32(h)) + 1 for b in _boxes(case)[0]]
    hi = np.array(_boxes(case)[0], F32) - F32(r)
    xf, vf = x32.cpu().numpy(), v32.cpu().numpy().copy()
    vf[:, 1] = vf[:, 1] + g32 * dt32
    pred = np.minimum(np.maximum(xf + vf * dt32, F32(r)), hi)
    cell = _cells_truncated(torch.from_numpy(pred).cuda(), h, grid)
    order = torch.sort((cell[:, 1] * grid[0] + cell[:, 0]) * grid[2] + cell[:, 2], stable=True).indices
    x, cell = x32.double()[order], cell[order]
    dt, box = float(dt32), torch.tensor(_boxes(case)[0], device="cuda").double()
    v = v32.double()[order]
    v[:, 1] += float(g32) * dt
    s = torch.minimum((x + v * dt).clamp(min=r), box - r)
    P = _Pairs(s, solid, cell, _cells_truncated(solid, h, grid), grid,
               torch.zeros(len(x), dtype=torch.long, device="cuda"), h)
    keep = P.i != P.j
    i, j = P.i[keep], P.j[keep]
    P.i, P.j, n = i, j, len(x)
    grain = (j < n)[:, None]
    for _ in range(4):
        pi, pj = s[i], torch.cat([s, solid])[j]
        d = pi - pj
        ln = d.norm(dim=1, keepdim=True)
        same = (ln == 0).expand_as(d)
        d = torch.where(same, torch.tensor([0, 1e-5, 0], device="cuda", dtype=torch.float64), d)
        ln = d.norm(dim=1, keepdim=True)
        t = torch.where(grain, 0.4, 0.8) * (ln - dia) * d / ln
        a = pi - t
        b = torch.where(grain, pj + t, pj)
        moved = torch.where(grain, b - torch.cat([x, solid])[j], torch.zeros_like(b))
        rel = (a - x[i]) - moved
        nx = a - b
        nx = nx / nx.norm(dim=1, keepdim=True)
        tan = rel - (rel * nx).sum(1, keepdim=True) * nx
        lt, depth = tan.norm(dim=1, keepdim=True) + 1e-9, t.norm(dim=1, keepdim=True)
        ratio = torch.where(depth * float(F32(0.95)) > lt, torch.ones_like(lt),
                            (float(F32(0.9)) * depth / lt).clamp(max=1))
        dp = torch.where(ln > dia, torch.zeros_like(t), -t - float(F32(0.7)) * tan * ratio)
        s = torch.minimum((s + P.sum(dp)).clamp(min=r), box - r)
    return s, (s - x) / dt


def exact(case, seed):
    if case["entry"] == "sort":
        k, order = torch.sort(_keys(case, seed).long(), stable=True)
        counts = torch.searchsorted(k, torch.arange(case["cells"] + 1, device="cuda"))
        return {"counts": counts.int(), "order": order.int()}
    if case["mode"] == "sand" and case["steps"] > 1:
        return None  # the order of the next step's particles turns on fp32 roundings of this one's
    if _total(case) * case["steps"] * (case["iterations"] if case["mode"] == "pbf" else 1) > 250_000_000:
        return None  # over 20 seconds
    x, v, solid = _scene(case, seed)
    f = {"pbf": _exact_pbf, "reference": _exact_reference, "sand": _exact_sand}[case["mode"]]
    if case["mode"] != "sand":
        x, v = x.double(), v.double()
    x, v = f(case, x, v, solid.double())
    return {"x": x, "v": v}
