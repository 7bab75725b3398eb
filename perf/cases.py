"""Performance cases: what users of the library have it do, through the C ABI
(include/sf_capi.h) and its ctypes binding.

Kinds of work:

* ``step``      adaptive substeps (``Simulation.step``, the reference's UpdateSystem) of one scene, with the sub-step
                count read back after each one, as the reference application's loop does;
* ``frame``     the same loop for a host program that couples or renders: velocities in from pinned host memory,
                positions, velocities and colours back to it at every substep;
* ``substeps``  fixed-dt substeps of one scene or of a batch of independent scenes (``Simulation.substeps_fixed``), the
                sizes of a batch given by its layout;
* ``adjoint``   gradient of a trajectory loss (``Simulation.adjoint``) of one scene or of a batch;
* ``cell_sort`` the allocation-free cell sort of positions in device memory (``sf_cell_sort_noalloc``).

Every pass of the simulation kinds starts from the prepared state: creation order, positions, velocities and colours
are put back from device memory, as a calibration or parameter study does between its runs. Scenes are the seeded
generators of ``sph_seepage_flows_gb300.scenes``, with a seeded flow laid over the water and, in some cases, the water
lattice disturbed as in a flowing state.

``exact`` restates the substep in torch float64 (pairs from a cell grid, sums by ``index_add_``), and takes the gradients
by autograd.
"""

from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from sph_seepage_flows_gb300 import capi, params, scenes

DEV = "cuda"
T_FRAME = 1.0 / 30.0
EPS = 1e-6
# state put back before every pass, and results copied out by particle id
RESET = ("pos", "vel", "col", "max_saturation")
RESULTS = ("pos", "vel", "acc", "density", "pressure", "voidage", "saturation", "max_saturation")


# ----------------------------------------------------------------- the cases
def listed():
    return [
        # smallest call: one substep of a test-sized scene, bound by latency and launches
        dict(name="step_tiny", kind="step", geometry="block", n_sand=800, n_water=960, pitch=0.02, substeps=1,
             flow=0.2, disorder=0.01, multi=True, wcsph=True),
        # the same loop on the reference application's scale, single-sand-type coupling and the linear equation of state
        dict(name="step_sph_7k", kind="step", geometry="embankment", n_sand=3511, n_water=3677, pitch=0.02, substeps=4,
             flow=0.2, disorder=0.05, multi=False, wcsph=False),
        # the plain-small workload of the benchmark (8,000 sand + 32,000 water), adaptive substeps
        dict(name="step_40k", kind="step", geometry="plain_small", n_sand=8000, n_water=32000, pitch=0.02, substeps=8,
             flow=0.3, disorder=0.01, multi=True, wcsph=True),
        # a coupled host program: velocities in, positions, velocities and colours out through pinned memory, every substep
        dict(name="frame_120k", kind="frame", geometry="embankment", n_sand=60000, n_water=60000, pitch=0.02, substeps=4,
             flow=0.3, disorder=0.05, multi=True, wcsph=True),
        # the adjoint workload's column (10k sand over a flooded base: interpenetrating lattices, long lists), forward
        dict(name="column_20k", kind="substeps", geometry="column", n_sand=10240, n_water=10000, pitch=0.02, scenes=1,
             substeps=16, flow=0.2, disorder=0.01, multi=True, wcsph=True),
        # an odd middle size, single sand type, disturbed water
        dict(name="embankment_251k", kind="substeps", geometry="embankment", n_sand=120037, n_water=131009, pitch=0.02,
             scenes=1, substeps=8, flow=0.3, disorder=0.1, multi=False, wcsph=True),
        # the benchmark's headline: 500k sand embankment + 500k water reservoir
        dict(name="plain_large_1M", kind="substeps", geometry="plain_large", n_sand=500000, n_water=500000, pitch=0.01,
             scenes=1, substeps=8, flow=0.2, disorder=0.01, multi=True, wcsph=True),
        # a breached state of that size: water moving through sand, the lattice lost, long neighbour lists
        dict(name="seepage_800k", kind="substeps", geometry="column", n_sand=400013, n_water=390007, pitch=0.02, scenes=1,
             substeps=4, flow=0.5, disorder=0.15, multi=True, wcsph=True),
        # the ensemble workload: 64 independent scenes of 2k to 60k particles in the same launches
        dict(name="ensemble_64", kind="substeps", geometry="batched", n_sand=2000, n_water=60000, pitch=0.02, scenes=64,
             layout=99, substeps=16, flow=0.2, disorder=0.05, multi=True, wcsph=True),
        # gradient of a trajectory loss on the adjoint workload's column, state gradients returned
        dict(name="adjoint_column_20k", kind="adjoint", geometry="column", n_sand=10240, n_water=10000, pitch=0.02,
             scenes=1, substeps=20, checkpoint=10, flow=0.2, disorder=0.01, state_grads=True),
        # one iteration of the batched calibration: parameter gradients only, several scenes of 10k to 50k particles
        dict(name="calibration_12", kind="adjoint", geometry="calibration", n_sand=10000, n_water=50000, pitch=0.02,
             scenes=12, layout=77, substeps=10, checkpoint=5, flow=0.1, disorder=0.01, state_grads=False),
        # cell sort without allocation, for callers with a device heap of their own
        dict(name="cell_sort_200k", kind="cell_sort", n=200003, cell=0.02, grid_x=96, grid_y=40, grid_z=64, ordered=True),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "frame", "substeps", "substeps", "substeps", "adjoint", "cell_sort"])
    if kind == "cell_sort":
        return dict(kind=kind, n=log_int(500, 262144), cell=rng.choice([0.02, 0.04]), grid_x=rng.randint(20, 130),
                    grid_y=rng.randint(10, 50), grid_z=rng.randint(20, 100), ordered=rng.random() < 0.5)
    common = dict(flow=round(rng.uniform(0.05, 0.5), 3), disorder=round(rng.uniform(0.01, 0.15), 3), pitch=0.02)
    if kind == "adjoint":
        if rng.random() < 0.5:
            return dict(kind=kind, geometry="calibration", n_sand=5000, n_water=log_int(10000, 40000),
                        scenes=rng.randint(2, 12), layout=rng.randint(1, 9999), substeps=rng.randint(4, 10), checkpoint=rng.randint(2, 10),
                        state_grads=False, **common)
        n = log_int(2000, 60000)
        return dict(kind=kind, geometry="column", n_sand=n, n_water=int(n * rng.uniform(0.5, 1.2)), scenes=1,
                    substeps=rng.randint(2, 16), checkpoint=rng.randint(2, 16), state_grads=True, **common)
    common.update(multi=rng.random() < 0.7, wcsph=rng.random() < 0.8)
    if kind == "substeps" and rng.random() < 0.3:
        return dict(kind=kind, geometry="batched", n_sand=2000, n_water=log_int(4000, 50000), scenes=rng.randint(2, 48),
                    layout=rng.randint(1, 9999), substeps=rng.randint(1, 8), **common)
    n = log_int(1500, 150000 if kind == "frame" else 900000)
    frac = rng.uniform(0.3, 0.7)
    k = rng.randint(1, 8 if n > 200000 else 16)
    out = dict(kind=kind, geometry=rng.choice(["block", "column", "embankment"]), n_sand=max(50, int(n * frac)),
               n_water=max(50, int(n * (1 - frac))), substeps=min(k, 8) if kind != "substeps" else k, **common)
    if kind == "substeps":
        out["scenes"] = 1
    return out


# ------------------------------------------------------------------- inputs
def _scenes(case, seed):
    g, ns, nw, pitch = case["geometry"], case["n_sand"], case["n_water"], case["pitch"]
    if g == "batched":
        out = scenes.batched(case["scenes"], case["layout"], ns, nw)
    elif g == "calibration":
        out = scenes.calibration_scenes(case["scenes"], case["layout"], ns, nw)
    elif g == "plain_small":
        out = [scenes.plain_small(seed)]
    elif g == "plain_large":
        out = [scenes.plain_large(seed, ns, nw)]
    elif g == "column":
        out = [scenes.column_scene("column", ns, nw, seed, pitch)]
    elif g == "embankment":
        out = [scenes.embankment_scene("embankment", ns, nw, seed, pitch)]
    else:  # a sand block and a water column that touch, in a box of their size
        s = max(2, round(ns ** (1 / 3)))
        sand = (s, max(2, round(ns / s / s)), s)
        w = max(2, round((nw / 2) ** (1 / 3)))
        water = (w, max(2, round(nw / w / w)), w)
        side = (max(sand[0] + water[0], sand[2], water[2]) + 4) * pitch
        box = (side, (max(sand[1], water[1]) + 4) * pitch, side)
        x0 = box[0] - pitch - (sand[0] - 1) * pitch
        out = [scenes.block_scene("block", tuple(float(np.float32(v)) for v in box), sand, water, pitch, seed,
                                  sand_origin=(x0, pitch, 3 * pitch), water_origin=(x0 - water[0] * pitch, pitch, 3 * pitch))]
    for k, sc in enumerate(out):
        rng = np.random.default_rng([seed, k])
        water = sc.label == params.SF_LABEL_WATER
        p = sc.params
        spacing = 2.0 * p.sph_particle_radius
        lo = np.asarray(sc.bparams.lowest_point[:]) + spacing
        hi = np.asarray(sc.bparams.highest_point[:]) - spacing
        d = case["disorder"] * spacing
        moved = sc.pos[water] + rng.uniform(-d, d, size=(int(water.sum()), 3))
        sc.pos[water] = np.clip(moved, lo, hi).astype(np.float32)
        if "layout" in case:  # sizes and lattice of the layout, positions of the seed
            sc.pos[~water] += rng.uniform(-0.005 * spacing, 0.005 * spacing, size=(sc.n_sand, 3)).astype(np.float32)
        flow = case["flow"]
        sc.vel[:] = (0.05 * flow * rng.standard_normal(sc.vel.shape)).astype(np.float32)
        height = (sc.pos[water, 1] - lo[1]) / (hi[1] - lo[1])
        sc.vel[water, 0] += (flow * (0.3 + 0.7 * height)).astype(np.float32)
        sc.vel[water, 2] += np.float32(0.2 * flow)
        if "multi" in case:
            p.sf_type = params.SF_TYPE_MULTI_SF if case["multi"] else params.SF_TYPE_SF
            p.solver_type = params.SF_SOLVER_WCSPH if case["wcsph"] else params.SF_SOLVER_SPH
    return out


def _dt(scs):
    return min(params.reference_dt(sc.params, sc.bparams, sc.sparams)[1] for sc in scs)


def _positions(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    size = torch.tensor([case["grid_x"], case["grid_y"], case["grid_z"]], device=DEV) * case["cell"]
    pos = torch.rand(case["n"], 3, generator=g, device=DEV) * size
    if case["ordered"]:  # nearly in cell order, as positions are a substep after the last sort
        c = (pos / case["cell"]).long()
        pos = pos[torch.argsort((c[:, 0] * case["grid_y"] + c[:, 1]) * case["grid_z"] + c[:, 2], stable=True)]
        pos = pos + (torch.rand(pos.shape, generator=g, device=DEV) - 0.5) * (0.02 * case["cell"])
    return pos.contiguous()


def _stream():
    """One stream for every handle, as a program has that runs one simulation after the other: what a pass takes is then
    not hidden by another simulation's."""
    if "s" not in _STREAM:
        _STREAM["s"] = torch.cuda.Stream()
    return _STREAM["s"].cuda_stream


_STREAM = {}


class _Fields:
    """Arguments of sf_set_fields / sf_get_fields for one scene's fields in device memory."""

    def __init__(self, tensors):
        self.t = tensors
        names = list(tensors)
        self.k = len(names)
        self.ids = (ctypes.c_int32 * self.k)(*[params.FIELDS[n][0] for n in names])
        self.ptrs = (ctypes.c_void_p * self.k)(*[tensors[n].data_ptr() for n in names])
        self.n = tensors[names[0]].shape[0]


def prepare(case, seed):
    if case["kind"] == "cell_sort":
        g = (case["grid_x"], case["grid_y"], case["grid_z"])
        hi = tuple(float(np.float32((c + 0.5) * case["cell"])) for c in g)
        b = params.boundary_params((0.0, 0.0, 0.0), hi, case["cell"])
        cells = b.grid_size[0] * b.grid_size[1] * b.grid_size[2]
        return dict(kind="cell_sort", lib=capi.load(), grid=b, pos=_positions(case, seed),
                    perm=torch.empty(case["n"], dtype=torch.int32, device=DEV),
                    start=torch.empty(cells + 1, dtype=torch.int32, device=DEV))
    scs = _scenes(case, seed)
    s = dict(kind=case["kind"], sim=capi.Simulation(scs if len(scs) > 1 else scs[0], stream=_stream()), substeps=case["substeps"], dt=_dt(scs))
    s["reset"] = [_Fields({"pos": torch.from_numpy(sc.pos).to(DEV), "vel": torch.from_numpy(sc.vel).to(DEV),
                           "col": torch.from_numpy(sc.col).to(DEV),
                           "max_saturation": torch.zeros(sc.n, device=DEV)}) for sc in scs]
    if case["kind"] == "adjoint":
        # a target near the start: every sand particle displaced by a few millimetres
        rng = np.random.default_rng([seed, 1 << 20])
        s["target"] = np.concatenate([sc.pos + rng.uniform(-4e-3, 4e-3, sc.pos.shape).astype(np.float32) for sc in scs])
        s["checkpoint"], s["state_grads"] = case["checkpoint"], case["state_grads"]
        return s
    if case["kind"] == "frame":
        n = scs[0].n
        s["pinned"] = torch.zeros(case["substeps"] + 1, 3, n, 3, pin_memory=True)
        s["pinned"][0, 1].copy_(torch.from_numpy(scs[0].vel))
        s["frames"] = [dict(zip(("pos", "vel", "col"), f)) for f in s["pinned"].numpy()]
    results = RESULTS if len(scs) == 1 else ("pos", "vel", "saturation")
    width = {k: params.FIELDS[k][1] for k in results}
    flat = {k: torch.empty(sum(sc.n for sc in scs) * w, device=DEV) for k, w in width.items()}
    s["out"], at = [], 0
    for sc in scs:
        s["out"].append(_Fields({k: flat[k][at * w:(at + sc.n) * w] for k, w in width.items()}))
        s["out"][-1].n = sc.n
        at += sc.n
    s["results"] = {k: flat[k].view(-1, w) if w > 1 else flat[k] for k, w in width.items()}
    return s


# --------------------------------------------------------------------- run
def _ok(sim, status):
    if status != capi.SF_OK:
        raise capi.SfError(status, sim.lib.sf_last_error_string(sim.h).decode())


def run(state):
    if state["kind"] == "cell_sort":
        st = state["lib"].sf_cell_sort_noalloc(ctypes.byref(state["grid"]), state["pos"].data_ptr(),
                                               state["pos"].shape[0], state["perm"].data_ptr(),
                                               state["start"].data_ptr(), None)
        if st != capi.SF_OK:
            raise RuntimeError(state["lib"].sf_last_error_string(None).decode())
        return [state["perm"], state["start"]]
    sim, kind = state["sim"], state["kind"]
    sim.reset_order()
    for k, f in enumerate(state["reset"]):
        _ok(sim, sim.lib.sf_set_fields(sim.h, k, f.k, f.ids, 1, f.ptrs, f.n, 1))
    if kind == "adjoint":
        r = sim.adjoint(state["dt"], state["substeps"], state["target"], checkpoint_every=state["checkpoint"],
                        want_state_grads=state["state_grads"])
        out = {"loss": r["loss"], "grad_params": r["grad_params"]}
        if state["state_grads"]:
            out.update(grad_pos0=r["grad_pos0"], grad_vel0=r["grad_vel0"])
        return out
    counts = []
    if kind == "substeps":
        sim.substeps_fixed(state["dt"], state["substeps"])
    elif kind == "step":
        for _ in range(state["substeps"]):
            counts.append(sim.step(T_FRAME))
    else:
        for before, after in zip(state["frames"], state["frames"][1:]):
            sim.set_fields({"vel": before["vel"]})
            counts.append(sim.step(T_FRAME))
            sim.get_fields(after)
    for k, f in enumerate(state["out"]):
        _ok(sim, sim.lib.sf_get_fields(sim.h, k, f.k, f.ids, 1, f.ptrs, f.n, 1))
    out = dict(state["results"])
    if counts:
        out["n_sub"] = np.array(counts, np.int64)
    if kind == "frame":
        out["frames"] = [[f["pos"], f["vel"], f["col"]] for f in state["frames"][1:]]
    return out


# -------------------------------------------------------------------- work
def work(case):
    """Per particle and substep: position, velocity, mass and label read, position and velocity written (52 B), about
    33 pairs of some 100 operations; the results once more per pass. The gradient reads the stored states again and
    does about twice the operations."""
    if case["kind"] == "cell_sort":
        cells = case["grid_x"] * case["grid_y"] * case["grid_z"]
        return {"bytes": 16 * case["n"] + 4 * (cells + 1), "flops": 0}
    n = case["n_sand"] + case["n_water"]
    if case["geometry"] == "batched" or case["geometry"] == "calibration":
        lo, hi = case["n_sand"], max(case["n_water"], case["n_sand"] + 1)  # log-uniform sizes
        n = case["scenes"] * (hi - lo) / math.log(hi / lo)
    k = case["substeps"]
    if case["kind"] == "adjoint":
        return {"bytes": n * (24 + 3 * 52 * k + 24), "flops": n * k * 33 * 300}
    per_pass = 28 + 4 * (14 if case["geometry"] != "batched" else 7)
    host = 48 * k if case["kind"] == "frame" else 0
    return {"bytes": n * (52 * k + per_pass + host), "flops": n * k * 33 * 100}


# ------------------------------------------------- the substep in 64 bits
def _cells(B, p):
    """Cell coordinates and sort order of positions on the grid of the boundary parameters."""
    lo = torch.tensor(B.lowest_point[:], dtype=torch.float64, device=DEV)
    g = torch.tensor(B.grid_size[:], device=DEV)
    c = torch.minimum(((p - lo) / B.kernel_radius).long().clamp_min(0), g - 1)
    key = (c[:, 0] * g[1] + c[:, 1]) * g[2] + c[:, 2]
    return c, key, torch.argsort(key)


def _pairs(B, a, b, reach):
    """(i, j) with |a_i - b_j| < reach, reach at most a cell."""
    gx, gy, gz = B.grid_size[:]
    ca = _cells(B, a)[0]
    _, kb, order = _cells(B, b)
    sorted_b, sorted_k = b[order], kb[order].contiguous()
    all_i, all_j = [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            x, y = ca[:, 0] + dx, ca[:, 1] + dy
            inside = ((x >= 0) & (x < gx) & (y >= 0) & (y < gy)).nonzero().squeeze(1)
            base = (x[inside] * gy + y[inside]) * gz
            z0 = (ca[inside, 2] - 1).clamp_min(0)
            z1 = (ca[inside, 2] + 1).clamp_max(gz - 1)
            first = torch.searchsorted(sorted_k, base + z0)
            count = torch.searchsorted(sorted_k, base + z1, right=True) - first
            i = torch.repeat_interleave(inside, count)
            at = torch.arange(i.numel(), device=DEV) - torch.repeat_interleave(count.cumsum(0) - count, count)
            j = at + torch.repeat_interleave(first, count)
            near = ((a[i] - sorted_b[j]).square().sum(1) < reach * reach).nonzero().squeeze(1)
            all_i.append(i[near])
            all_j.append(order[j[near]])
    return torch.cat(all_i), torch.cat(all_j)


def _sum(n, i, v):
    return torch.zeros((n,) + v.shape[1:], dtype=v.dtype, device=DEV).index_add(0, i, v)


def _set(base, at, v):
    return base.index_copy(0, at, v)


def _bezier(py0, py1, px1, py2, s):
    first = s <= px1
    t = torch.where(first, s, torch.zeros_like(s)) / px1
    out = (1 - t) ** 2 * py0 + 2 * t * (1 - t) * py1 + t * t * py1
    b = -2.0 * (px1 + 1) / 4
    k = 1 + b - px1
    r = torch.where(first, torch.full_like(s, px1), s)
    t = (b + torch.sqrt(b * b - 4 * k * (px1 - r))) / (2 * k)
    out = torch.where(first, out, (1 - t) ** 2 * py1 + 2 * t * (1 - t) * py1 + t * t * py2)
    out = torch.where(s < 0, torch.full_like(out, 1.0) * py0, out)
    return torch.where(s >= 1, torch.full_like(out, 1.0) * py2, out)


class _Exact:
    """One scene in float64: the passes of the substep, differentiable in the state and the three parameters."""

    def __init__(self, sc):
        f64 = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=DEV)  # noqa: E731
        self.p, self.B, self.sp = sc.params, sc.bparams, sc.sparams
        self.h = self.B.kernel_radius
        sand = torch.as_tensor(sc.label == params.SF_LABEL_SAND, device=DEV)
        self.sand, self.water = sand.nonzero().squeeze(1), (~sand).nonzero().squeeze(1)
        self.n, self.m, self.cd = sc.n, f64(sc.mass), f64(sc.cda0asat)[:, 0]
        self.x, self.v = f64(sc.pos), f64(sc.vel)
        self.max_sat = torch.zeros(sc.n, dtype=torch.float64, device=DEV)
        self.col = f64(sc.col)
        one = lambda v: torch.tensor(float(v), dtype=torch.float64, device=DEV)  # noqa: E731
        self.tan, self.cap, self.perm = one(self.p.dem_tan_friction_angle), one(1.0), one(1.0)
        self.b = f64(sc.bpos)
        i, j = _pairs(self.B, self.b, self.b, self.h)
        off = i != j
        w = self._w((self.b[i[off]] - self.b[j[off]]).square().sum(1))
        self.bvol = 1.0 / _sum(self.b.shape[0], i[off], w).clamp_min(EPS)
        if bool(sc.blabel.any()):
            raise ValueError("shape boundaries are not restated")

    def _w(self, r2):
        return 315.0 / (64 * math.pi * self.h ** 9) * (self.h * self.h - r2).clamp_min(0) ** 3

    def _grad(self, d):
        r = d.square().sum(1).sqrt()
        k = torch.where(r < EPS, torch.zeros_like(r), -45.0 / (math.pi * self.h ** 6) * (self.h - r).clamp_min(0) ** 2 / r)
        return k[:, None] * d

    def _dem(self, d, dv, rij):
        p = self.p
        kn = p.dem_young * p.dem_particle_radius
        dist = d.square().sum(1).sqrt()
        n = d / dist[:, None]
        vt = dv - (dv * n).sum(1, keepdim=True) * n
        fn = kn * (rij - dist)[:, None] * n
        fs = -kn * p.dem_poisson * vt
        fs2, most = fs.square().sum(1), fn.square().sum(1) * self.tan ** 2
        over = fs2 > most
        ratio = torch.sqrt(torch.where(over, most, torch.ones_like(most)) / torch.where(over, fs2, torch.ones_like(fs2)))
        return -fn - fs * torch.where(over, ratio, torch.ones_like(ratio))[:, None]

    def _bridge(self, d, sat):
        p, r = self.p, self.p.dem_particle_radius
        angle = 30.0 / 180.0 * math.pi
        volume = 4.0 / 3.0 * math.pi * r ** 3 * 0.01 * 0.01
        dist = d.square().sum(1).sqrt()
        H = dist - 2 * r
        k = _bezier(p.sf_c0, p.sf_cmc, p.sf_cmc_p, p.sf_csat, sat) * self.cap
        e = -H + torch.sqrt(H * H + volume / (math.pi * r))
        phi = torch.sqrt(2 * H / r * (-1 + torch.sqrt(1 + volume / (math.pi * r * H * H))))
        f = -2 * math.pi * k * r * (math.cos(angle) / (1 + H / (2 * e)) + phi * math.sin(angle))
        return -d / dist[:, None] * f[:, None]

    def substep(self, dt=None):
        """dt None: the adaptive rule for a frame of T_FRAME."""
        p, h, n, m, x, v = self.p, self.h, self.n, self.m, self.x, self.v
        sand, water, B = self.sand, self.water, self.B
        xd = x.detach()
        index = lambda a, b, r: tuple(q[k] for q, k in zip((a, b), _pairs(B, xd[a], xd[b], r)))  # noqa: E731
        wi, wj = index(water, water, h)
        si, sj = index(sand, sand, h)
        ui, uj = index(water, sand, h)  # water u, sand
        bi, bj = _pairs(B, xd[water], self.b, h)
        bi = water[bi]
        W = lambda i, j: self._w((x[i] - x[j]).square().sum(1))  # noqa: E731
        # density and pressure
        db = x[bi] - self.b[bj]
        rho_w = m * self._w(torch.zeros((), dtype=torch.float64, device=DEV)) + _sum(n, wi, m[wj] * W(wi, wj))
        rho_w = rho_w + _sum(n, bi, p.sph_density * self.bvol[bj] * self._w(db.square().sum(1)))
        rho = _set(torch.full((n,), p.dem_density, dtype=torch.float64, device=DEV), water, rho_w[water])
        rw = rho[water]
        if p.solver_type == params.SF_SOLVER_WCSPH:
            q = p.sph_stiff * ((rw / p.sph_density) ** 7 - 1)
            q = torch.where(q < 0, q * self.sp.negative_scale, q)
        else:
            q = p.sph_stiff * (rw - p.sph_density)
        pressure = _set(torch.zeros(n, dtype=torch.float64, device=DEV), water, q)
        # average flow, fluid voidage, saturation
        V = m / rho
        w_us = W(ui, uj)
        vol_s = _sum(n, si, V[sj] * W(si, sj)) + _sum(n, ui, V[uj] * w_us)
        flow_s, sat = _sum(n, uj, (V[ui] * w_us)[:, None] * v[ui]), _sum(n, uj, V[ui] * w_us)
        safe = lambda a: torch.where(a != 0, a, torch.ones_like(a))  # noqa: E731
        flow = flow_s / safe(sat)[:, None]
        eps_f = 1 - vol_s
        # sand voidage, water adhesion, colour
        num = _sum(n, uj, eps_f[ui] * V[ui] * w_us)
        voidage = _set(eps_f, sand, (num / safe(sat) * (sat != 0))[sand])
        d = x[ui] - x[uj]
        l_d = d.detach().square().sum(1).sqrt()
        band = ((2 * l_d > h) & (l_d <= h)).nonzero().squeeze(1)
        l = d[band].square().sum(1).sqrt()
        spline = 0.007 / h ** 3.25 * (-4 * l * l / h + 6 * l - 2 * h).clamp_min(0) ** 0.25
        bz = (0.0, 1.5, 0.5, 0.8) if p.sf_type == params.SF_TYPE_MULTI_SF else (p.sf_a0, p.sf_amc, p.sf_amc_p, p.sf_asat)
        f_ad = (_bezier(*bz, sat[uj[band]]) * m[ui[band]] * m[uj[band]] * spline / l)[:, None] * d[band]
        adhesion = _sum(n, ui[band], f_ad)
        v_s = _sum(n, ui, V[uj] * w_us)
        avg_adhesion = adhesion / safe(v_s)[:, None]
        wetter = (sat > self.max_sat) & (self.m > 0)
        wetter[water] = False
        dry, wet = (torch.tensor(c[:], dtype=torch.float64, device=DEV) for c in (p.sf_dry_sand_color, p.sf_wet_sand_color))
        self.col = torch.where(wetter[:, None], dry + (wet - dry) * sat[:, None], self.col).detach()
        self.max_sat = torch.where(wetter, sat, self.max_sat).detach()
        D = rho / voidage.clamp_min(EPS)
        # sand momentum
        ci, cj = index(sand, sand, 2 * p.dem_particle_radius * 1.1)
        other = ci != cj
        ci, cj = ci[other], cj[other]
        dc = x[cj] - x[ci]
        gap = dc.detach().square().sum(1).sqrt() - 2 * p.dem_particle_radius
        touch, bridge = (gap < 0).nonzero().squeeze(1), ((gap > 0) & (gap < scenes.capillary_rupture(p.dem_particle_radius))).nonzero().squeeze(1)
        f = _sum(n, ci[touch], self._dem(dc[touch], (v[cj] - v[ci])[touch], 2 * p.dem_particle_radius))
        f = f + _sum(n, ci[bridge], self._bridge(dc[bridge], 0.5 * (sat[ci[bridge]] + sat[cj[bridge]])))
        grad_us = self._grad(d)  # at water i, from sand j: G(x_i - x_j)
        open_ = ((voidage[ui] > 0) & (voidage[ui] <= 1)).nonzero().squeeze(1)
        oi, oj = ui[open_], uj[open_]
        f = f + _sum(n, oj, (m[oj] * m[oi] * pressure[oi] / (rho[oj] * D[oi]).clamp_min(EPS))[:, None] * grad_us[open_])
        v_w = _sum(n, oj, m[oi] / D[oi] * w_us[open_])
        f = f + _sum(n, uj, (w_us * V[uj])[:, None] * avg_adhesion[ui])
        rij = p.sph_particle_radius + p.dem_particle_radius
        for axis in range(3):
            for side, wall in ((1.0, B.highest_point[axis]), (-1.0, B.lowest_point[axis])):
                far = 2 * rij if axis == 2 and side < 0 else rij  # the z-min wall is tested at twice the distance
                gap = side * (wall - xd[sand, axis])
                at = sand[((gap < far) & ((xd[sand, axis] - wall).abs() < rij)).nonzero().squeeze(1)]
                dist = torch.zeros(at.numel(), 3, dtype=torch.float64, device=DEV)
                unit = torch.zeros(3, dtype=torch.float64, device=DEV)
                unit[axis] = side
                dist = dist + unit * (x[at, axis] - wall).abs()[:, None]
                f = f + _sum(n, at, self._dem(dist, -v[at], rij))
        in_band = sand[((voidage[sand] > 0) & (voidage[sand] < 1)).nonzero().squeeze(1)]
        e = voidage[in_band]
        cd = (self.cd[in_band] if p.sf_type == params.SF_TYPE_MULTI_SF else p.sf_cd) * self.perm * e ** 3 / (1 - e) ** 2
        drag = (abs(p.gravity[1]) * p.sph_density * e * e / cd * m[in_band] / rho[in_band])[:, None] * (flow - v)[in_band]
        df = _sum(n, in_band, drag)
        avg_drag = df / safe(v_w)[:, None] * (v_w != 0)[:, None]
        g = torch.tensor(p.gravity[:], dtype=torch.float64, device=DEV)
        acc = g + 2 * (f + df) / m[:, None]
        # water momentum
        P = pressure / (D * D).clamp_min(EPS)
        other = wi != wj
        i, j = wi[other], wj[other]
        dw = x[i] - x[j]
        dd = ((v[i] - v[j]) * dw).sum(1)
        visc = torch.where(dd < 0, -p.sph_nu / (D[i] + D[j]) * dd / (dw.square().sum(1) + EPS), torch.zeros_like(dd))
        a = _sum(n, i, (-m[j] * (P[i] + P[j] + visc))[:, None] * self._grad(dw))
        a = a + _sum(n, ui, (-m[uj] * pressure[ui] / (D[ui] * rho[uj]).clamp_min(EPS))[:, None] * grad_us
                     - (w_us / D[ui])[:, None] * avg_drag[uj])
        dd = (v[bi] * db).sum(1)
        visc = torch.where(dd < 0, -p.sph_bnu / (2 * p.sph_density) * dd / (db.square().sum(1) + EPS), torch.zeros_like(dd))
        per_b = -p.sph_density * self.bvol[bj] * (pressure[bi] / p.sph_density ** 2 + visc)
        a = a + _sum(n, bi, per_b[:, None] * self._grad(db))
        acc = _set(acc, water, (g + a - adhesion / m[:, None])[water])
        # time step, damping, Euler, clamp
        if dt is None:
            count, dt = self._cfl(float(acc.detach().square().sum(1).max().sqrt()))
        else:
            count = None
        sign = torch.sign(acc.detach() * (v.detach() + 0.5 * dt * acc.detach()))
        sign[water] = 0
        acc = acc * (1 - p.dem_damping * sign)
        v = v + dt * acc
        x = x + dt * v
        edge = 2 * p.sph_particle_radius
        lo = torch.tensor(B.lowest_point[:], dtype=torch.float64, device=DEV) + edge
        hi = torch.tensor(B.highest_point[:], dtype=torch.float64, device=DEV) - edge
        xw, vw = x[water], v[water]
        vw = torch.where(xw > hi, vw.clamp_max(0), torch.where(xw < lo, vw.clamp_min(0), vw))
        xw = torch.minimum(torch.maximum(xw, lo), hi)
        self.x, self.v = _set(x, water, xw), _set(v, water, vw)
        self.fields = dict(acc=acc, density=rho, pressure=pressure, voidage=voidage, saturation=sat)
        return count

    def _cfl(self, amax):
        """(sub-step count of T_FRAME, time step); the count in float32, since it is a truncated quotient."""
        p, f = self.p, np.float32
        if p.solver_type != params.SF_SOLVER_WCSPH:
            return int(f(T_FRAME) / f(p.dt)), p.dt
        by_force = f(0.25) * np.sqrt(f(self.h) * f(p.sph_mass) / (f(amax) * f(p.sph_mass)))
        by_speed = f(0.4) * f(self.h) / f(self.sp.speed_of_sound)
        count = int(f(T_FRAME) / min(f(p.dt), f(self.sp.time_step_limit_scale) * min(by_force, by_speed)))
        return count, float(f(T_FRAME)) / count


def exact(case, seed):
    if case["kind"] == "cell_sort":
        return None  # whole numbers alone
    # at most some 10 s: about 1.5 s a substep of a million particles
    n = case["n_sand"] + case["n_water"] if case["geometry"] not in ("batched", "calibration") else case["scenes"] * 20000
    if n * case["substeps"] > 9e6:
        return None
    scs = _scenes(case, seed)
    dt = float(np.float32(_dt(scs)))
    if case["kind"] == "adjoint":
        return _exact_gradient(case, seed, scs, dt)
    every = [_Exact(sc) for sc in scs]
    with torch.no_grad():
        for e in every:
            for _ in range(case["substeps"]):
                e.substep(None if case["kind"] in ("step", "frame") else dt)
    names = RESULTS if len(scs) == 1 else ("pos", "vel", "saturation")
    out = {k: torch.cat([{"pos": e.x, "vel": e.v, "max_saturation": e.max_sat, **e.fields}[k] for e in every]) for k in names}
    if case["kind"] in ("step", "frame"):
        out["n_sub"] = None
    if case["kind"] == "frame":  # in cell order, which a particle on a cell face has another place in
        out["frames"] = [[None] * 3] * case["substeps"]
    return out


def _exact_gradient(case, seed, scs, dt):
    rng = np.random.default_rng([seed, 1 << 20])
    loss, gp, gx, gv = [], [], [], []
    # after three substeps a contact on its threshold may be open in float32 and closed in float64: from there on the
    # two trajectories have other gradients, and only the loss can be compared
    far = case["substeps"] > 3
    for sc in scs:
        target = torch.as_tensor(sc.pos + rng.uniform(-4e-3, 4e-3, sc.pos.shape).astype(np.float32), dtype=torch.float64,
                                 device=DEV)
        e = _Exact(sc)
        x0, v0 = e.x, e.v
        leaves = [e.tan, e.cap, e.perm, x0, v0]
        for t in leaves:
            t.requires_grad_(True)
        with torch.set_grad_enabled(not far):
            for _ in range(case["substeps"]):
                e.substep(dt)
        value = (e.x[e.sand] - target[e.sand]).square().sum(1).mean()
        loss.append(float(value.detach()))
        if far:
            continue
        grads = torch.autograd.grad(value, leaves)
        gp.append([float(g) for g in grads[:3]])
        gx.append(grads[3])
        gv.append(grads[4])
    out = {"loss": np.array(loss), "grad_params": None if far else np.array(gp)}
    if case["state_grads"] and not far:
        out.update(grad_pos0=torch.cat(gx), grad_vel0=torch.cat(gv))
    return out
