"""The work a program has this library do, as cases that can be timed.

A case is one call (or the few calls) that a user's program makes: a step of
a scene held on the GPU, a rollout replayed from a checkpoint, a step of a
state kept in host memory, the separate phases, a batch of scenes, a
differentiated rollout, a sampled volume. `exact` restates one step (and the
derivative of a short rollout) in 64 bits with plain torch.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from fluids3_gb300._lib import call
from fluids3_gb300.system import (FCLR, FFORCE, FGCELL, FPOS, FPRESS, FVEL, FVEVAL, FluidSystem, default_params,
                                  derive_params)

DEV = "cuda"

# Two parameter sets: "cell2h", the dam-break set of the repository's own
# scenes (cell = 2h, 2 x 2 x 2 search block), and "default", the library's
# defaults (cell = 0.75h, 3 x 3 x 3 search block).
COMMON = dict(sim_scale=0.004, pmass=0.00020543, pvisc=0.35, pradius=0.015, bound_slope=0.0, bound_friction=0.0,
              grav_dir=(0.0, -9.8, 0.0), grav_amt=1.0, dt=0.003)
SETS = {
    "cell2h": dict(COMMON, psmoothradius=0.01, prest_dens=600.0, pintstiff=1.0, bound_stiff=10000.0, bound_damp=256.0,
                   AL=200.0, VL=3.0, grid_density=0.75),
    "default": dict(COMMON, psmoothradius=0.015, prest_dens=400.0, pintstiff=1.5, bound_stiff=50000.0,
                    bound_damp=150.0, AL=150.0, VL=50.0, grid_density=2.0),
}
SPACING = 0.0059 / 0.004   # rest distance in world units
MARGIN = 4.0


def listed():
    return [
        # one frame of a tiny interactive scene: launches and latency
        dict(name="step_2k", kind="step", n=2048, params="cell2h", packing=0.9, wall=False),
        # one frame of a mid-sized scene with the library's default parameters (3 x 3 x 3 search block)
        dict(name="step_default_100k", kind="step", n=100003, params="default", packing=0.95, wall=False),
        # the 32,768-point dam break over its 100 steps, as one call
        dict(name="rollout_dam_32k", kind="rollout", n=32768, params="cell2h", fill=0.5, steps=100, wall=False),
        # a second of simulation with the default parameters
        dict(name="rollout_default_250k", kind="rollout", n=250000, params="default", fill=0.3, steps=20, wall=False),
        # the headline scene: 4,000,000 points with the moving wall
        dict(name="rollout_tank_4m", kind="rollout", n=4000000, params="cell2h", fill=0.4, steps=10, wall=True),
        # a scene that collapses into crowded cells as it runs
        dict(name="rollout_collapse_65k", kind="rollout", n=65536, params="cell2h", fill=0.5, steps=160, wall=False),
        # many scenes of uneven sizes, each with its own parameters
        dict(name="batch_64", kind="batch", scenes=64, nmin=2048, nmax=65536, steps=20),
        # a state kept in page-locked host memory, stepped and read back
        dict(name="host_1500k", kind="host", n=1500001, params="cell2h", packing=0.9, wall=False),
        # the phases called one by one, with a program's own work between them
        dict(name="phases_262k", kind="phases", n=262144, params="cell2h", packing=0.9, wall=False),
        # gradients of a rollout: checkpoints and replay, and a large scene that keeps every step's pair lists
        dict(name="grad_65k", kind="grad", n=65536, params="cell2h", steps=10, every=5, keep=False),
        dict(name="grad_1200k", kind="grad", n=1200000, params="cell2h", steps=4, every=1, keep=True),
        # a frame's volume for rendering
        dict(name="volume_128", kind="volume", n=250001, params="cell2h", packing=0.9, res=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("step", "step", "rollout", "rollout", "host", "phases", "batch", "grad", "volume"))
    params = rng.choice(("cell2h", "cell2h", "default"))
    if kind in ("step", "phases"):
        return dict(kind=kind, n=_log(rng, 2048, 2000000), params=params, packing=round(rng.uniform(0.85, 1.0), 3),
                    wall=rng.random() < 0.5)
    if kind == "host":
        return dict(kind=kind, n=_log(rng, 2048, 1500001), params=params, packing=round(rng.uniform(0.85, 1.0), 3),
                    wall=False)
    if kind == "rollout":
        n = _log(rng, 2048, 1000000)
        most = 100 if n <= 65536 else 5 if params == "default" else 20
        return dict(kind=kind, n=n, params=params, fill=round(rng.uniform(0.25, 0.6), 2),
                    steps=_log(rng, 2, most), wall=rng.random() < 0.5)
    if kind == "batch":
        scenes = _log(rng, 2, 64)
        return dict(kind=kind, scenes=scenes, nmin=_log(rng, 500, 4000), nmax=_log(rng, 5000, 65536),
                    steps=_log(rng, 1, 20))
    if kind == "grad":
        every = rng.choice((1, 2, 5))
        steps = every * rng.choice((1, 2))
        most = 4800000 // steps // (4 if params == "default" else 1)
        return dict(kind=kind, n=_log(rng, 2048, min(1200000, most)), params=params, steps=steps, every=every,
                    keep=rng.random() < 0.5)
    return dict(kind=kind, n=_log(rng, 2048, 1000000), params=params, packing=round(rng.uniform(0.85, 1.0), 3),
                res=_log(rng, 16, 160))


# ---------------------------------------------------------------------------
# inputs


def _lattice(n, fill, packing=1.0):
    """Shape of a block of n points filling the low-x part of a box: lattice
    counts, spacing and the box."""
    s = SPACING * packing
    edge = SPACING * (n / fill) ** (1.0 / 3.0)
    nz = max(2, int((edge - 2 * MARGIN) / s))
    nx = max(2, int(round(fill * edge / s)))
    layers = -(-n // (nx * nz))
    lx = (nx * s + 2 * MARGIN) / fill
    lz = nz * s + 2 * MARGIN
    ly = max(layers * s + 2 * MARGIN, lz)
    return nx, nz, s, (round(lx, 1), round(ly, 1), round(lz, 1))


def _points(n, fill, packing, jitter, speed, seed):
    """Positions (a jittered lattice block, y layers outermost as the
    reference fills a volume), velocities, evaluated velocities and an id
    per point, on the GPU."""
    nx, nz, s, box = _lattice(n, fill, packing)
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    k = torch.arange(n, device=DEV)
    xz = k % (nx * nz)
    idx = torch.stack([xz % nx, k // (nx * nz), xz // nx], 1).float()
    u = torch.rand(n, 3, generator=g, device=DEV)
    pos = idx * s + MARGIN + (2 * u - 1) * (jitter * s)
    if speed == 0:
        return box, pos, torch.zeros_like(pos), torch.zeros_like(pos), k.int()
    vel = torch.randn(n, 3, generator=g, device=DEV) * (0.4 * speed)
    vel[:, 1] -= speed
    veval = vel + torch.randn(n, 3, generator=g, device=DEV) * (0.02 * speed)
    return box, pos.contiguous(), vel, veval, k.int()


def _raw(case, box):
    """A case's parameter inputs."""
    raw = dict(SETS[case.get("params", "cell2h")], bound_min=(0.0, 0.0, 0.0), bound_max=box, bound_wall_force=0.0,
               bound_wall_freq=0.0)
    if case.get("wall"):
        raw.update(bound_wall_force=0.3, bound_wall_freq=0.2)
    return raw


def _params(raw):
    p = default_params()
    p.set(**raw)
    return derive_params(p)


def _inputs(case, seed):
    """(raw parameters, pos, vel, veval, id) of a single-scene case. Rollouts
    start at rest; single frames, phases and volumes from a flowing state."""
    if case["kind"] == "rollout":
        box, *pts = _points(case["n"], case["fill"], 1.0, 0.05, 0.0, seed)
    elif case["kind"] == "grad":
        box, *pts = _points(case["n"], 0.5, 0.95, 0.15, 0.3, seed)
    else:
        box, *pts = _points(case["n"], 0.4, case["packing"], 0.3, 0.5, seed)
    return (_raw(case, box), *pts)


def _batch_inputs(case, seed):
    """Per scene: (raw parameters, pos, vel, veval, id)."""
    r = np.random.RandomState(seed % (1 << 31))
    sizes = np.random.RandomState(7).uniform(size=(case["scenes"], 2))   # the batch's shape; values by the seed
    out = []
    for k in range(case["scenes"]):
        n = int(round(case["nmin"] * (case["nmax"] / case["nmin"]) ** sizes[k, 0]))
        box, *pts = _points(n, 0.2 + 0.4 * sizes[k, 1], 1.0, 0.05, 0.2, seed * 1000 + k)
        raw = _raw(case, box)
        raw.update(pvisc=float(np.float32(r.uniform(0.1, 0.5))), prest_dens=float(np.float32(r.uniform(500, 700))))
        out.append((raw, *pts))
    return out


# ---------------------------------------------------------------------------
# states


class _State:
    pass


_SHAPE = {FPOS: 3, FVEL: 3, FVEVAL: 3, FFORCE: 3, FPRESS: 1, FCLR: 0, FGCELL: 0}
_NAME = {FPOS: "pos", FVEL: "vel", FVEVAL: "veval", FFORCE: "force", FPRESS: "density", FCLR: "id", FGCELL: "cell"}


def _buffers(st, n, ids):
    st.out = {}
    for b in ids:
        w = _SHAPE[b]
        st.out[b] = torch.empty((n, 3) if w == 3 else (n,), dtype=torch.int32 if w == 0 else torch.float32, device=DEV)
    st.exports = [(b, C.c_void_p(t.data_ptr()), t.numel() * 4) for b, t in st.out.items()]


def _export(st):
    for b, ptr, nbytes in st.exports:
        call("fl_export_device", st.sys.handle, b, ptr, nbytes)
    return {_NAME[b]: t for b, t in st.out.items()}


def _host(t):
    return t.cpu().numpy()


def prepare(case, seed):
    st = _State()
    st.kind = kind = case["kind"]
    if kind == "batch":
        scs = _batch_inputs(case, seed)
        st.steps = case["steps"]
        st.sys = FluidSystem.batch([_params(s[0]) for s in scs], [s[1].shape[0] for s in scs])
        pos, vel, veval, ids = (torch.cat([s[k] for s in scs]) for k in (1, 2, 3, 4))
        st.sys.SetParticles(_host(pos), _host(vel), _host(veval), clr=_host(ids))
        st.sys.SaveCheckpoint(0)
        _buffers(st, pos.shape[0], (FPOS, FVEL, FPRESS, FCLR))
        return st
    raw, pos, vel, veval, ids = _inputs(case, seed)
    n = case["n"]
    p = _params(raw)
    st.sys = FluidSystem(p, n)
    st.dt, st.ss = float(p.dt), float(p.sim_scale)
    if kind == "host":
        st.arrays = [t.cpu().pin_memory() for t in (pos, vel, veval, ids)]
        st.pos_out = torch.empty((n, 3), dtype=torch.float32, pin_memory=True)
        _buffers(st, n, (FVEL, FVEVAL, FPRESS, FCLR))
        return st
    st.sys.SetParticles(_host(pos), _host(vel), _host(veval), clr=_host(ids))
    st.sys.SaveCheckpoint(0)
    if kind in ("step", "rollout"):
        st.steps = case.get("steps", 1)
        _buffers(st, n, (FPOS, FVEL, FVEVAL, FPRESS, FCLR))
    elif kind == "phases":
        _buffers(st, n, (FPOS, FVEL, FVEVAL, FPRESS, FFORCE, FCLR, FGCELL))
    elif kind == "grad":
        st.steps, st.every, st.keep = case["steps"], case["every"], case["keep"]
        st.target = _target(case, seed, pos)
        st.grads = [torch.empty((n, 3), dtype=torch.float32, device=DEV) for _ in range(3)]
        st.order = torch.empty(n, dtype=torch.int32, device=DEV)
        st.gparams = np.zeros(3, np.float64)
        _buffers(st, n, (FPOS, FVEL))
    elif kind == "volume":
        st.res = (case["res"],) * 3
        st.lo, st.hi = raw["bound_min"], raw["bound_max"]
        st.out = torch.empty(st.res[::-1], dtype=torch.float32, device=DEV)
    return st


def _target(case, seed, pos):
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
    return pos + torch.randn(pos.shape, generator=g, device=DEV)


def run(st):
    s = st.sys
    if st.kind in ("rollout", "batch"):
        s.RestoreCheckpoint(0)
        s.RunSteps(st.steps)
        return _export(st)
    if st.kind == "step":
        s.RestoreCheckpoint(0)
        s.Run()
        return _export(st)
    if st.kind == "host":
        pos, vel, veval, ids = (a.numpy() for a in st.arrays)
        s.RunFromHost(pos, vel, veval, ids.view(np.uint32), st.pos_out.numpy())
        return dict(_export(st), pos=st.pos_out)
    if st.kind == "phases":
        s.RestoreCheckpoint(0)
        s.InsertParticlesCUDA()
        s.PrefixSumCellsCUDA()
        s.CountingSortFullCUDA()
        s.ComputePressureCUDA()
        s.ComputeForceCUDA()
        s.AdvanceCUDA(0.0, st.dt, st.ss)
        return _export(st)
    if st.kind == "grad":
        # mean squared distance of the final positions to a target cloud
        s.RestoreCheckpoint(0)
        s.TapeBegin(st.steps, st.every, st.keep)
        s.RunSteps(st.steps)
        out = _export(st)
        call("fl_tape_order", s.handle, C.c_void_p(st.order.data_ptr()))   # returns when the rollout is done
        dpos = (out["pos"] - st.target[st.order.long()]) * (2.0 / st.order.numel())
        torch.cuda.ExternalStream(s.stream()).wait_stream(torch.cuda.current_stream())
        call("fl_backward", s.handle, C.c_void_p(dpos.data_ptr()), None, None,
             *[C.c_void_p(g.data_ptr()) for g in st.grads], st.gparams.ctypes.data_as(C.c_void_p))
        return {"gpos": st.grads[0], "gvel": st.grads[1], "gveval": st.grads[2], "gparams": st.gparams}
    s.RestoreCheckpoint(0)
    s.SampleParticles(st.res, st.lo, st.hi, out=C.c_void_p(st.out.data_ptr()))
    return st.out


def work(case):
    """Per step the state is read and written once (positions, velocities,
    evaluated velocities, ids: 40 B each way, density 4 B); a pair costs
    about 12 operations in the density sum and 40 in the force sum, twice
    that backward; a volume reads the positions and writes the voxels."""
    h = SETS[case.get("params", "cell2h")]["psmoothradius"] / 0.004
    pairs = 4.0 / 3.0 * math.pi * (h / (SPACING * case.get("packing", 1.0))) ** 3
    if case.get("params", "cell2h") == "cell2h":
        pairs *= 0.45      # the 2 x 2 x 2 search block covers part of the sphere
    kind = case["kind"]
    if kind == "batch":
        sizes = np.random.RandomState(7).uniform(size=(case["scenes"], 2))
        n = float(np.sum(np.round(case["nmin"] * (case["nmax"] / case["nmin"]) ** sizes[:, 0])))
        return {"bytes": case["steps"] * n * 84.0, "flops": case["steps"] * n * pairs * 52.0}
    n = float(case["n"])
    if kind == "volume":
        v = float(case["res"]) ** 3
        return {"bytes": 4 * v + 12 * n, "flops": 0.4 * v * pairs * 20.0}
    if kind == "grad":
        return {"bytes": case["steps"] * n * (84.0 + 36.0 * 3), "flops": case["steps"] * n * pairs * 3 * 52.0}
    steps = case.get("steps", 1)
    return {"bytes": steps * n * 84.0, "flops": steps * n * pairs * 52.0}


# ---------------------------------------------------------------------------
# 64-bit restatement (plain torch)


class _Const:
    """The step's constants from the parameter inputs: grid and kernel
    factors in 32 bits as a program's parameter block holds them."""

    def __init__(self, raw):
        f = np.float32
        self.raw = raw
        h, ss = f(raw["psmoothradius"]), f(raw["sim_scale"])
        size = f(1.5 * float(h) / float(f(raw["grid_density"])))
        border = f(2.0 * float(size / ss))
        world = size / ss
        self.res, self.gmin, self.delta = [], [], []
        for k in range(3):
            lo, hi = f(raw["bound_min"][k]) - border, f(raw["bound_max"][k]) + border
            r = int(np.ceil((hi - lo) / world))
            self.res.append(r)
            self.gmin.append(float(lo))
            self.delta.append(float(f(r) / (f(r) * size / ss)))
        srch = max(2, int(np.floor(f(2.0) * (h / ss) / world) + f(1.0)))
        self.scan_max = [r - srch for r in self.res]
        rx, ry, rz = self.res
        self.cells = rx * ry * rz
        self.adj = [(y * rz + z) * rx + x - ((rz + 1) * rx + 1)
                    for y in range(srch) for z in range(srch) for x in range(srch)]
        pi, p6, p9 = f(3.141592), float(h) ** 6, float(h) ** 9
        self.h = float(h)
        self.ss = float(ss)
        self.d2 = float(ss * ss)
        self.rd2 = float(h * h / (ss * ss))
        self.poly6 = 315.0 / (64.0 * float(pi) * p9)
        self.spiky = -45.0 / (float(pi) * p6)
        self.lap = 45.0 / (float(pi) * p6)

    def v(self, name):
        return float(np.float32(self.raw[name]))

    def cell(self, pos):
        p = pos.detach().float()
        c = [((p[:, k] - self.gmin[k]) * self.delta[k]).trunc().long() for k in range(3)]
        ok = torch.ones(p.shape[0], dtype=torch.bool, device=p.device)
        for k in range(3):
            ok &= (c[k] >= 1) & (c[k] <= self.scan_max[k])
        return torch.where(ok, (c[1] * self.res[2] + c[2]) * self.res[0] + c[0], self.cells)


def _candidates(K, cell, cnt, off, most=20_000_000):
    """(i, j) index chunks: queries against the members of their search blocks."""
    q = torch.nonzero(cell < K.cells).squeeze(1)
    adj = torch.tensor(K.adj, device=cell.device)
    at, m = 0, max(1, q.numel())
    per = max(1, int(most / 60))
    while at < m and q.numel():
        i = q[at:at + per]
        cc = cell[i][:, None] + adj[None, :]
        ln = cnt[cc].reshape(-1)
        total = int(ln.sum())
        if total > 3 * most and per > 1:
            per = max(1, per // 4)
            continue
        start = off[cc].reshape(-1)
        owner = i[:, None].expand(-1, adj.numel()).reshape(-1)
        rep = torch.repeat_interleave(torch.arange(ln.numel(), device=cell.device), ln, output_size=total)
        first = torch.cumsum(ln, 0) - ln
        j = start[rep] + torch.arange(total, device=cell.device) - first[rep]
        yield owner[rep], j
        at += per


def _pairs(K, pos, cell, cnt, off):
    x = pos.detach()
    out = []
    for i, j in _candidates(K, cell, cnt, off):
        d = x[i] - x[j]
        d = (d * d).sum(1)
        keep = (d < K.rd2) & (d > 0)
        out.append((i[keep], j[keep]))
    if not out:
        e = torch.zeros(0, dtype=torch.long, device=x.device)
        return e, e
    return torch.cat([o[0] for o in out]), torch.cat([o[1] for o in out])


def _step64(K, pos, vel, veval, ids, time, phys=None):
    """One step in 64 bits: the sorted new state, densities and forces.
    phys: (viscosity, rest density, stiffness) as tensors to differentiate."""
    v = K.v
    visc, rest, stiff = phys if phys is not None else (v("pvisc"), v("prest_dens"), v("pintstiff"))
    cell = K.cell(pos)
    order = torch.sort(cell, stable=True)[1]
    cell, pos, vel, veval, ids = cell[order], pos[order], vel[order], veval[order], ids[order]
    cnt = torch.bincount(cell, minlength=K.cells + 1)
    off = torch.cumsum(cnt, 0) - cnt
    inside = cell < K.cells
    i, j = _pairs(K, pos, cell, cnt, off)
    d = pos[i] - pos[j]
    dsq = (d * d).sum(1)
    rho = torch.zeros(pos.shape[0], dtype=torch.float64, device=pos.device).index_add(
        0, i, ((K.rd2 - dsq) * K.d2) ** 3) * (v("pmass") * K.poly6)
    rho = torch.where(rho == 0, torch.where(inside, 1.0, 0.0).double(), rho)
    safe = torch.where(inside, rho, torch.ones_like(rho))
    r = torch.sqrt(dsq * K.d2)
    c = K.h - r
    p = (safe - rest) * stiff
    pterm = K.ss * -0.5 * c * K.spiky * (p[i] + p[j]) / r
    f = (d * pterm[:, None] + (veval[j] - veval[i]) * (K.lap * visc)) * (c / (safe[i] * safe[j]))[:, None]
    force = torch.zeros_like(pos).index_add(0, i, f)
    new = _advance64(K, pos, vel, veval, force, time)
    keep = inside[:, None]
    zero = torch.zeros_like(pos)
    return dict(pos=torch.where(keep, new[0], zero - 1000.0), vel=torch.where(keep, new[1], zero),
                veval=torch.where(keep, new[2], veval), rho=rho, force=torch.where(keep, force, zero), ids=ids,
                order=order, inside=inside)


def _advance64(K, pos, vel, veval, force, time):
    v = K.v
    lo, hi = K.raw["bound_min"], K.raw["bound_max"]
    lo, hi = [float(np.float32(x)) for x in lo], [float(np.float32(x)) for x in hi]
    a = force * v("pmass")
    stiff, damp, rad = v("bound_stiff"), v("bound_damp"), v("pradius")
    wall = (torch.sin(time * v("bound_wall_freq") + pos[:, 2] / 400.0) * 0.5 + 0.5) * v("bound_wall_force")
    ax = [a[:, k] for k in range(3)]

    def push(diff, axis, sign, scale=1.0):
        adj = scale * stiff * diff - damp * sign * veval[:, axis]
        ax[axis] = ax[axis] + torch.where(diff > 1e-5, sign * adj, torch.zeros_like(adj))

    push(rad - (pos[:, 1] - lo[1]) * K.ss, 1, 1.0)
    push(rad - (hi[1] - pos[:, 1]) * K.ss, 1, -1.0)
    push(rad - (pos[:, 0] - (lo[0] + wall)) * K.ss, 0, 1.0, wall)
    push(rad - (hi[0] - pos[:, 0]) * K.ss, 0, -1.0)
    push(rad - (pos[:, 2] - lo[2]) * K.ss, 2, 1.0)
    push(rad - (hi[2] - pos[:, 2]) * K.ss, 2, -1.0)
    g = [float(np.float32(x) * np.float32(K.raw["grav_amt"])) for x in K.raw["grav_dir"]]
    a = torch.stack([ax[k] + g[k] for k in range(3)], 1)

    def limit(u, most):
        s = (u * u).sum(1, keepdim=True)
        over = s > most * most
        return u * torch.where(over, most / torch.sqrt(torch.where(over, s, torch.ones_like(s))), torch.ones_like(s))

    a, vel = limit(a, v("AL")), limit(vel, v("VL"))
    dt = v("dt")
    nxt = a * dt + vel
    return pos + nxt * (dt / K.ss), nxt, (vel + nxt) * 0.5


def _grads64(case, seed):
    raw, pos0, vel0, veval0, ids = _inputs(case, seed)
    K = _Const(raw)
    target = _target(case, seed, pos0).double()
    x = [t.double().requires_grad_(True) for t in (pos0, vel0, veval0)]
    phys = [torch.tensor(K.v(k), dtype=torch.float64, device=DEV, requires_grad=True)
            for k in ("pvisc", "prest_dens", "pintstiff")]
    pos, vel, veval = x
    t = 0.0
    for _ in range(case["steps"]):
        s = _step64(K, pos, vel, veval, ids, t, phys)
        pos, vel, veval, ids = s["pos"], s["vel"], s["veval"], s["ids"]
        t = float(np.float32(t) + np.float32(K.v("dt")))
    m = ids.numel()
    loss = ((pos - target[ids.long()]) ** 2).sum() / m
    loss.backward()
    return {"gpos": x[0].grad, "gvel": x[1].grad, "gveval": x[2].grad,
            "gparams": np.array([float(p.grad) for p in phys])}


def _volume64(case, seed):
    raw, pos, *_ = _inputs(case, seed)
    K = _Const(raw)
    cell = K.cell(pos)
    order = torch.sort(cell, stable=True)[1]
    cell, pos = cell[order], pos[order].double()
    cnt = torch.bincount(cell, minlength=K.cells + 1)
    off = torch.cumsum(cnt, 0) - cnt
    m = case["res"]
    hi = [np.float32(x) for x in raw["bound_max"]]
    ax = [torch.tensor((np.arange(m, dtype=np.float32) / np.float32(m)) * hi[k], device=DEV) for k in range(3)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    q = torch.stack([x, y, z], -1).reshape(-1, 3)
    qc = K.cell(q)
    q = q.double()
    out = torch.zeros(q.shape[0], dtype=torch.float64, device=DEV)
    h2 = 2.0 * K.h * K.h / 8.0
    kern = 1.0 / (float(np.float32(3.141592)) * 2.0 * K.h * K.h) ** 1.5
    for i, j in _candidates(K, qc, cnt, off):
        d = q[i] - pos[j]
        d = (d * d).sum(1)
        keep = (d < K.rd2) & (d > 0)
        out.index_add_(0, i[keep], kern * torch.exp(-(d[keep] * K.d2) / h2))
    return (out * float(np.float32(0.01))).reshape(m, m, m)


def exact(case, seed):
    kind = case["kind"]
    if kind == "grad":
        return _grads64(case, seed)
    if kind == "volume":
        return _volume64(case, seed)
    if case.get("steps", 1) != 1:
        return None      # a rollout's trajectory is chaotic: rounding grows about 1.4x a step
    if kind == "batch":
        parts = []
        for raw, pos, vel, veval, ids in _batch_inputs(case, seed):
            s = _step64(_Const(raw), pos.double(), vel.double(), veval.double(), ids, 0.0)
            parts.append(s)
        cat = lambda k: torch.cat([p[k] for p in parts])   # noqa: E731
        # every scene's points outside its grid come last in the scene, as in the batch's slots
        return {"pos": cat("pos"), "vel": cat("vel"), "density": cat("rho"), "id": None}
    raw, pos, vel, veval, ids = _inputs(case, seed)
    s = _step64(_Const(raw), pos.double(), vel.double(), veval.double(), ids, 0.0)
    out = {"pos": s["pos"], "vel": s["vel"], "veval": s["veval"], "density": s["rho"], "id": None}
    if kind == "phases":
        out.update(force=s["force"], cell=None)
    return out
