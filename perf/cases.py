"""Workloads of the contact engine as a program that uses it runs them, for timing and comparison.

A pass of a single-scene case is one leg of a host-driven simulation: the program writes the
state it holds (pinned buffers: positions, quaternions, velocities, angular velocities) into
the solver, runs the steps to its next output and reads the state back.  A pass of a batch
case is the same leg of a running ensemble: its next steps, then every scene read back (a
batch has no state write-back, so its passes go on from where the last one ended).

Scenes (sizes and material settings are those of the repository's configurations, scaled by
the body count; radii +-`spread` around r0):
  inward   bodies on a jittered lattice driven to its centre (vap_fixed), in 3D inside a box
           of six planes, in 2D without obstacles;
  gravity  a bed of bodies on a floor plane falling under gravity (vap_fpd);
  se       superellipsoids on a lattice above a floor plane, with friction (vap_fpd);
  batch    many 2D beds, each on its own floor segment, of log-uniform sizes.
`gap` is the clear distance between mean-sized neighbours and `jitter` their displacement,
both in units of r0; `vmax` the agitation of the bodies in m/s (0.1 m/s closes a gap of
0.05 r0 of 2 mm bodies in one step), which sets how many contacts are active.
"""
import math

import numpy as np
import torch

from scopi_b200 import (FP64, FRICTION, MIXED, NOFRICTION, VAP_FIXED, VAP_FPD, VISCOUS, ScopiBatch, ScopiSolver,
                        configs)
from scopi_b200.container import PLANE, SEGMENT, SPHERE, ParticleArrays

PROBLEM = {"nofriction": NOFRICTION, "friction": FRICTION, "viscous": VISCOUS}
PRECISION = {"fp64": FP64, "mixed": MIXED}
MU = 0.3
TOL = 1e-6
MAX_ITE = 40000


def _case(name, scene, dim, count, problem, precision, steps, gap=0.1, spread=0.1, jitter=0.1, vmax=0.1, scenes=0):
    c = dict(scene=scene, dim=dim, count=count, problem=problem, precision=precision, steps=steps, gap=gap,
             spread=spread, jitter=jitter, vmax=vmax, scenes=scenes)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a desktop-sized crowd or granular model: one thousand disks pulled to a point, the plain FP64 form
        _case("disks_1k_fp64", "inward", 2, 1024, "nofriction", "fp64", 2, gap=0.5, spread=0.2, jitter=0.2, vmax=0.05),
        # a small bed with friction between script-side decisions (control, coupling): launches and latency
        _case("bed_2d_friction_700", "gravity", 2, 701, "friction", "fp64", 1, vmax=0.2),
        # a mid-sized drop-in run of the reference's own precision, ragged count
        _case("bed_3d_fp64_30k", "gravity", 3, 30011, "nofriction", "fp64", 1, vmax=0.1),
        # spheres filling a box, the chosen mixed form
        _case("bed_3d_mixed_100k", "gravity", 3, 100_000, "nofriction", "mixed", 2, vmax=0.1),
        # friction with rolling, the plain FP64 form
        _case("bed_3d_friction_fp64_10k", "gravity", 3, 10_007, "friction", "fp64", 1, vmax=0.1),
        # friction with rolling at scale, mixed
        _case("bed_3d_friction_mixed_150k", "gravity", 3, 150_000, "friction", "mixed", 1, vmax=0.1),
        # lubricated suspension: the viscous problem, gamma carried from step to step
        _case("viscous_3d_mixed_200k", "inward", 3, 200_000, "viscous", "mixed", 2, vmax=0.1),
        # a million spheres, mixed: the compression run between two outputs
        _case("inward_3d_mixed_1m", "inward", 3, 1_000_000, "nofriction", "mixed", 2, vmax=0.1),
        # the same in the plain FP64 form
        _case("inward_3d_fp64_1m", "inward", 3, 1_000_000, "nofriction", "fp64", 1, vmax=0.1),
        # a parameter study: many small 2D beds of uneven size in one batch, mixed
        _case("batch_mixed_256", "batch", 2, 5000, "nofriction", "mixed", 40, vmax=0.2, scenes=256),
        # a study with friction (FP64), fewer scenes
        _case("batch_friction_96", "batch", 2, 2000, "friction", "fp64", 3, vmax=0.2, scenes=96),
        # non-spherical bodies poured on a plate
        _case("se_friction_mixed_4k", "se", 3, 4001, "friction", "mixed", 1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["inward2", "bed2", "bed3", "bed3", "friction3", "viscous3", "inward3", "batch", "se"])
    prec = rng.choice(["fp64", "mixed"])
    vmax = round(rng.uniform(0.05, 0.2), 3)
    if kind == "inward2":
        return _case(None, "inward", 2, _log(rng, 200, 60_000), "nofriction", prec, 1, 0.5, 0.2, 0.2, vmax)
    if kind == "bed2":
        return _case(None, "gravity", 2, _log(rng, 100, 20_000), rng.choice(["nofriction", "friction"]), prec, 1, vmax=vmax)
    if kind == "bed3":
        return _case(None, "gravity", 3, _log(rng, 300, 300_000), "nofriction", prec, 1, vmax=vmax)
    if kind == "friction3":
        return _case(None, "gravity", 3, _log(rng, 300, 100_000 if prec == "mixed" else 20_000), "friction", prec, 1,
                     vmax=vmax)
    if kind == "viscous3":
        return _case(None, "inward", 3, _log(rng, 1000, 200_000), "viscous", prec, 1, vmax=vmax)
    if kind == "inward3":
        return _case(None, "inward", 3, _log(rng, 1000, 1_000_000 if prec == "mixed" else 500_000), "nofriction", prec, 1,
                     vmax=vmax)
    if kind == "batch":
        fr = rng.random() < 0.4
        return _case(None, "batch", 2, rng.randrange(800, 2000 if fr else 5000), "friction" if fr else "nofriction",
                     "fp64" if fr else prec, 2 if fr else 20, vmax=vmax, scenes=rng.randrange(8, 96 if fr else 200))
    return _case(None, "se", 3, _log(rng, 200, 4000), "friction", prec, 1)


# ------------------------------------------------------------------ scenes
def _quat(angle, axis):
    s = math.sin(angle / 2)
    return [math.cos(angle / 2), s * axis[0], s * axis[1], s * axis[2]]


def _arrays(dim, shape, pos, q, v, vd, f, m, j, radius, length, nin):
    n = len(shape)
    z = np.zeros((n, 3))
    return ParticleArrays(dim=dim, nb_inactive=nin, shape=np.ascontiguousarray(shape, np.int32), pos=pos, q=q, v=v,
                          omega=z.copy(), vd=vd, omega_d=z.copy(), f=f, m=m, j=j, radius=radius, length=length)


def _radius0(c):
    return 0.01 if c["dim"] == 2 else 0.002


def _bodies(c, count, rng, obstacles):
    """`count` spheres or disks on the first points of a lattice (last axis fastest) centred at
    0.5 in the horizontal axes, their lowest layer half a spacing above 0 (gravity) or centred
    (inward), after the obstacles (position, quaternion, shape, length)."""
    dim, r0 = c["dim"], _radius0(c)
    sp = (2 + c["gap"]) * r0
    gravity = c["scene"] != "inward"
    if dim == 2:
        nx = max(1, int(round(math.sqrt(count * (2 if gravity else 1)))))
        k = np.arange(count)
        grid = np.stack([k % nx, k // nx, 0 * k], 1).astype(np.float64)  # layer by layer from the floor
        size = np.array([nx, -(-count // nx), 1])
    else:
        side = max(1, math.ceil(round(count ** (1 / 3), 9)))
        k = np.arange(count)
        grid = np.stack([k // (side * side), (k // side) % side, k % side], 1).astype(np.float64)
        size = np.array([side, side, side])
    x = np.zeros((count, 3))
    up = dim - 1
    for d in range(dim):
        lo = (1.02 * r0) if (gravity and d == up) else 0.5 - (size[d] - 1) / 2 * sp
        x[:, d] = lo + sp * grid[:, d] + (rng.random(count) * 2 - 1) * c["jitter"] * r0
    if gravity:
        x[:, up] += c["jitter"] * r0
    rr = (1 + (rng.random(count) * 2 - 1) * c["spread"]) * r0
    nin, n = len(obstacles), len(obstacles) + count
    shape = np.full(n, SPHERE, np.int32)
    pos, q, vec = np.zeros((n, 3)), np.zeros((n, 4)), np.zeros((n, 3))
    q[:, 0] = 1
    length, radius, m, j = np.zeros(n), np.zeros(n), np.ones(n), np.ones((n, 3))
    for i, (p, qq, sh, ln) in enumerate(obstacles):
        pos[i, :len(p)], q[i], shape[i], length[i] = p, qq, sh, ln
    pos[nin:], radius[nin:] = x, rr
    m[nin:] = (rr / r0) ** dim
    j[nin:] = ((0.5 if dim == 2 else 0.4) * m[nin:] * rr * rr)[:, None]
    v, vd, f = vec.copy(), vec.copy(), vec.copy()
    agitation = (rng.random((count, dim)) * 2 - 1) * c["vmax"]
    if gravity:
        v[nin:, :dim] = agitation
        f[nin:, up] = -9.81 * m[nin:]
    else:
        d = 0.5 - x[:, :dim]
        vd[nin:, :dim] = 0.1 * d / np.maximum(np.sqrt((d * d).sum(1)), 1e-9)[:, None] + agitation
    return _arrays(dim, shape, pos, q, v, vd, f, m, j, radius, length, nin)


def _scene(c, seed):
    rng = np.random.default_rng(seed)
    if c["scene"] == "se":
        return configs.se_pile(c["count"], side=max(2, int(round(math.sqrt(c["count"] / 3)))), seed=seed & 0x7FFFFFFF)
    if c["scene"] == "gravity":
        if c["dim"] == 2:
            return _bodies(c, c["count"], rng, [((0.0, 0.0), _quat(math.pi / 2, (0, 0, 1)), PLANE, 0.0)])
        return _bodies(c, c["count"], rng, [((0.0, 0.0, 0.0), _quat(-math.pi / 2, (0, 1, 0)), PLANE, 0.0)])
    if c["dim"] == 2:
        return _bodies(c, c["count"], rng, [])
    xq, yq, zq = _quat(0.0, (0, 0, 1)), _quat(math.pi / 2, (0, 0, 1)), _quat(-math.pi / 2, (0, 1, 0))
    walls = [((0, 0, 0), xq), ((1, 0, 0), xq), ((0, 0, 0), yq), ((0, 1, 0), yq), ((0, 0, 0), zq), ((0, 0, 1), zq)]
    return _bodies(c, c["count"], rng, [(p, qq, PLANE, 0.0) for p, qq in walls])


def _scenes(c, seed):
    """Scene sizes log-uniform in [200, count] (the case's own, whatever the seed); every bed on
    a segment a little wider than it."""
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng([c["scenes"], c["count"]]).uniform(math.log(200), math.log(c["count"]), c["scenes"])
    sizes = np.exp(sizes).round().astype(int)
    out = []
    for n in sizes:
        w = (math.sqrt(2.0 * n) + 4) * (2 + c["gap"]) * _radius0(c)
        out.append(_bodies(c, int(n), rng, [((0.5, 0.0), _quat(-math.pi / 2, (0, 0, 1)), SEGMENT, w)]))
    return out


def _settings(c):
    r0 = _radius0(c)
    if c["scene"] == "se":
        st = configs.SETTINGS["se_pile"]
        return dict(dmax=st["dmax"], vap=VAP_FPD), st["dt"]
    if c["scene"] == "inward" and c["dim"] == 2:
        st = configs.SETTINGS["disks_2d"]
        return dict(dmax=st["dmax"], vap=VAP_FIXED), st["dt"]
    return dict(dmax=0.9 * r0, vap=VAP_FIXED if c["scene"] == "inward" else VAP_FPD), 1e-3


def _pinned(shape):
    t = torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return t.numpy()


# ------------------------------------------------------------------ one pass
def prepare(case, seed):
    c = dict(case)
    kw, dt = _settings(c)
    kw.update(tolerance=TOL, max_ite=MAX_ITE, problem=PROBLEM[c["problem"]], precision=PRECISION[c["precision"]])
    if c["problem"] == "friction":
        kw["mu"] = MU
    if c["problem"] == "viscous":
        kw["gamma_min"] = -2.0
    if c["scenes"]:
        return dict(case=c, batch=ScopiBatch(_scenes(c, seed), **kw), dt=dt)
    pa = _scene(c, seed)
    s = ScopiSolver(pa, **kw)
    host, out = pa.copy(), pa.copy()
    for k in ("pos", "q", "v", "omega"):
        buf = _pinned(getattr(pa, k).shape)
        buf[...] = getattr(pa, k)
        setattr(host, k, buf)
        setattr(out, k, _pinned(getattr(pa, k).shape))
    s.stream_handle()  # creates the handle and uploads the container
    return dict(case=c, solver=s, host=host, out=out, dt=dt)


def run(state):
    c, dt = state["case"], state["dt"]
    if c["scenes"]:
        b = state["batch"].run(dt, c["steps"])
        got = [b.scene(k) for k in range(c["scenes"])]
        return {k: np.concatenate([getattr(p, k) for p in got]) for k in ("pos", "q", "v", "omega")}
    s, out = state["solver"], state["out"]
    s.upload_state(state["host"])
    s.step(dt, c["steps"])
    s.download(out)
    return {"pos": out.pos, "q": out.q, "v": out.v, "omega": out.omega, "contacts": int(s.stats()["contacts"])}


def _sizes(c):
    """Bodies of a case (a batch's expected number)."""
    if c["scenes"]:
        lo, hi = 200.0, float(c["count"])
        return c["scenes"] * (hi - lo) / math.log(hi / lo)
    return c["count"]


def work(case):
    """Per step: every body's state read and written once, its fixed fields (mass, inertia,
    force or desired velocity, radius) read once; per contact (about 4 a body in 3D, 2 in 2D)
    its row of the Jacobian and its multipliers written and read once.  Flops: one
    multiplication of the contact matrix and one projection, the least a solve can take."""
    n, dim = _sizes(case), case["dim"]
    per = {"nofriction": 1, "viscous": 2, "friction": 3}[case["problem"]]
    size = 8 if case["precision"] == "fp64" else 4
    contacts = n * (4 if dim == 3 else 2)
    row = 2 * (dim if per < 3 else 6 * per) * size + 8 + 2 * per * size
    return {"bytes": float(case["steps"] * (n * (2 * 13 * 8 + 11 * 8) + 2 * contacts * row)),
            "flops": float(case["steps"] * contacts * per * 4 * (dim if per < 3 else 6))}


# ------------------------------------------------------------------ the same in plain 64-bit torch
def _rotation(q):
    w, x, y, z = q.unbind(1)
    return torch.stack([1 - 2 * y * y - 2 * z * z, 2 * x * y - 2 * w * z, 2 * x * z + 2 * w * y,
                        2 * x * y + 2 * w * z, 1 - 2 * x * x - 2 * z * z, 2 * y * z - 2 * w * x,
                        2 * x * z - 2 * w * y, 2 * y * z + 2 * w * x, 1 - 2 * x * x - 2 * y * y], 1).view(-1, 3, 3)


def _pairs(x, reach):
    """Pairs i < j of points closer than `reach`, by cells of that edge."""
    key3 = torch.floor((x - x.min(0).values) / reach).long() + 1
    dims = key3.max(0).values + 2
    key = (key3[:, 0] * dims[1] + key3[:, 1]) * dims[2] + key3[:, 2]
    key, order = torch.sort(key)
    found = []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                other = key + (dx * dims[1] + dy) * dims[2] + dz
                lo, hi = torch.searchsorted(key, other), torch.searchsorted(key, other, right=True)
                cnt = hi - lo
                a = torch.repeat_interleave(torch.arange(len(x), device=x.device), cnt)
                b = torch.arange(len(a), device=x.device) - torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt, cnt)
                a, b = order[a], order[b + torch.repeat_interleave(lo, cnt)]
                keep = a < b
                a, b = a[keep], b[keep]
                near = ((x[a] - x[b]) ** 2).sum(1) < reach * reach
                found.append((a[near], b[near]))
    return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])


def _apgd(mult, c, project, alpha):
    """Accelerated projected gradient with backtracking and restart on 1/2 l.Ql + c.l."""
    lam = torch.zeros_like(c)
    y, qy, qlam = lam.clone(), torch.zeros_like(c), torch.zeros_like(c)
    theta, lip = 1.0, 1.0 / alpha
    for _ in range(MAX_ITE):
        g = qy + c
        fy = (0.5 * (y * qy).sum() + (c * y).sum()).item()
        while True:
            new = project(y - g / lip)
            qnew = mult(new)
            d = new - y
            lhs = (0.5 * (new * qnew).sum() + (c * new).sum()).item()
            if not lhs >= fy + (g * d).sum().item() + 0.5 * lip * (d * d).sum().item():
                break
            lip *= 2
        step = torch.linalg.vector_norm(new - lam).item()
        if step < TOL:
            return new
        t1 = 0.5 * (theta * math.sqrt(4 + theta * theta) - theta * theta)
        beta = theta * (1 - theta) / (theta * theta + t1)
        if (g * (new - lam)).sum().item() > 0:
            y, qy, theta = new, qnew, 1.0
        else:
            y, qy, theta = new + beta * (new - lam), qnew + beta * (qnew - qlam), t1
        lip *= 0.97
        lam, qlam = new, qnew
    return lam


def _cone(z, n):
    zn = (z * n).sum(1, keepdim=True)
    t = z - zn * n
    nt = torch.linalg.vector_norm(t, dim=1, keepdim=True)
    s = MU * MU * (nt + zn / MU) / (MU * MU + 1)
    edge = s * t / torch.where(nt > 0, nt, torch.ones_like(nt)) + s / MU * n
    return torch.where(nt <= MU * zn, z, torch.where(zn <= -MU * nt, torch.zeros_like(z), edge))


def exact(case, seed):
    c = dict(case)
    if c["scenes"] or c["scene"] == "se" or c["problem"] == "viscous" or c["count"] * c["steps"] > 150_000:
        return None  # per-scene loops, MINPACK solves or minutes of iterations
    kw, dt = _settings(c)
    pa = _scene(c, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    nin, dim, friction = pa.nb_inactive, c["dim"], c["problem"] == "friction"
    get = {k: torch.tensor(getattr(pa, k)[nin:], dtype=torch.float64, device=dev)
           for k in ("pos", "q", "v", "omega", "vd", "f", "m", "j", "radius")}
    x, q, v, w, r = get["pos"], get["q"], get["v"], get["omega"], get["radius"]
    im = 1.0 / get["m"][:, None]
    ij = 1.0 / get["j"]
    if dim == 2:
        ij[:, :2] = 0
    walls = _rotation(torch.tensor(pa.q[:nin], device=dev))[:, :, 0]
    wpos = torch.tensor(pa.pos[:nin], device=dev)
    contacts = 0
    for _ in range(c["steps"]):
        a, b = _pairs(x, 2 * r.max().item() + kw["dmax"])
        diff = x[a] - x[b]
        dist = torch.linalg.vector_norm(diff, dim=1)
        keep = dist - r[a] - r[b] < kw["dmax"]
        a, b, nrm, dij = a[keep], b[keep], (diff / dist[:, None])[keep], (dist - r[a] - r[b])[keep]
        ia, ra = torch.ones_like(dij), -r[a][:, None] * nrm
        for k in range(nin):
            s = (x - wpos[k]) @ walls[k]
            hit = torch.nonzero(s.abs() - r < kw["dmax"])[:, 0]
            n = -torch.sign(s[hit])[:, None] * walls[k]
            a, b = torch.cat([a, hit]), torch.cat([b, hit])  # the obstacle's side counts for nothing (ia = 0)
            ia, ra = torch.cat([ia, torch.zeros_like(s[hit])]), torch.cat([ra, torch.zeros_like(n)])
            nrm, dij = torch.cat([nrm, n]), torch.cat([dij, s[hit].abs() - r[hit]])
        rb, ia = r[b][:, None] * nrm, ia[:, None]
        contacts = len(dij)
        if kw["vap"] == VAP_FIXED:
            v, w = get["vd"].clone(), torch.zeros_like(w)
        else:
            v = v + dt * get["f"] * im
            if dim == 3:
                jj = get["j"]
                w = w + torch.stack([w[:, 1] * w[:, 2] * (jj[:, 2] - jj[:, 1]), w[:, 0] * w[:, 2] * (jj[:, 0] - jj[:, 2]),
                                     w[:, 0] * w[:, 1] * (jj[:, 1] - jj[:, 0])], 1)
        rot = _rotation(q)

        def apply(vel, om):  # relative velocity of the contact points
            ow = torch.einsum("bij,bj->bi", rot, om)
            return ia * (vel[a] - torch.cross(ra, ow[a], dim=1)) - (vel[b] - torch.cross(rb, ow[b], dim=1))

        def force(f):  # M^-1 B^T f
            fv = torch.zeros_like(v).index_add_(0, a, ia * f).index_add_(0, b, -f)
            tq = torch.zeros_like(v).index_add_(0, a, ia * torch.cross(ra, f, dim=1))
            tq = tq.index_add_(0, b, -torch.cross(rb, f, dim=1))
            return im * fv, ij * torch.einsum("bji,bj->bi", rot, tq)

        if contacts:
            rel = apply(v, w)
            if friction:
                lam = _apgd(lambda l: dt * dt * apply(*force(l)), dij[:, None] * nrm + dt * rel,
                            lambda z: _cone(z, nrm), 0.05)
                dv, dw = force(lam)
            else:
                lam = _apgd(lambda l: dt * dt * (apply(*force(l[:, None] * nrm)) * nrm).sum(1),
                            dij + dt * (rel * nrm).sum(1), lambda z: z.clamp_min(0.0), 0.05)
                dv, dw = force(lam[:, None] * nrm)
            v, w = v + dt * dv, w + (dt * dw if friction else 0.0)
        x = x + dt * v
        nw = torch.linalg.vector_norm(w, dim=1)
        nw = torch.where(nw == 0, torch.ones_like(nw), nw)[:, None]
        e0, e = torch.cos(0.5 * nw * dt), torch.sin(0.5 * nw * dt) / nw * w
        q = torch.cat([q[:, :1] * e0 - (q[:, 1:] * e).sum(1, keepdim=True),
                       q[:, :1] * e + e0 * q[:, 1:] + torch.cross(q[:, 1:], e, dim=1)], 1)
        q = q / torch.linalg.vector_norm(q, dim=1, keepdim=True)
    res = {"contacts": contacts}
    for k, got in (("pos", x), ("q", q), ("v", v), ("omega", w)):
        full = getattr(pa, k).copy()
        full[nin:] = got.cpu().numpy()
        res[k] = full
    return res
