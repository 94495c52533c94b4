"""Workloads of the MPCD step through the framework's public entry points.

Each case is a dict of plain values; `kind` says which program it stands for:

  fields     pympcd.Simulation: step_and_sample(steps) + get_mean_fields(), the flow-profile
             measurement of the reference's README and benchmark
  particles  pympcd.Simulation: step(steps) + get_particle_positions() + get_particle_velocities(),
             a trajectory analysed on the host
  coupled    capi.Handle: device particles in, one step, device particles out, as a program that
             exchanges momentum with the fluid on every step does
  ensemble   capi.Handle(boxes=...): step_and_sample(steps) + sample_mean() of a mix of channels
  pressure   capi.Handle: the wall-pressure estimator with the density and velocity profile
  adjoint    adjoint.channel_profile forward and backward (body force and initial velocities)

Box sizes are container sizes (wall layers included); `walls` closes z.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import cudampcd_gb300 as pympcd
from cudampcd_gb300 import capi
from cudampcd_gb300.adjoint import channel_profile

DEVICE = "cuda:0"
DT = 0.02
DRAG = 0.001
ALPHA = 2.0 * math.pi / 3.0
EXACT_STEPS = 10               # steps that exact() follows: a chaotic flow has no trajectory to compare beyond
EXACT_LIMIT = {"srd": 20_000_000, "extended": 1_500_000}   # particle-steps that it follows, by collision
PRESCRIBED_LIMIT = 2_000_000   # particles up to which a `fields` or `particles` program sets its own start

SRD, EXTENDED = 0, 1


def _case(name, kind, L, walls, n, steps, algorithm="srd", **more):
    return dict(name=name, kind=kind, Lx=L[0], Ly=L[1], Lz=L[2], walls=walls, n=n, steps=steps, algorithm=algorithm, **more)


def listed():
    return [
        # the smallest call: a coupled program's single step on a small periodic box (latency and launches)
        _case("coupled_small", "coupled", (16, 16, 16), False, 10, 1),
        # the same program with the non-ideal fluid between walls
        _case("coupled_extended", "coupled", (40, 40, 42), True, 10, 1, "extended"),
        # a dilute, large box with odd sides, every step in and out on the device
        _case("coupled_dilute", "coupled", (151, 203, 97), False, 5, 1),
        # a short trajectory read back to the host, odd sides
        _case("trajectory", "particles", (33, 47, 29), False, 10, 100),
        # the reference's viscosity check: the 10 x 10 x 100 channel, a block of its long sampled run
        _case("viscosity_channel", "fields", (10, 10, 102), True, 10, 600),
        # an ordinary channel with odd sides and an odd density
        _case("odd_channel", "fields", (61, 61, 85), True, 7, 60),
        # the large channel of the benchmark, 4e8 particles
        _case("large_channel", "fields", (1000, 1000, 22), True, 20, 30),
        # the non-ideal channel of the benchmark
        _case("extended_channel", "fields", (256, 256, 66), True, 20, 12, "extended"),
        # the non-ideal fluid on a small box, where a step is short
        _case("extended_small", "fields", (24, 24, 26), True, 10, 60, "extended"),
        # many channels of uneven size, density and drag in one handle
        _case("ensemble", "ensemble", (64, 64, 200), True, 20, 12, boxes=64, mix=4),
        # the equation of state: wall pressure with its density profile
        _case("wall_pressure", "pressure", (64, 64, 34), True, 20, 30, "extended"),
        # the differentiable channel: gradients of a profile loss
        _case("adjoint_channel", "adjoint", (64, 64, 34), True, 10, 200, every=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["coupled", "particles", "fields", "fields", "ensemble", "pressure", "adjoint"])
    algorithm = rng.choice(["srd", "srd", "extended"])
    walls = rng.random() < 0.6
    n = rng.choice([5, 7, 10, 13, 20])
    side = _log_int(rng, 10, 200)
    L = [side, _log_int(rng, 10, 200), _log_int(rng, 10, 100) + (2 if walls else 0)]
    steps, more = 1, {}
    if kind in ("fields", "particles"):
        L[1] = L[0]   # the reference binding's field strides are exact for square cross-sections
        steps = _log_int(rng, 2, max(3, min(300, int(4e9 / (n * L[0] * L[1] * L[2])))))
    elif kind == "ensemble":
        walls, L, n = True, [64, 64, 200], 20   # the largest replica
        steps = _log_int(rng, 3, 30)
        more = dict(boxes=_log_int(rng, 4, 64), mix=rng.randrange(1 << 20))
    elif kind == "pressure":
        walls, steps = True, _log_int(rng, 4, 60)
        L[2] = max(L[2], 12)
    elif kind == "adjoint":
        walls, algorithm = True, "srd"
        L = [_log_int(rng, 8, 64), _log_int(rng, 8, 64), _log_int(rng, 10, 40) + 2]
        steps = _log_int(rng, 4, 100)
        more = dict(every=rng.randint(2, 20))
    c = _case("", kind, L, walls, n, steps, algorithm, **more)
    del c["name"]
    return c


# ---------------------------------------------------------------- what a case holds

def _geometry(case):
    L = (case["Lx"], case["Ly"], case["Lz"])
    fluid = (L[0], L[1], L[2] - (2 if case["walls"] else 0))
    return L, fluid, case["n"] * fluid[0] * fluid[1] * fluid[2]


def _replicas(case, seed):
    """Channels of uneven size, density and drag; the mix is the case's, the seeds are the inputs'."""
    rng = random.Random(case["mix"])
    out = []
    for r in range(case["boxes"]):
        L = (rng.choice([8, 16, 32, 64]), rng.choice([8, 16, 32, 64]), rng.randint(20, 200))
        out.append(dict(L=L, periodic=(1, 1, 0), n=rng.choice([5, 10, 20]), dt=DT,
                        drag=10.0 ** rng.uniform(-4.0, -2.0), algorithm=SRD if case["algorithm"] == "srd" else EXTENDED,
                        seed=seed * 1000003 + r))
    return out


def _particles(case, seed):
    """Uniform positions in the fluid and Maxwell-Boltzmann velocities at T = 1 without net momentum."""
    _, fluid, N = _geometry(case)
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    scale = torch.tensor(fluid, dtype=torch.float32, device=DEVICE)
    pos = (torch.rand((N, 3), generator=g, device=DEVICE) - 0.5) * scale
    vel = torch.randn((N, 3), generator=g, device=DEVICE)
    return pos, vel - vel.mean(0)


def _handle(case, seed):
    L, _, _ = _geometry(case)
    return capi.Handle(L=L, periodic=(1, 1, 0 if case["walls"] else 1), n=case["n"], dt=DT, drag=DRAG,
                       algorithm=SRD if case["algorithm"] == "srd" else EXTENDED, seed=seed)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("fields", "particles"):
        _, fluid, N = _geometry(case)
        p = pympcd.Params()
        p.n = case["n"]
        p.periodicity = (1, 1, 0 if case["walls"] else 1)
        p.volume_size = fluid
        p.algorithm = case["algorithm"]
        p.drag = DRAG
        p.delta_t = DT
        p.seed = seed
        sim = pympcd.Simulation(p, "cuda")
        if N <= PRESCRIBED_LIMIT:
            sim.set_particles(*(t.cpu().numpy() for t in _particles(case, seed)))
        return dict(case=case, sim=sim)
    if kind == "ensemble":
        return dict(case=case, handle=capi.Handle(boxes=_replicas(case, seed)))
    h = _handle(case, seed)
    state = dict(case=case, handle=h)
    if kind in ("coupled", "adjoint"):
        pos, vel = _particles(case, seed)
        state.update(pos=pos, vel=vel)
        torch.cuda.synchronize()
    if kind == "coupled":
        state.update(out_pos=torch.empty_like(pos), out_vel=torch.empty_like(vel))
    if kind == "adjoint":
        state.update(drag=torch.tensor(DRAG, dtype=torch.float64, requires_grad=True), v0=vel.requires_grad_(True),
                     target=_target(case))
    return state


def _target(case):
    """1.1 x the Poiseuille parabola of the analytic SRD viscosity."""
    n, h = case["n"], case["Lz"] / 2.0 - 1.0
    eta = (1.0 - math.cos(ALPHA)) / (18.0 * DT) * (n - 1 + math.exp(-n))
    z = torch.arange(case["Lz"], dtype=torch.float64, device=DEVICE) + 0.5 - case["Lz"] / 2.0
    return 1.1 * n * DRAG * (h * h - z * z) / (2.0 * eta)


def _loss(profile, target):
    return ((profile[1:-1].double() - target[1:-1]) ** 2).mean()


def run(state):
    case = state["case"]
    kind, steps = case["kind"], case["steps"]
    if kind == "fields":
        state["sim"].step_and_sample(steps)
        density, velocity = state["sim"].get_mean_fields()
        return dict(density=density, velocity=velocity)
    if kind == "particles":
        sim = state["sim"]
        sim.step(steps)
        return dict(positions=sim.get_particle_positions(), velocities=sim.get_particle_velocities())
    h = state["handle"]
    if kind == "ensemble":
        h.step_and_sample(steps)
        density, velocity = h.sample_mean()
        return dict(density=density, velocity=velocity)
    if kind == "pressure":
        h.wall_pressure(restart=True)
        h.step_and_sample(steps)
        bottom, top, measured = h.wall_pressure()
        density, velocity = h.sample_mean()
        return dict(pressure=np.array([bottom, top]), measured=measured, density=density, velocity=velocity)
    if kind == "coupled":
        h.set_particles_device(state["pos"].data_ptr(), state["vel"].data_ptr())
        h.step(steps)
        h.get_particles_device(state["out_pos"].data_ptr(), state["out_vel"].data_ptr())
        return dict(positions=state["out_pos"], velocities=state["out_vel"])
    profile = channel_profile(h, state["pos"], state["v0"], state["drag"], steps, case["every"])
    dv0, ddrag = torch.autograd.grad(_loss(profile, state["target"]), (state["v0"], state["drag"]))
    return dict(profile=profile.detach(), velocity_gradient=dv0, drag_gradient=ddrag)


def work(case):
    """Bytes: every step reads and writes the FP32 position and velocity of each particle once; results are
    written once.  Operations: streaming, two wraps and the collision, counted from the arithmetic of the model."""
    per_step = 100.0 if case["algorithm"] == "srd" else 220.0
    if case["kind"] == "ensemble":
        boxes = _replicas(case, 0)
        N = sum(b["n"] * b["L"][0] * b["L"][1] * (b["L"][2] - 2) for b in boxes)
        C = sum(b["L"][0] * b["L"][1] * b["L"][2] for b in boxes)
    else:
        L, _, N = _geometry(case)
        C = L[0] * L[1] * L[2]
    kind, steps = case["kind"], case["steps"]
    bytes_, flops = 48.0 * N * steps, per_step * N * steps
    if kind == "coupled":
        flops = per_step * N
    elif kind == "particles":
        bytes_ += 24.0 * N
    elif kind == "adjoint":   # forward, and a reverse sweep over the adjoint velocities with its recomputation
        bytes_, flops = (48.0 + 48.0 + 24.0) * N * steps, (2 * per_step + 60.0) * N * steps
    else:
        bytes_ += 16.0 * C
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------- the same step in 64 bits

def _philox(a, step, purpose, d, seed):
    """Philox4x32-10 of counter (a, step, purpose, d) and key seed: four uint32 arrays."""
    a, d = np.broadcast_arrays(np.asarray(a, np.uint64), np.asarray(d, np.uint64))
    low = np.uint64(0xFFFFFFFF)
    c = [a.copy(), np.full(a.shape, step & 0xFFFFFFFF, np.uint64), np.full(a.shape, purpose | ((step >> 32) << 8), np.uint64),
         d.copy()]
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _uniform(u):
    return (u >> np.uint64(8)).astype(np.float64) * 2.0 ** -24


def _gaussians(ua, ub):
    r = np.sqrt(-2.0 * np.log(_uniform(ua) + 2.0 ** -24))
    phi = 2.0 * np.pi * _uniform(ub)
    return r * np.cos(phi), r * np.sin(phi)


def _tensor(x):
    return torch.as_tensor(np.ascontiguousarray(x), device=DEVICE)


class _Exact:
    """The MPCD step of one box in float64, with the framework's documented Philox draws."""

    def __init__(self, case, seed, pos, vel):
        self.case, self.seed = case, seed
        self.L, _, _ = _geometry(case)
        self.size = torch.tensor(self.L, dtype=torch.float64, device=DEVICE)
        self.x, self.v = pos.double(), vel.double()
        self.dt = float(np.float32(DT))
        self.kick = float(np.float32(DRAG)) * self.dt
        self.step = 0
        x, y, z = np.meshgrid(*(np.arange(n) for n in self.L), indexing="ij")
        self.ref = (x + self.L[0] * (y + self.L[1] * z)).reshape(-1)   # storage: x slowest, z fastest
        self.z = z.reshape(-1)
        self.centre = _tensor(np.stack([v.reshape(-1) + 0.5 - n / 2.0 for v, n in zip((x, y, z), self.L)], 1))
        self.C = self.ref.size

    def wrap(self, x):
        return torch.remainder(x + self.size / 2, self.size) - self.size / 2

    def cell(self, x):
        c = torch.remainder(torch.floor(x + self.size / 2), self.size).long()
        return (c[:, 0] * self.L[1] + c[:, 1]) * self.L[2] + c[:, 2]

    def stream(self):
        x, v, dt = self.x, self.v, self.dt
        moved = x + v * dt
        if self.case["walls"]:
            wall = self.L[2] / 2.0 - 1.0
            hit = moved[:, 2].abs() > wall
            vz = torch.where(hit, v[:, 2], torch.ones_like(v[:, 2]))
            left = ((torch.sign(moved[:, 2]) * wall - x[:, 2]) / vz)[:, None]
            moved = torch.where(hit[:, None], x + v * left - v * (dt - left), moved)
            v = torch.where(hit[:, None], -v, v)
        self.x, self.v = moved, v

    def ghosts(self, shift):
        """Wall cells (storage index), their ghost counts, and the layer-xor-sign bit of each."""
        if not self.case["walls"]:
            return np.zeros(0, np.int64), np.zeros(0, np.int64), np.zeros(0, bool)
        sign = shift > 0
        layer = self.z == self.L[2] - (1 if sign else 2)
        cells = np.nonzero(layer | (self.z == int(sign)))[0]
        flip = layer[cells] ^ sign
        n = self.case["n"]
        u = np.concatenate([np.stack(_philox(self.ref[cells], self.step, 3, i, self.seed), 1) for i in range((n + 3) // 4)], 1)
        return cells, ((_uniform(u[:, :n]) > abs(shift)) ^ flip[:, None]).sum(1), flip

    def sums(self, values, cell):
        return torch.zeros((self.C,) + values.shape[1:], dtype=torch.float64, device=DEVICE).index_add(0, cell, values)

    def advance(self, drag=None):
        """One step; `drag`: the body force as a tensor, for gradients."""
        kick = self.kick if drag is None else drag * self.dt
        self.stream()
        o = _philox(0, self.step, 1, 0, self.seed)
        s = [float(_uniform(o[i])) - 0.5 for i in range(3)]
        shift = torch.tensor(s, dtype=torch.float64, device=DEVICE)
        x = self.wrap(self.x + shift)
        cell = self.cell(x.detach())
        push = torch.zeros_like(self.v)
        push = push + torch.stack([torch.ones_like(cell, dtype=torch.float64) * kick, push[:, 1], push[:, 2]], 1)
        collide = self.srd if self.case["algorithm"] == "srd" else self.extended
        entries, v, x_unshifted = collide(x, cell, s, shift, push)
        hit = (entries[cell] > 1)[:, None]
        self.x, self.v = torch.where(hit, x_unshifted, x), torch.where(hit, v, self.v)
        self.step += 1

    def srd(self, x, cell, s, shift, push):
        cells, g, _ = self.ghosts(s[2])
        total = self.sums(self.v, cell)
        entries = torch.bincount(cell, minlength=self.C)
        if cells.size:
            o = _philox(self.ref[cells], self.step, 7, 0, self.seed)
            g0, g1 = _gaussians(o[0], o[1])
            g2, _ = _gaussians(o[2], o[3])
            at = _tensor(cells)
            total = total.index_add(0, at, _tensor(np.stack([g0, g1, g2], 1) * np.sqrt(g)[:, None]))
            entries = entries.index_add(0, at, _tensor(g))
        mean = (total / entries.clamp(min=1)[:, None])[cell]
        o = _philox(self.ref, self.step, 2, 0, self.seed)
        z = 1.0 - 2.0 * _uniform(o[0])
        rho, phi = np.sqrt(np.maximum(0.0, 1.0 - z * z)), 2.0 * np.pi * _uniform(o[1])
        axis = _tensor(np.stack([rho * np.cos(phi), rho * np.sin(phi), z], 1))[cell]
        r = self.v - mean
        along = axis * (r * axis).sum(1, keepdim=True)
        across = r - along
        v = mean + along + math.cos(ALPHA) * across + math.sin(ALPHA) * torch.linalg.cross(across, axis) + push
        return entries, v, self.wrap(x - shift)

    def extended(self, x, cell, s, shift, push):
        N = x.shape[0]
        cells, g, flip = self.ghosts(s[2])
        real = torch.bincount(cell, minlength=self.C)
        order = torch.argsort(cell, stable=True)   # participants in particle order within a cell, then the ghosts
        rank = torch.empty_like(order)
        rank[order] = torch.arange(N, device=DEVICE) - (torch.cumsum(real, 0) - real)[cell[order]]
        px, pv, pc, pk = x, self.v, cell, rank
        if g.sum():
            at, j = np.repeat(cells, g), np.concatenate([np.arange(k) for k in g])
            up, a = np.repeat(flip, g), abs(s[2])
            o = _philox(self.ref[at], self.step, 4, 2 * j, self.seed)
            z = np.where(up, a * _uniform(o[2]), a + (1.0 - a) * _uniform(o[2]))
            gx = _tensor(np.stack([_uniform(o[0]) - 0.5, _uniform(o[1]) - 0.5, z - 0.5], 1)) + self.centre[_tensor(at)]
            o = _philox(self.ref[at], self.step, 4, 2 * j + 1, self.seed)
            g0, g1 = _gaussians(o[0], o[1])
            g2, _ = _gaussians(o[2], o[3])
            px, pv = torch.cat([px, gx]), torch.cat([pv, _tensor(np.stack([g0, g1, g2], 1))])
            pc, pk = torch.cat([pc, _tensor(at)]), torch.cat([pk, real[_tensor(at)] + _tensor(j)])
        entries = torch.bincount(pc, minlength=self.C)
        count = entries.clamp(min=1).double()[:, None]
        com = self.sums(px - self.centre[pc], pc) / count + self.centre
        mean = self.sums(pv, pc) / count
        px, pv = px - com[pc], pv - mean[pc]
        o = _philox(self.ref, self.step, 2, 0, self.seed)
        axis = self.axes()[_tensor((o[0] >> np.uint64(1)).astype(np.int64) % 13)]
        axis = torch.where(_tensor(((o[1] >> np.uint64(1)) & np.uint64(1)) == 1)[:, None], -axis, axis)
        gate, pa = _tensor(_uniform(o[2])), axis[pc]
        below = (px * pa).sum(1) < 0
        along = (pv * pa).sum(1)
        n0 = self.sums(below.double(), pc)
        n1 = entries.double() - n0
        proj = self.sums(torch.where(below, along, torch.zeros_like(along)), pc)
        proj0, proj1 = proj / n0, -proj / n1
        hit = (gate < 1 - torch.exp(0.01 * (proj1 - proj0) * n0 * n1)) & (entries > 1)
        o = np.stack(_philox(self.ref[pc.cpu().numpy()], self.step, 5, pk.cpu().numpy() // 4, self.seed), 1)
        g0, g1 = _gaussians(o[:, 0], o[:, 1])
        g2, g3 = _gaussians(o[:, 2], o[:, 3])
        thermal = _tensor(np.stack([g0, g1, g2, g3], 1)).gather(1, (pk % 4)[:, None])[:, 0]
        before = torch.linalg.cross(px, pv)
        swap = torch.where(below, (proj1 * (n1 / n0))[pc], (proj0 * (n0 / n1))[pc])
        drift = torch.where(below, (self.sums(torch.where(below, thermal, torch.zeros_like(thermal)), pc) / n0)[pc],
                            (self.sums(torch.where(below, torch.zeros_like(thermal), thermal), pc) / n1)[pc])
        new = pv + pa * (thermal - along + swap - drift)[:, None]
        turn = self.sums(before - torch.linalg.cross(px, new), pc)
        inertia = (self.sums((px * px).sum(1), pc)[:, None, None] * torch.eye(3, dtype=torch.float64, device=DEVICE)
                   - self.sums(px[:, :, None] * px[:, None, :], pc))
        det, trace = torch.linalg.det(inertia).clamp(min=0), torch.diagonal(inertia, dim1=1, dim2=2).sum(1)
        solid = det > 1e-5
        inverse = torch.linalg.inv(torch.where(solid[:, None, None], inertia, torch.eye(3, dtype=torch.float64, device=DEVICE)))
        flat = torch.where((trace > 1e-5)[:, None, None], inertia * (4 / trace.clamp(min=1e-5) ** 2)[:, None, None], torch.zeros_like(inertia))
        omega = (torch.where(solid[:, None, None], inverse, flat) @ turn[:, :, None])[:, :, 0]
        spin = new - torch.linalg.cross(px, omega[pc])
        v = torch.where(hit[pc][:, None], spin, pv) + mean[pc]
        return entries, v[:N] + push, self.wrap(x - shift)

    def axes(self):
        """The 13 axes of the extended collision (the reference's table of angles)."""
        out = []
        for k in range(13):
            i, j = k % 4 + 1, k // 4 + 1
            magic = 0.95531661812450927816
            theta = (magic if j == 1 else math.pi - magic) if i % 2 and j % 2 else j * math.pi / 4
            phi = i * math.pi / 4
            out.append((math.sin(theta) * math.cos(phi), math.sin(theta) * math.sin(phi), math.cos(theta)))
        return torch.tensor(out, dtype=torch.float64, device=DEVICE)

    def sample(self):
        """Particles and mean velocity of every lab cell."""
        cell = self.cell(self.x.detach())
        count = torch.bincount(cell, minlength=self.C).double()
        return count, self.sums(self.v, cell) / count.clamp(min=1)[:, None]


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    _, _, N = _geometry(case)
    if kind in ("fields", "particles") and N > PRESCRIBED_LIMIT:
        return None   # it starts from the framework's own distribution
    if kind in ("ensemble", "pressure") or steps > EXACT_STEPS or N * steps > EXACT_LIMIT[case["algorithm"]]:
        return None
    pos, vel = _particles(case, seed)
    if kind == "adjoint":
        v0 = vel.double().requires_grad_(True)
        drag = torch.tensor(DRAG, dtype=torch.float64, device=DEVICE, requires_grad=True)
        box, profile = _Exact(case, seed, pos, v0), 0.0
        for _ in range(steps):
            box.advance(drag)
            box.x = box.x.detach()   # cells, bounces and shifts are held fixed; positions act only through them
            profile = profile + box.sample()[1][:, 0].reshape(-1, case["Lz"]).mean(0) / steps
        dv0, ddrag = torch.autograd.grad(_loss(profile, _target(case)), (v0, drag))
        return dict(profile=profile.detach(), velocity_gradient=dv0, drag_gradient=ddrag)
    box = _Exact(case, seed, pos, vel)
    density, velocity = 0.0, 0.0
    for _ in range(steps):
        box.advance()
        if kind == "fields":
            count, mean = box.sample()
            density, velocity = density + count, velocity + mean
    if kind == "fields":   # S samples are divided by S - 1, as in the reference
        L = box.L
        density, velocity = density.reshape(L) / (steps - 1), velocity.reshape(*L, 3) / (steps - 1)
        return dict(density=density, velocity=velocity)
    return dict(positions=box.x, velocities=box.v)
