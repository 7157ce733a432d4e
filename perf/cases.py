"""The framework's work, as cases that can be timed and checked.

Kinds of case (``kind``):

* ``sim``: one call of ``Simulation.iterate`` on a running simulation, with its read-back of the
  fields into the host arrays. Scenes: ``shear`` (periodic 2D shear layer), ``vortex`` (periodic
  Taylor-Green vortex, 2D or 3D), ``channel`` (walls, a bounce-back cylinder, fixed inflow and
  outflow), each with or without a tracer that is coupled back by buoyancy.
* ``ensemble``: one call of ``Ensemble.iterate`` on lid-driven cavities of uneven sizes.
* ``train``: one training step of the learned closure: forward, loss, gradients, Adam.
* ``closed``: a coarse channel run with the trained closure refreshing its relaxation rates.

``exact`` restates each in 64-bit torch.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from boltzmann_b200 import closure as cl
from boltzmann_b200.core import CellFlags, Simulation, bgk, trt
from boltzmann_b200.ensemble import Ensemble

TAU_NEG = 0.52  # TRT: the odd relaxation time of the vortex-street example
BUOYANCY = 1e-5
TRACER_TAU = 0.503


def _sim(name, scene, counts, steps, collision="bgk", storage="f32", tracer="", tau=0.55):
    nx, ny, nz = (list(counts) + [1])[:3]
    return {"name": name, "kind": "sim", "scene": scene, "dim": len(counts), "nx": nx, "ny": ny,
            "nz": nz, "steps": steps, "collision": collision, "storage": storage,
            "tracer": tracer, "tau": tau}


def listed():
    return [
        # A tutorial-sized vortex, a few steps between two looks at the fields: every call is
        # launches and latency.
        _sim("vortex_64", "vortex", (64, 64), 20, tau=0.6),
        # The shear layer of the benchmark, the size that examples and sweeps use.
        _sim("shear_256", "shear", (256, 256), 400),
        # A vortex street on a domain of no particular size: odd rows, walls, TRT.
        _sim("street_1000x501", "channel", (1000, 501), 100, "trt", tau=0.52),
        # The benchmark's channel: TRT, a tracer, buoyancy; the largest 2D domain in use.
        _sim("channel_4096x2048", "channel", (4096, 2048), 100, "trt", tracer="f32", tau=0.502),
        # A wide channel in half-precision storage, fluid and tracer, on ragged rows.
        _sim("channel_f16_3000x1001", "channel", (3000, 1001), 100, "trt", "f16", "f16", 0.51),
        # The benchmark's 3D vortex, in single precision and in half-precision storage.
        _sim("vortex_256_3d", "vortex", (256, 256, 256), 40, tau=0.504),
        _sim("vortex_256_3d_f16", "vortex", (256, 256, 256), 40, storage="f16", tau=0.504),
        # A 3D duct with an obstacle and a warm, buoyant tracer, on odd rows.
        _sim("duct_180x100x90", "channel", (180, 100, 90), 60, "trt", tracer="f32", tau=0.53),
        # The double-precision run that other precisions are judged by.
        _sim("vortex_160_3d_f64", "vortex", (160, 160, 160), 20, storage="f64", tau=0.51),
        # A parameter sweep: cavities of 64 to 512 cells a side.
        {"name": "cavities_128", "kind": "ensemble", "domains": 128, "lo": 64, "hi": 512,
         "steps": 300, "storage": "f32"},
        # One step of training the closure at its own batch and grid.
        {"name": "train_8x1024x512", "kind": "train", "nx": 1024, "ny": 512, "batch": 8},
        # Using it: the coarse channel, the closure every ten steps.
        {"name": "closed_1024x512", "kind": "closed", "nx": 1024, "ny": 512, "steps": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """2D domains of 32 to 4096 cells a side, 3D ones of 16 to 256, in the storages, scenes and
    tracer forms above; smaller sweeps, batches and coarse grids than the listed ones."""
    pick = rng.random()
    if pick < 0.45:
        nx, ny = _log_int(rng, 32, 4096), _log_int(rng, 32, 2048)
        return _draw_sim(rng, (nx, ny), 4096 * 2048 * 60)
    if pick < 0.75:
        n = [_log_int(rng, 16, 256) for _ in range(3)]
        return _draw_sim(rng, n, 256**3 * 12)
    if pick < 0.83:
        lo = _log_int(rng, 16, 200)
        return {"kind": "ensemble", "domains": _log_int(rng, 4, 128), "lo": lo,
                "hi": min(512, lo + _log_int(rng, 16, 312)), "steps": 2 * rng.randint(10, 100),
                "storage": rng.choice(["f32", "f32", "f16"])}
    if pick < 0.92:
        return {"kind": "train", "nx": _log_int(rng, 40, 1024), "ny": _log_int(rng, 40, 512),
                "batch": rng.randint(1, 8)}
    return {"kind": "closed", "nx": _log_int(rng, 128, 1024), "ny": _log_int(rng, 64, 512),
            "steps": 10 * rng.randint(1, 10)}


def _draw_sim(rng, counts, most):
    dim = len(counts)
    scene = rng.choice(["vortex", "channel"] if dim == 3 else ["shear", "vortex", "channel"])
    storage = rng.choice(["f32", "f32", "f32", "f16", "bf16", "f64"])
    tracer = rng.choice(["", "", "f64" if storage == "f64" else "f32",
                         storage if storage in ("f16", "bf16") else ""])
    cells = math.prod(counts)
    steps = 2 * _log_int(rng, 5, max(6, min(200, most // (2 * cells))))
    case = _sim("", scene, counts, steps, rng.choice(["bgk", "trt"]), storage, tracer,
                round(rng.uniform(0.53, 0.7), 3))
    del case["name"]
    return case


# ---- inputs ---------------------------------------------------------------------------------


def _phases(seed, count):
    return np.random.default_rng([seed, 17]).uniform(0, 2 * np.pi, count)


def _waves(n, k, phase, f):
    return f(2 * np.pi * k * np.arange(n) / n + phase).astype(np.float32)


def _noise(seed, shape, amp):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return ((torch.rand(shape, generator=g, device="cuda") - 0.5) * (2 * amp)).cpu().numpy()


def _fields(case, seed):
    """flags, rho, vel, tracer value (or None) of a ``sim`` case, as host arrays."""
    dim = case["dim"]
    counts = [case["nx"], case["ny"], case["nz"]][:dim]
    flags = np.zeros(counts, np.int32)
    rho = np.ones(counts, np.float32)
    vel = np.zeros(counts + [dim], np.float32)
    ph = _phases(seed, 3)
    u0 = 0.05
    if case["scene"] == "shear":
        y = np.arange(counts[1])
        half, w = counts[1] / 2, max(2.0, counts[1] / 64)
        ux = u0 * np.where(y < half, np.tanh((y - half / 2) / w), np.tanh((1.5 * half - y) / w))
        vel[..., 0] = ux.astype(np.float32)
        vel[..., 1] = 1e-3 * _waves(counts[0], 1, ph[0], np.sin)[:, None]
        vel[..., 1] += _noise(seed, counts, 1e-4)
    elif case["scene"] == "vortex":
        s = [_waves(n, 1, p, np.sin) for n, p in zip(counts, ph)]
        c = [_waves(n, 1, p, np.cos) for n, p in zip(counts, ph)]
        c2 = [_waves(n, 2, 2 * p, np.cos) for n, p in zip(counts, ph)]
        ax = [(slice(None),) + (None,) * (dim - 1), (None, slice(None)) + (None,) * (dim - 2)]
        vel[..., 0] = u0 * s[0][ax[0]] * c[1][ax[1]]
        vel[..., 1] = -u0 * c[0][ax[0]] * s[1][ax[1]]
        p = (c2[0][ax[0]] + c2[1][ax[1]]) * np.float32(3 * u0 * u0 / 16)
        if dim == 3:
            vel[..., 0] *= c[2]
            vel[..., 1] *= c[2]
            p = p * (c2[2] + 2)
        rho += p
    else:
        flags[:, 0] = CellFlags.WALL
        flags[:, -1] = CellFlags.WALL
        x, y = np.arange(counts[0])[:, None], np.arange(counts[1])[None, :]
        disc = (x - counts[0] // 4) ** 2 + (y - counts[1] // 2) ** 2 <= (counts[1] / 12) ** 2
        flags[disc] = CellFlags.WALL
        flags[0, 1:-1] = CellFlags.FIXED_FLUID | CellFlags.FIXED_SCALAR_VALUE
        flags[-1, 1:-1] = CellFlags.FIXED_FLUID | CellFlags.FIXED_SCALAR_VALUE
        vel[..., 0] = u0
        inner = slice(1, -1)
        vel[inner] += _noise(seed, [counts[0] - 2] + counts[1:] + [dim], 1e-3)
        vel[flags == CellFlags.WALL] = 0.0
    val = None
    if case["tracer"]:
        val = _noise(seed + 1, counts, 0.5) + np.float32(0.5)
        val[:, : counts[1] // 3] *= 0.1
        if case["scene"] == "channel":
            val[0] = 0.0
            val[-1] = 0.0
    return flags, rho, vel, val


def _omega(case):
    return bgk(case["tau"]) if case["collision"] == "bgk" else trt(case["tau"], TAU_NEG)


def _gravity(dim):
    return np.array([0.0, -BUOYANCY, 0.0][:dim], np.float32)


def _prepare_sim(case, seed):
    dim = case["dim"]
    counts = [case["nx"], case["ny"], case["nz"]][:dim]
    t16 = case["tracer"] if case["tracer"] in ("f16", "bf16") else None
    sim = Simulation("gpu", counts, _omega(case), storage=case["storage"], tracer_storage=t16)
    flags, rho, vel, val = _fields(case, seed)
    sim.cells.flags[...] = flags
    sim.fluid.rho[...] = rho
    sim.fluid.vel[...] = vel
    tracer = None
    if val is not None:
        tracer = sim.add_tracer("tracer", bgk(TRACER_TAU))
        tracer.val[...] = val
        sim.add_boussinesq_coupling(tracer, 1.0, 0.0, _gravity(dim))
    sim.iterate(2)  # a running simulation: its fields are on the device
    return {"sim": sim, "tracer": tracer, "steps": case["steps"], "run": _run_sim}


def _run_sim(st):
    sim = st["sim"]
    sim.iterate(st["steps"])
    out = {"rho": sim.fluid.rho, "vel": sim.fluid.vel}
    if st["tracer"] is not None:
        out["val"] = st["tracer"].val
    return out


def _cavities(case, seed):
    rng = np.random.default_rng([seed, 23])
    # The sizes are the sweep's, the same for every seed; the flow in them is the seed's.
    sides = np.random.default_rng(case["domains"]).integers(case["lo"], case["hi"] + 1,
                                                            case["domains"])
    res = np.exp(rng.uniform(np.log(100.0), np.log(5000.0), case["domains"]))
    taus = [0.5 + 3.0 * 0.05 * int(side) / re for side, re in zip(sides, res)]
    return [int(s) for s in sides], [max(0.51, t) for t in taus]


def _prepare_ensemble(case, seed):
    sides, taus = _cavities(case, seed)
    ens = Ensemble([(s, s) for s in sides], tau=taus, storage=case["storage"])
    at = 0
    for s in sides:
        flags = ens.flags[at : at + s * s].reshape(s, s)
        vel = ens.vel[at : at + s * s].reshape(s, s, 2)
        flags[0, :] = flags[-1, :] = flags[:, 0] = CellFlags.WALL
        flags[1:-1, -1] = CellFlags.FIXED_FLUID
        vel[1:-1, -1, 0] = 0.05
        at += s * s
    ens.iterate(2, mode="persistent")
    return {"ens": ens, "steps": case["steps"], "run": _run_ensemble}


def _run_ensemble(st):
    ens = st["ens"]
    ens.iterate(st["steps"], mode="graph")
    return {"rho": ens.rho, "vel": ens.vel}


def _smooth(seed, nx, ny, count, scale):
    """``count`` smooth random fields [nx, ny] of that scale, on the device."""
    rng = np.random.default_rng([seed, nx, ny])
    x = torch.linspace(0, 2 * math.pi, nx, device="cuda")[:, None]
    y = torch.linspace(0, 2 * math.pi, ny, device="cuda")[None, :]
    out = torch.zeros(count, nx, ny, device="cuda")
    for k in range(count):
        for _ in range(6):
            a, b = rng.integers(1, 17, 2)
            p, q = rng.uniform(0, 2 * math.pi, 2)
            out[k] += torch.sin(float(a) * x + p) * torch.cos(float(b) * y + q)
    return out * (scale / 2.0)


def _channel_flags(nx, ny):
    flags = np.zeros((nx, ny), np.int32)
    flags[:, 0] = flags[:, -1] = CellFlags.WALL
    x, y = np.arange(nx)[:, None], np.arange(ny)[None, :]
    flags[(x - nx // 4) ** 2 + (y - ny // 2) ** 2 <= (ny / 32) ** 2] = CellFlags.WALL
    flags[0, 1:-1] = flags[-1, 1:-1] = CellFlags.FIXED_FLUID | CellFlags.FIXED_SCALAR_VALUE
    return flags


def _net(seed):
    # Means and inverse standard deviations of rho - 1, u_x, u_y, curl u in such a channel.
    norm = np.array([0.0, 0.05, 0.0, 0.0, 1e3, 60.0, 80.0, 400.0], np.float32)
    return cl.Net(cl.init_params(seed % 1000), norm, target_scale=2e-3, gain=3e-3)


def _prepare_train(case, seed):
    nx, ny, batch = case["nx"], case["ny"], case["batch"]
    stream = torch.cuda.current_stream().cuda_stream
    net = _net(seed)
    bufs = cl.Buffers(nx, ny, batch, train=True)
    flags = torch.tensor(_channel_flags(nx, ny), device="cuda")
    rho = 1.0 + _smooth(seed, nx, ny, batch, 1e-3)
    vel = torch.stack([_smooth(seed + 1, nx, ny, batch, 0.02) + 0.05,
                       _smooth(seed + 2, nx, ny, batch, 0.02)], dim=-1).contiguous()
    cl.features(rho, vel, flags, net.norm, bufs, stream)
    target = _smooth(seed + 3, nx, ny, batch, 1.0).abs().contiguous()
    opt = cl.Adam(net)
    opt.step_count = 200  # an optimiser in mid-run: its moments have seen many gradients
    g = torch.Generator(device="cuda").manual_seed(seed)
    opt.m.copy_((torch.rand(opt.m.shape, generator=g, device="cuda") - 0.5) * 2e-3)
    opt.v.fill_(1e-4)
    torch.cuda.synchronize()
    return {"net": net, "bufs": bufs, "x": bufs.x, "target": target, "flags": flags, "opt": opt,
            "stream": stream, "run": _run_train}


def _run_train(st):
    net, bufs = st["net"], st["bufs"]
    cl.forward(net, bufs, st["stream"], x=st["x"])
    cl.loss_and_grad(net, bufs, st["target"], st["flags"], st["stream"], x=st["x"])
    st["opt"].step(bufs.grad, st["stream"], lr=1e-3)
    return {"y": bufs.y, "loss": bufs.loss, "grad": bufs.grad, "params": net.params,
            "m": st["opt"].m, "v": st["opt"].v}


CLOSED_EVERY, CLOSED_TAU = 10, 0.505


def _closed_fields(case, seed):
    nx, ny = case["nx"], case["ny"]
    flags = _channel_flags(nx, ny)
    rho = 1.0 + _smooth(seed, nx, ny, 1, 1e-3)[0]
    vel = torch.stack([_smooth(seed + 1, nx, ny, 1, 0.01)[0] + 0.05,
                       _smooth(seed + 2, nx, ny, 1, 0.01)[0]], dim=-1)
    rho, vel = rho.cpu().numpy(), vel.cpu().numpy()
    wall, fixed = (flags & 1) != 0, (flags & 6) != 0
    rho[wall | fixed] = 1.0
    vel[wall] = 0.0
    vel[fixed] = (0.05, 0.0)
    val = _noise(seed + 3, [nx, ny], 0.5) + np.float32(0.5)
    val[fixed] = 0.0
    return flags, rho, vel, val


def _prepare_closed(case, seed):
    flags, rho, vel, val = _closed_fields(case, seed)
    sim = Simulation("gpu", list(flags.shape), trt(CLOSED_TAU, TAU_NEG))
    sim.cells.flags[...] = flags
    sim.fluid.rho[...] = rho
    sim.fluid.vel[...] = vel
    tracer = sim.add_tracer("tracer", bgk(TRACER_TAU))
    tracer.val[...] = val
    sim.add_boussinesq_coupling(tracer, 1.0, 0.0, _gravity(2))
    sim.iterate(2)
    closed = cl.ClosedRun(sim, flags, _net(seed), CLOSED_EVERY, CLOSED_TAU)
    return {"sim": sim, "closed": closed, "tracer": tracer, "steps": case["steps"],
            "run": _run_closed}


def _run_closed(st):
    st["closed"].advance(st["steps"])
    st["sim"]._read_back()
    return {"rho": st["sim"].fluid.rho, "vel": st["sim"].fluid.vel, "val": st["tracer"].val,
            "omega": st["closed"].omega}


_PREPARE = {"sim": _prepare_sim, "ensemble": _prepare_ensemble, "train": _prepare_train,
            "closed": _prepare_closed}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


# ---- what a pass cannot do without ----------------------------------------------------------

_BYTES = {"f32": 4, "f16": 2, "bf16": 2, "f64": 8, "": 0}
_NET_FLOPS = 2 * (36 * 32 + 288 * 32 + 288)  # per cell, forward


def work(case):
    """The state read once and written once a call, whatever its steps: a method that keeps a
    part of the domain on the chip over several steps needs no more. Operations: about 9 a
    population for its moments and collision."""
    if case["kind"] == "sim":
        d, cells = case["dim"], case["nx"] * case["ny"] * case["nz"]
        q, qt = (9, 5) if d == 2 else (27, 7)
        pops = q * _BYTES[case["storage"]] + qt * _BYTES[case["tracer"]]
        fields = 4 * (1 + d + (1 if case["tracer"] else 0)) + 1
        return {"bytes": cells * (2 * pops + fields),
                "flops": 9 * cells * case["steps"] * (q + (qt if case["tracer"] else 0))}
    if case["kind"] == "ensemble":
        cells = sum(s * s for s in _cavities(case, 0)[0])
        return {"bytes": cells * (18 * _BYTES[case["storage"]] + 13),
                "flops": 81 * cells * case["steps"]}
    cells = case["nx"] * case["ny"]
    if case["kind"] == "train":
        # Features, targets, predictions; the backward pass is twice the forward's products
        # (no input gradient in the first layer).
        n = cells * case["batch"]
        return {"bytes": n * (8 + 4 + 4) + cells * 4,
                "flops": n * (3 * _NET_FLOPS - 2 * 36 * 32)}
    return {"bytes": cells * (2 * 56 + 16 + 1 + 4),
            "flops": cells * (9 * 14 * case["steps"] + _NET_FLOPS * (case["steps"] // CLOSED_EVERY))}


# ---- the same in 64 bits --------------------------------------------------------------------


def _lattice(dim, tracer):
    """Velocities and weights in the framework's slot order: opposite directions adjacent."""
    half2 = [(1, 0), (0, 1), (1, 1), (1, -1)]
    half3 = [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, -1, 0), (1, 0, 1), (0, 1, 1),
             (1, 0, -1), (0, 1, -1), (1, 1, 1), (1, -1, 1), (1, 1, -1), (1, -1, -1)]
    half = (half2 if dim == 2 else half3)[: dim if tracer else None]
    c = [(0,) * dim]
    for h in half:
        c += [h, tuple(-v for v in h)]
    if tracer:
        w = {2: {0: 1 / 3, 1: 1 / 6}, 3: {0: 1 / 20, 1: 19 / 120}}[dim]
    else:
        w = {2: {0: 4 / 9, 1: 1 / 9, 2: 1 / 36},
             3: {0: 8 / 27, 1: 2 / 27, 2: 1 / 54, 3: 1 / 216}}[dim]
    return c, [w[sum(abs(a) for a in v)] for v in c]


def _upstream(counts, c):
    """Flat index of the cell upstream of c for every cell of a periodic domain."""
    idx = torch.zeros([1] * len(counts), dtype=torch.int64, device="cuda")
    for a, n in enumerate(counts):
        shape = [1] * len(counts)
        shape[a] = n
        idx = idx * n + ((torch.arange(n, device="cuda") - c[a]) % n).reshape(shape)
    return idx.reshape(-1)


def _opp(i):
    return 0 if i == 0 else (i + 1 if i % 2 else i - 1)


class _Exact:
    """The lattice-Boltzmann method of one or several domains in doubles: in-place streaming
    (even steps exchange with the neighbours, odd steps locally), walls never updated."""

    def __init__(self, domains, flags, rho, vel, om_pos, om_neg, trt_, val=None, om_tracer=0.0,
                 force=None):
        dim = vel.shape[-1]
        dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
        self.flags = dev(flags).reshape(-1)
        self.wall = (self.flags & 1) != 0
        self.fixed = (self.flags & 6) != 0
        self.tfixed = (self.flags & 8) != 0
        self.rho = dev(rho).double().reshape(-1)
        self.vel = dev(vel).double().reshape(-1, dim)
        self.c, self.w = _lattice(dim, False)
        self.up = [self._all_up(domains, c) for c in self.c]
        self.om_pos, self.om_neg, self.trt = om_pos, om_neg, trt_
        self.f = self._equilibria(self.c, self.w, self.rho, self.vel)
        self.force, self.val, self.field = force, None, None
        if val is not None:
            self.val = dev(val).double().reshape(-1)
            self.tc, self.tw = _lattice(dim, True)
            self.tup = [self.up[self.c.index(c)] for c in self.tc]
            self.om_tracer = om_tracer
            self.g = self._equilibria(self.tc, self.tw, self.val, self.vel)

    @staticmethod
    def _all_up(domains, c):
        out, at = [], 0
        for counts in domains:
            out.append(_upstream(counts, c) + at)
            at += math.prod(counts)
        return out[0] if len(out) == 1 else torch.cat(out)

    @staticmethod
    def _eq(c, w, r, u, uu):
        cu = sum(u[:, a] * v for a, v in enumerate(c) if v) if any(c) else torch.zeros_like(r)
        return w * r * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * uu)

    def _equilibria(self, cs, ws, r, u):
        uu = (u * u).sum(1)
        return [self._eq(c, w, r, u, uu) for c, w in zip(cs, ws)]

    def _advance(self, f, cs, ws, up, even, moments, om_pos, om_neg, trt_):
        """One step of one velocity set in place; ``moments(loaded)`` gives r, u."""
        v = [f[i][up[i]] if even else f[_opp(i)] for i in range(len(cs))]
        r, u = moments(v)
        uu = (u * u).sum(1)
        post = []
        for i in range(len(cs)):
            j = _opp(i)
            e = self._eq(cs[i], ws[i], r, u, uu)
            if trt_:
                ej = self._eq(cs[j], ws[j], r, u, uu)
                post.append(v[i] + om_pos * ((e + ej) - (v[i] + v[j])) / 2
                            + om_neg * ((e - ej) - (v[i] - v[j])) / 2)
            else:
                post.append(v[i] + om_pos * (e - v[i]))
        new = []
        for i in range(len(cs)):
            if even:
                p = torch.where(self.wall, f[i][up[i]], post[_opp(i)])
                out = torch.empty_like(p)
                out[up[i]] = p
                new.append(out)
            else:
                new.append(torch.where(self.wall, f[i], post[i]))
        return new, r, u

    def step(self, even):
        keep = self.wall | self.fixed

        def fluid(v):
            r = sum(v)
            m = torch.stack([sum(v[i] * c[a] for i, c in enumerate(self.c) if c[a])
                             for a in range(self.vel.shape[1])], dim=1)
            u = m / r[:, None]
            if self.force is not None:
                u = u + self.val[:, None] * self.force
            r = torch.where(self.fixed, self.rho, r)
            return r, torch.where(self.fixed[:, None], self.vel, u)

        om_p = self.om_pos if self.field is None else self.field
        om_p = torch.where(self.fixed, torch.ones_like(self.rho), om_p)
        om_n = torch.where(self.fixed, torch.ones_like(self.rho), self.om_neg)
        self.f, r, u = self._advance(self.f, self.c, self.w, self.up, even, fluid, om_p, om_n,
                                     self.trt)
        if self.val is not None:
            om = torch.where(self.tfixed, torch.ones_like(self.rho), self.om_tracer)
            self.g, t, _ = self._advance(
                self.g, self.tc, self.tw, self.tup, even,
                lambda v: (torch.where(self.tfixed, self.val, sum(v)), u), om, om, False)
            self.val = torch.where(self.wall, self.val, t)
        self.rho = torch.where(keep, self.rho, r)
        self.vel = torch.where(keep[:, None], self.vel, u)

    def steps(self, n):
        for k in range(n):
            self.step(k % 2 == 0)


def _f32(v):
    return float(np.float32(v))


def _exact_sim(case, seed):
    dim = case["dim"]
    counts = [case["nx"], case["ny"], case["nz"]][:dim]
    flags, rho, vel, val = _fields(case, seed)
    om = _f32(1.0 / case["tau"])
    force = None
    if val is not None:
        force = torch.as_tensor(_gravity(dim), device="cuda").double() / om
    one = torch.ones((), dtype=torch.float64, device="cuda")
    e = _Exact([counts], flags, rho, vel, om * one, _f32(1.0 / TAU_NEG) * one,
               case["collision"] == "trt", val, _f32(1.0 / TRACER_TAU) * one, force)
    e.steps(2 + case["steps"])
    out = {"rho": e.rho.reshape(counts), "vel": e.vel.reshape(counts + [dim])}
    if val is not None:
        out["val"] = e.val.reshape(counts)
    return out


def _exact_ensemble(case, seed):
    sides, taus = _cavities(case, seed)
    flags, vel, om = [], [], []
    for s, tau in zip(sides, taus):
        fl, v = np.zeros((s, s), np.int32), np.zeros((s, s, 2), np.float32)
        fl[0, :] = fl[-1, :] = fl[:, 0] = CellFlags.WALL
        fl[1:-1, -1] = CellFlags.FIXED_FLUID
        v[1:-1, -1, 0] = 0.05
        flags.append(fl.reshape(-1))
        vel.append(v.reshape(-1, 2))
        om.append(np.full(s * s, np.float32(1.0 / tau), np.float64))
    flags = np.concatenate(flags)
    om = torch.as_tensor(np.concatenate(om), device="cuda")
    e = _Exact([[s, s] for s in sides], flags, np.ones(flags.size, np.float32),
               np.concatenate(vel), om, om, False)
    e.steps(2 + case["steps"])
    return {"rho": e.rho, "vel": e.vel}


def _net64(params):
    """Layer weights of a parameter vector, as doubles in torch's layout."""
    p = torch.as_tensor(params).detach().double().cuda()
    at, out = 0, []
    for co, ci in ((32, 4), (32, 32), (1, 32)):
        w = p[at : at + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2).contiguous()
        at += co * 9 * ci
        out.append((w, p[at : at + co].clone()))
        at += co
    return out


def _forward64(layers, x):
    conv = torch.nn.functional.conv2d
    h = x
    for k, (w, b) in enumerate(layers):
        h = conv(h, w, b, padding=1)
        if k < 2:
            h = torch.nn.functional.gelu(h, approximate="tanh")
    return h[:, 0]


def _exact_train(case, seed):
    st = _prepare_train(case, seed)
    nx, ny, batch = case["nx"], case["ny"], case["batch"]
    x = st["x"].view(torch.bfloat16).double().reshape(batch, nx, ny, 4).permute(0, 3, 1, 2)
    fluid = (st["flags"] & 7) == 0
    layers = [(w.requires_grad_(), b.requires_grad_()) for w, b in _net64(st["net"].params)]
    total = float(fluid.sum()) * batch
    ys, loss = [], 0.0
    for k in range(batch):  # one sample at a time: the gradients add up
        y = _forward64(layers, x[k : k + 1].contiguous())
        part = ((y[0] - st["target"][k].double())[fluid] ** 2).sum() / total
        part.backward()
        ys.append(y[0].detach())
        loss += part.detach()
    grad = torch.cat([t for w, b in layers
                      for t in (w.grad.permute(0, 2, 3, 1).reshape(-1), b.grad.reshape(-1))])
    opt = st["opt"]
    b1, b2 = opt.betas
    m = b1 * opt.m.double() + (1 - b1) * grad
    v = b2 * opt.v.double() + (1 - b2) * grad * grad
    t = opt.step_count + 1
    step = 1e-3 * (m / (1 - b1**t)) / ((v / (1 - b2**t)).sqrt() + opt.eps)
    return {"y": torch.stack(ys).reshape(-1), "loss": loss.reshape(1), "grad": grad,
            "params": st["net"].params.double() - step, "m": m, "v": v}


def _gradient64(f, dim):
    """np.gradient with unit spacing."""
    lo, hi = f.narrow(dim, 0, 1), f.narrow(dim, f.shape[dim] - 1, 1)
    n = f.shape[dim]
    inner = (f.narrow(dim, 2, n - 2) - f.narrow(dim, 0, n - 2)) / 2
    return torch.cat([f.narrow(dim, 1, 1) - lo, inner, hi - f.narrow(dim, n - 2, 1)], dim)


def _exact_closed(case, seed):
    nx, ny = case["nx"], case["ny"]
    flags, rho, vel, val = _closed_fields(case, seed)
    om = _f32(1.0 / CLOSED_TAU)
    one = torch.ones((), dtype=torch.float64, device="cuda")
    force = torch.as_tensor(_gravity(2), device="cuda").double() / om
    e = _Exact([[nx, ny]], flags, rho, vel, om * one, _f32(1.0 / TAU_NEG) * one, True, val,
               _f32(1.0 / TRACER_TAU) * one, force)
    e.steps(2)
    net = _net(seed)
    layers = _net64(net.params)
    wall = e.wall.reshape(nx, ny)
    fluid = (e.flags & 7) == 0
    mean, inv = torch.as_tensor(net.norm, device="cuda").double().reshape(2, 4)
    for _ in range(case["steps"] // CLOSED_EVERY):
        u = e.vel.reshape(nx, ny, 2)
        still = torch.where(wall[..., None], torch.zeros_like(u), u)
        curl = _gradient64(still[..., 0], 1) - _gradient64(still[..., 1], 0)
        x = torch.stack([e.rho.reshape(nx, ny) - 1, u[..., 0], u[..., 1], curl], dim=-1)
        x = torch.where(wall[..., None], torch.zeros_like(x), (x - mean) * inv)
        y = _forward64(layers, x.permute(2, 0, 1)[None].contiguous())[0].reshape(-1)
        extra = (net.gain * y.clamp_min(0)).clamp_max(net.max_dtau)
        omega = 1 / (CLOSED_TAU + torch.where(fluid, extra, torch.zeros_like(extra)))
        e.field = omega
        e.steps(CLOSED_EVERY)
    return {"rho": e.rho.reshape(nx, ny), "vel": e.vel.reshape(nx, ny, 2),
            "val": e.val.reshape(nx, ny), "omega": omega}


def exact(case, seed):
    if not torch.cuda.is_available():
        return None
    return {"sim": _exact_sim, "ensemble": _exact_ensemble, "train": _exact_train,
            "closed": _exact_closed}[case["kind"]](case, seed)
