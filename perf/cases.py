"""The work a user of this framework has it do, as cases that can be timed.

Five paths, each through the public entry points:

  call      tslb_step_noalloc on caller-owned device buffers (FP32): a host
            that owns its device memory steps its state in place of the
            library; the output is the whole state after the steps
  run       a Lattice: steps with the FP64 diagnostics of every step queued,
            and the print stamp of the reference's drivers (rho, u, v, w,
            phi to page-locked host memory) at the end
  ensemble  droplet-in-Couette domains of uneven size, steps replayed from a
            CUDA graph, and phi of every domain (the deformation study)
  jet       the round jet with sponge, device-drawn inlet and the learned
            closure refreshed every second step, and the print stamp
  train     Adam steps of the closure's network on a device training set

The lattice sizes are those of the workloads, tests and benchmark of this
repository (the 24^3 and 64^3 droplet, the 384 x 192 x 128 channel, the
192 x 192 x 384 jet, 48 Couette domains of 48..128 x 32..96 x 32..96) and odd
sizes between them.
"""
import ctypes
import math
import random

import numpy as np
import torch

from entropicthreadsafe_b200 import capi, workloads
from entropicthreadsafe_b200.closure import Closure, init_params, lattice_attach, trained_closure
from entropicthreadsafe_b200.ensemble import Ensemble
from entropicthreadsafe_b200.solver import Lattice, TslbError

DEV = "cuda"
NF = 11
MODES = {"phase": capi.MODE_PHASEFIELD, "colour": capi.MODE_COLOUR, "single": capi.MODE_SINGLE}
PRECS = {"fp32": capi.PREC_FP32, "bf16": capi.PREC_BF16, "fp16s": capi.PREC_FP16S}
STAMP = ("rho", "u", "v", "w", "phi")


def _lattice(name, path, mode, nx, ny, nz, steps, walls="periodic", precision="fp32", obstacle=False):
    c = dict(path=path, mode=mode, nx=nx, ny=ny, nz=nz, steps=steps, walls=walls, precision=precision, obstacle=obstacle)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: one step of a small periodic droplet, where launch and host latency count
        _lattice("call_droplet_24", "call", "colour", 24, 24, 24, 1),
        # the static-droplet (Laplace) benchmark size
        _lattice("call_droplet_64", "call", "colour", 64, 64, 64, 10),
        # the headline workload: two-component channel with bounce-back walls, body force, 40 droplets
        _lattice("call_channel", "call", "colour", 384, 192, 128, 4, "channel"),
        # the reference program's own operator (phase field, D3Q7 + CSF) on the same channel
        _lattice("call_channel_phase", "call", "phase", 384, 192, 128, 2, "channel"),
        # single-component channel
        _lattice("call_channel_single", "call", "single", 384, 192, 128, 2, "channel"),
        # odd sizes, moving walls, viscosity ratio (a Couette cell as a user cuts it, no multiple of any tile)
        _lattice("call_couette_ragged", "call", "colour", 173, 59, 91, 4, "couette"),
        # closed box with an obstacle in it, odd sizes, phase field, diagnostics and print stamp
        _lattice("run_obstacle_phase", "run", "phase", 101, 64, 47, 20, "box", obstacle=True),
        # the channel in BF16 storage with diagnostics every step and a print stamp
        _lattice("run_channel_bf16", "run", "colour", 384, 192, 128, 10, "channel", "bf16"),
        # a smaller channel in scaled FP16 storage
        _lattice("run_channel_fp16s", "run", "colour", 192, 96, 64, 10, "channel", "fp16s"),
        # 48 droplet-in-Couette domains advanced together
        dict(name="ensemble_couette_48", path="ensemble", members=48, sizes=2024, steps=20),
        # the coarse round jet with the packaged closure
        dict(name="jet_closure", path="jet", nx=192, ny=192, nz=384, steps=10),
        # training the closure: forward, backward and Adam on the tensor cores
        dict(name="train_closure", path="train", samples=262144, batch=16384, steps=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.random()
    if kind < 0.55:
        mode = rng.choice(["colour", "colour", "phase", "single"])
        walls = rng.choice(["periodic", "channel", "box", "couette"] if mode == "colour" else ["periodic", "channel", "box"])
        while True:
            nx, ny, nz = _log(rng, 16, 400), _log(rng, 16, 256), _log(rng, 16, 256)
            if nx * ny * nz <= 8_000_000:
                return _lattice(None, "call", mode, nx, ny, nz, rng.randint(1, 4), walls)
    if kind < 0.8:
        mode = rng.choice(["colour", "colour", "phase"])
        prec = rng.choice(["fp32", "bf16", "fp16s"]) if mode == "colour" else "fp32"
        walls = rng.choice(["channel", "box"])
        while True:
            nx, ny, nz = _log(rng, 24, 256), _log(rng, 24, 192), _log(rng, 24, 128)
            if nx * ny * nz <= 3_000_000:
                return _lattice(None, "run", mode, nx, ny, nz, rng.randint(4, 10), walls, prec,
                                prec == "fp32" and rng.random() < 0.4)
    if kind < 0.9:
        return dict(path="ensemble", members=rng.randint(4, 40), sizes=rng.randrange(1 << 20), steps=2 * rng.randint(2, 8))
    if kind < 0.95:
        return dict(path="jet", nx=_log(rng, 64, 192), ny=_log(rng, 64, 192), nz=_log(rng, 96, 384), steps=2 * rng.randint(2, 5))
    return dict(path="train", samples=_log(rng, 1 << 14, 1 << 18), batch=128 * _log(rng, 8, 128), steps=rng.randint(10, 40))


# ---------------------------------------------------------------- inputs

def _params(case):
    """The lattice's parameters as keywords of capi.make_params."""
    mode, walls = case["mode"], case["walls"]
    phase = mode == "phase"
    kw = dict(mode=MODES[mode], precision=PRECS[case["precision"]], beta=0.7, sharp_c=0.9, grad_threshold=1e-3,
              bc_phi=[0.0 if phase else -1.0] * 6, wall_phi_mode=1, force=(0.0, 0.0, 0.0),
              bc=[capi.BC_PERIODIC] * 6, bc_u=[[0.0] * 3] * 6)
    if walls == "channel":
        tau = 3 * 0.0015 + 0.5
        kw.update(tau_a=tau, tau_b=tau, sigma=0.005, force=(2.5e-6, 0.0, 0.0),
                  bc=[capi.BC_PERIODIC] * 4 + [capi.BC_BOUNCEBACK] * 2)
    elif walls == "couette":
        kw.update(tau_a=1.4, tau_b=0.9, sigma=0.002, bc=[capi.BC_PERIODIC] * 4 + [capi.BC_VELOCITY] * 2,
                  bc_u=[[0.0] * 3] * 4 + [[-0.05, 0.0, 0.0], [0.05, 0.0, 0.0]])
    else:
        kw.update(tau_a=0.8, tau_b=0.8, sigma=0.01, bc=[capi.BC_BOUNCEBACK if walls == "box" else capi.BC_PERIODIC] * 6)
    return kw


def _axes(nx, ny, nz):
    f = dict(dtype=torch.float32, device=DEV)
    return torch.arange(nx, **f).view(1, 1, -1), torch.arange(ny, **f).view(1, -1, 1), torch.arange(nz, **f).view(-1, 1, 1)


def _drops(nx, ny, nz, centres, radius):
    """phi in [-1, 1]: 1 inside the droplets (periodic distance in x and y)."""
    x, y, z = _axes(nx, ny, nz)
    phi = torch.full((nz, ny, nx), -1.0, device=DEV)
    for cx, cy, cz in centres:
        dx, dy = (x - cx).abs(), (y - cy).abs()
        r2 = torch.minimum(dx, nx - dx) ** 2 + torch.minimum(dy, ny - dy) ** 2 + (z - cz) ** 2
        phi = torch.maximum(phi, torch.tanh((radius - r2.sqrt()) / 2.0))
    return phi


def _state(case, seed):
    """(11, nz, ny, nx) FP32 moments on the GPU (row 0 is rho - 1): a mean flow
    with 5% noise, the small density and stress fluctuations of a running
    flow, and droplets."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    r = random.Random(int(seed))
    s = torch.empty((NF, nz, ny, nx), device=DEV)
    s[0].normal_(0.0, 2e-4, generator=g)
    z = _axes(nx, ny, nz)[2]
    walls = case["walls"]
    u0 = 0.05
    prof = 4.0 * (z + 0.5) * (nz - z - 0.5) / nz ** 2 if walls == "channel" else 2.0 * (z + 0.5) / nz - 1.0
    for k in (1, 2, 3):
        s[k].uniform_(-0.05 * u0, 0.05 * u0, generator=g)
    if walls in ("channel", "couette"):
        s[1] += u0 * prof
    s[4:10].normal_(0.0, 2e-5, generator=g)
    if case["precision"] == "fp16s":
        # the channel workload's start, rho = 1 and no stress: the upload then
        # keeps the scales meant for a running flow
        s[0] = 0.0
        s[4:10] = 0.0
    if case["mode"] == "single":
        s[10] = 1.0
    else:
        radius = min(8.0, 0.22 * min(nx, ny, nz))
        count = max(1, min(40, int(0.02 * nx * ny * nz / (4.2 * radius ** 3))))
        gap = 1.5 * radius
        cen = [(r.uniform(0, nx), r.uniform(0, ny), r.uniform(min(gap, nz / 2), max(nz - gap, nz / 2))) for _ in range(count)]
        phi = _drops(nx, ny, nz, cen, radius)
        s[10] = 0.5 * (1.0 + phi) if case["mode"] == "phase" else phi
    return s


def _obstacle(case):
    """isfluid of a solid sphere off the middle of the box, (nz, ny, nx) uint8 on the GPU."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    x, y, z = _axes(nx, ny, nz)
    r = 0.15 * min(nx, ny, nz)
    inside = (x - 0.35 * nx) ** 2 + (y - 0.5 * ny) ** 2 + (z - 0.4 * nz) ** 2 <= r * r
    return (~inside).to(torch.uint8)


def _host_fields(s):
    """The state as the dict of host arrays that upload_moments takes."""
    h = s.cpu()
    h[0] += 1.0
    return {k: h[i].numpy() for i, k in enumerate(capi.FIELDS)}


def _members(case, seed):
    """The domains' sizes (from the case) and droplets (from the seed)."""
    rs, r = random.Random(int(case["sizes"])), random.Random(int(seed))
    out = []
    for _ in range(case["members"]):
        lx, lz = 8 * rs.randint(6, 16), 8 * rs.randint(4, 12)
        radius, ca, lam = r.uniform(0.2, 0.3) * lz, r.uniform(0.1, 0.5), r.uniform(1.0, 4.0)
        nu = 0.5 / 3.0
        sigma = nu * (2.0 * 0.05 / lz) * radius / ca
        kw = dict(mode=capi.MODE_COLOUR, precision=capi.PREC_FP32, tau_a=3.0 * lam * nu + 0.5, tau_b=1.0, sigma=sigma,
                  beta=0.7, grad_threshold=1e-3, force=(0.0, 0.0, 0.0), bc=[capi.BC_PERIODIC] * 4 + [capi.BC_VELOCITY] * 2,
                  bc_u=[[0.0] * 3] * 4 + [[-0.05, 0.0, 0.0], [0.05, 0.0, 0.0]], bc_phi=[-1.0] * 6, wall_phi_mode=1)
        out.append((kw, (lx, lz, lz), radius))
    return out


def _member_state(dims, radius):
    nx, ny, nz = dims
    s = torch.zeros((NF, nz, ny, nx), device=DEV)
    s[1] = 0.05 * (2.0 * (_axes(nx, ny, nz)[2] + 0.5) / nz - 1.0)
    s[10] = _drops(nx, ny, nz, [((nx - 1) / 2, (ny - 1) / 2, (nz - 1) / 2)], radius)
    return s


def _jet_state(case, seed):
    """A developed jet column: phi and w smooth across the disc's edge, 3% noise."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    x, y, z = _axes(nx, ny, nz)
    edge = torch.tanh((8.0 - ((x - nx / 2 + 0.5) ** 2 + (y - ny / 2 + 0.5) ** 2).sqrt()) / 2.0)
    inside = (edge * torch.ones_like(z)).contiguous()
    s = torch.zeros((NF, nz, ny, nx), device=DEV)
    for k in (1, 2, 3):
        s[k].uniform_(-0.03 * 0.08, 0.03 * 0.08, generator=g)
        s[k] *= 0.5 * (1.0 + inside)
    s[3] += 0.04 * (1.0 + inside)
    s[10] = inside
    return s


def _train_set(case, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    n = case["samples"]
    scale = torch.tensor([1e-4] * 6 + [1.0, 0.3, 0.05, 2e-4], device=DEV)
    f = torch.randn((n, 10), device=DEV, generator=g) * scale
    f[:, 7:] = f[:, 7:].abs()
    t = 0.01 * torch.sigmoid(2.0 * f[:, 9] / 2e-4 - 2.0) * torch.rand(n, device=DEV, generator=g)
    w = torch.rand(n, device=DEV, generator=g) + 0.5
    return f, t, w


def _ptr(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_float))


class _Pointers:
    """Field pointers into one page-locked (k, n) buffer, in the order of capi.FIELDS, NULL where none is wanted."""

    def __init__(self, buf, names):
        at = {k: _ptr(buf[i]) for i, k in enumerate(names)}
        self.args = [at.get(k) for k in capi.FIELDS]


def prepare(case, seed):
    path = case["path"]
    L = capi.lib()
    if path == "call":
        s = _state(case, seed)
        n = s[0].numel()
        stride = (n + 31) // 32 * 32
        bufs = [torch.zeros((NF, stride), device=DEV) for _ in range(3)]
        bufs[0][:, :n] = s.view(NF, n)
        if case["mode"] == "single":
            for b in bufs:
                b[10] = 1.0   # not stepped: held at 1 in every buffer
        p = capi.make_params(**_params(case))
        return dict(case=case, L=L, bufs=bufs, p=p, stride=stride)
    if path == "run":
        lat = Lattice(capi.make_params(**_params(case)), case["nx"], case["ny"], case["nz"])
        if case["obstacle"]:
            lat.set_solid_mask(_obstacle(case).cpu().numpy())
        lat.upload_moments(_host_fields(_state(case, seed)))
        stamp = torch.empty((len(STAMP), lat.n), dtype=torch.float32, pin_memory=True)
        return dict(case=case, L=L, lat=lat, stamp=stamp, to=_Pointers(stamp, STAMP))
    if path == "ensemble":
        m = _members(case, seed)
        ens = Ensemble([capi.make_params(**kw) for kw, _, _ in m], [d for _, d, _ in m])
        for i, (_, dims, radius) in enumerate(m):
            ens.upload_moments(i, _host_fields(_member_state(dims, radius)))
        sizes = [a * b * c for _, (a, b, c), _ in m]
        phi = torch.empty(sum(sizes), dtype=torch.float32, pin_memory=True)
        parts = list(torch.split(phi, sizes))
        return dict(case=case, L=L, ens=ens, phi=phi, to=[_Pointers(v.view(1, -1), ("phi",)) for v in parts])
    if path == "jet":
        p, _, spec = workloads.jet(1, nx=case["nx"], ny=case["ny"], nz=case["nz"])
        lat, clo = Lattice(p, case["nx"], case["ny"], case["nz"]), trained_closure()
        lat.upload_moments(_host_fields(_jet_state(case, seed)))
        lat.set_tau_correction(workloads.jet_sponge(spec))
        lattice_attach(lat, clo, 2)
        stamp = torch.empty((len(STAMP), lat.n), dtype=torch.float32, pin_memory=True)
        return dict(case=case, L=L, lat=lat, closure=clo, spec=spec, seed=int(seed), at=0, stamp=stamp, to=_Pointers(stamp, STAMP))
    f, t, w = _train_set(case, seed)
    clo = Closure()
    clo.set_params(init_params(0), np.zeros(10), np.array([1e-4] * 6 + [1.0, 0.3, 0.05, 2e-4]), 0.02)
    clo.dataset_add(f.cpu().numpy(), t.cpu().numpy(), w.cpu().numpy())
    return dict(case=case, closure=clo, seed=int(seed) % (1 << 31))


def _stamp(state):
    """The print stamp of the reference's drivers; 16-bit runs keep 16-bit stamps."""
    lat, stamp = state["lat"], state["stamp"]
    rc = state["L"].tslb_download_moments(lat.h, *state["to"].args)
    if rc != capi.OK:
        raise TslbError(rc, state["L"].tslb_last_error(lat.h).decode())
    prec = state["case"].get("precision", "fp32")
    if prec == "fp32":
        return {"stamp": stamp}
    if prec == "bf16":   # the stored fields are BF16 numbers: the upper halves of their FP32 words
        return {"stamp": stamp.view(torch.bfloat16)[:, 1::2]}
    return {"stamp": stamp.to(torch.float16)}


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "call":
        L, p, bufs = state["L"], ctypes.addressof(state["p"]), state["bufs"]
        stream = torch.cuda.current_stream().cuda_stream
        src = 0
        for k in range(case["steps"]):
            dst = 1 + k % 2
            rc = L.tslb_step_noalloc(p, case["nx"], case["ny"], case["nz"], bufs[src].data_ptr(), bufs[dst].data_ptr(),
                                     state["stride"], stream)
            if rc != capi.OK:
                raise TslbError(rc, L.tslb_last_error(None).decode())
            src = dst
        return bufs[src]
    if path == "run":
        lat = state["lat"]
        for _ in range(case["steps"]):
            lat.step(1)
            lat.reduce_async()
        diag = lat.reduce_collect()
        out = _stamp(state)
        # totals over the lattice, one row a step, as a log keeps them
        kind = torch.float32 if case["precision"] == "fp32" else torch.bfloat16
        out["totals"] = torch.tensor([[d["mass"], d["mass_a"], d["kinetic"]] for d in diag], dtype=kind)
        return out
    if path == "ensemble":
        ens, L = state["ens"], state["L"]
        ens.step_graph(case["steps"])
        for i, to in enumerate(state["to"]):
            rc = L.tslb_ensemble_download_moments(ens.h, i, *to.args)
            if rc != capi.OK:
                raise TslbError(rc, L.tslb_ensemble_last_error(ens.h).decode())
        return {"phi": state["phi"]}
    if path == "jet":
        lat, spec = state["lat"], state["spec"]
        for _ in range(case["steps"]):
            if state["at"] % spec["refresh"] == 0:
                workloads.jet_inlet(lat, spec, state["seed"], state["at"])
            lat.step(1)
            state["at"] += 1
        return _stamp(state)
    clo = state["closure"]
    hist = clo.train(case["steps"], case["batch"], 2e-3, state["seed"])
    return {"loss": hist, "params": clo.get_params()["params"]}


def work(case):
    path = case["path"]
    if path == "train":
        rows = case["batch"] * case["steps"]
        net = 10 * 64 + 64 * 64 + 64
        return {"bytes": rows * 4 * 12 + case["steps"] * 4 * 5313 * 6, "flops": rows * 6 * net}
    if path == "ensemble":
        n = sum(a * b * c for _, (a, b, c), _ in _members(case, 0))
        return {"bytes": n * (88 * case["steps"] + 4), "flops": n * case["steps"] * 700}
    n = case["nx"] * case["ny"] * case["nz"]
    k = case["steps"]
    if path == "jet":
        # the closure reads the 10 moments of its features and writes dtau, every second step
        return {"bytes": n * (92 * k + 52 * ((k + 1) // 2) + 4 * len(STAMP)), "flops": n * (700 * k + 10240 * ((k + 1) // 2))}
    per = {"single": 80}.get(case["mode"], 88)
    if case["precision"] != "fp32":
        per //= 2
    # every step reads the moments once and writes them once; the stamp is written to the host
    return {"bytes": n * (per * k + (4 * len(STAMP) if path == "run" else 0)), "flops": n * k * 700}


# ---------------------------------------------------------------- 64-bit reference
# The step written population by population from its definition, in FP64.

_C = [(cx, cy, cz) for cz in (-1, 0, 1) for cy in (-1, 0, 1) for cx in (-1, 0, 1)]
_W = {0: 8.0 / 27.0, 1: 2.0 / 27.0, 2: 1.0 / 54.0, 3: 1.0 / 216.0}


def _pad(a, periodic, wall):
    """One ghost layer on each side: wrapped, or `wall` ("edge": the nearest node, "zero")."""
    for dim, per in ((2, periodic[0]), (1, periodic[1]), (0, periodic[2])):
        lo, hi = a.narrow(dim, 0, 1), a.narrow(dim, a.shape[dim] - 1, 1)
        if per:
            lo, hi = hi, lo
        elif wall == "zero":
            lo, hi = torch.zeros_like(lo), torch.zeros_like(hi)
        a = torch.cat([lo, a, hi], dim)
    return a


def _grad(p, comps=(0, 1, 2)):
    """Isotropic gradient 3 sum w_c c s(x + c) of a padded field."""
    nz, ny, nx = (k - 2 for k in p.shape)
    g = [0.0, 0.0, 0.0]
    for c in _C:
        c2 = sum(k * k for k in c)
        if c2 == 0 or not any(c[a] for a in comps):
            continue
        v = p[1 + c[2]:1 + c[2] + nz, 1 + c[1]:1 + c[1] + ny, 1 + c[0]:1 + c[0] + nx] * (3.0 * _W[c2])
        for a in comps:
            if c[a]:
                g[a] = g[a] + c[a] * v
    return g


def _herm(c):
    t = 1.0 / 3.0
    x, y, z = (float(k) for k in c)
    h2 = (x * x - t, x * y, x * z, y * y - t, y * z, z * z - t)
    h3 = ((x * x - t) * y, (x * x - t) * z, (y * y - t) * x, (y * y - t) * z, (z * z - t) * x, (z * z - t) * y, x * y * z)
    return h2, h3


def _combine(coef, terms):
    out = 0.0
    for k, t in zip(coef, terms):
        if k != 0.0:
            out = out + k * t
    return out


def _eq_terms(u, v, w):
    return (u * u * v, u * u * w, u * v * v, v * v * w, u * w * w, v * w * w, u * v * w)


def _feq(c, rho, u, v, w, cubic):
    """f^eq / w, third-order Hermite form."""
    _, h3 = _herm(c)
    cu = _combine(c, (u, v, w))
    uu = u * u + v * v + w * w
    s = _combine([13.5 * k for k in h3[:6]] + [27.0 * h3[6]], cubic)
    return rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * uu + s)


def _fneq(c, P, third):
    h2, h3 = _herm(c)
    a = _combine((4.5 * h2[0], 9.0 * h2[1], 9.0 * h2[2], 4.5 * h2[3], 9.0 * h2[4], 4.5 * h2[5]), P)
    return a + _combine([13.5 * k for k in h3[:6]] + [27.0 * h3[6]], third)


def _third(P, u, v, w):
    xx, xy, xz, yy, yz, zz = P
    return (2 * u * xy + v * xx, 2 * u * xz + w * xx, u * yy + 2 * v * xy, 2 * v * yz + w * yy, u * zz + 2 * w * xz,
            v * zz + 2 * w * yz, u * yz + v * xz + w * xy)


def _f32(x):
    return float(np.float32(x))


def _exact_step(s, kw, isfluid=None):
    """One step of the state s = [rho - 1, u, v, w, 6 x Pi^neq, phi] (FP64 tensors)."""
    d, u, v, w = s[0], s[1], s[2], s[3]
    P, phi = s[4:10], s[10]
    rho = 1.0 + d
    nz, ny, nx = rho.shape
    per = [kw["bc"][2 * a] == capi.BC_PERIODIC for a in range(3)]
    colour, phase = kw["mode"] == capi.MODE_COLOUR, kw["mode"] == capi.MODE_PHASEFIELD
    sigma, force = _f32(kw["sigma"]), [_f32(k) for k in kw["force"]]
    tau_a, tau_b = _f32(kw["tau_a"]), _f32(kw["tau_b"])
    us, vs, ws = u, v, w
    if colour:
        g = _grad(_pad(phi, per, "edge"))
        m2 = g[0] ** 2 + g[1] ** 2 + g[2] ** 2
        m = m2.sqrt()
        on = m > _f32(kw["grad_threshold"])
        safe = torch.where(on, m, torch.ones_like(m))
        ca, cb = 0.5 * (1.0 + phi), 0.5 * (1.0 - phi)
        nu = 1.0 / (ca * 3.0 / (tau_a - 0.5) + cb * 3.0 / (tau_b - 0.5))
        omega = 2.0 / (6.0 * nu + 1.0)
        A = torch.where(on, 0.5 * 4.5 * sigma * omega * m, torch.zeros_like(m))
        n = [torch.where(on, k / safe, torch.zeros_like(k)) for k in g]
        rec = _f32(kw["beta"]) * ca * cb * rho
    else:
        omega = 1.0 / tau_a
        us, vs, ws = u + force[0], v + force[1], w + force[2]
        if phase:
            g = _grad(_pad(phi, per, "edge"))
            den = (g[0] ** 2 + g[1] ** 2 + g[2] ** 2).sqrt() + 1e-9
            n = [k / den for k in g]
            if isfluid is not None:
                n = [k * isfluid for k in n]
            curv = -(_grad(_pad(n[0], per, "zero"), (0,))[0] + _grad(_pad(n[1], per, "zero"), (1,))[1] +
                     _grad(_pad(n[2], per, "zero"), (2,))[2])
            ind = phi * (1.0 - phi) * (n[0] ** 2 + n[1] ** 2 + n[2] ** 2)
            curv = torch.where(ind > 0.2, curv, torch.zeros_like(curv))
            us, vs, ws = us + sigma * curv * n[0], vs + sigma * curv * n[1], ws + sigma * curv * n[2]
    cubic, third = _eq_terms(us, vs, ws), _third(P, u, v, w)

    def post(c):
        """Post-collision f_c, and for two components the colour difference of the population."""
        c2 = sum(k * k for k in c)
        wq = _W[c2]
        # the weight's own share is added at the end: rho - 1 keeps its digits
        f = wq * (_feq(c, rho, us, vs, ws, cubic) - 1.0 + (1.0 - omega) * _fneq(c, P, third))
        if not colour:
            return f, None
        f = f + 3.0 * wq * _combine(c, force) if any(force) else f
        cn = _combine(c, n) if c2 else 0.0
        f = f + A * (wq * cn * cn - (wq if c2 else -10.0 / 27.0))
        q = (f + wq) * phi
        if c2:
            q = q + 2.0 * rec * wq * cn / math.sqrt(c2)
        return f, q

    def g_post(axis, sign):
        e = (u, v, w)[axis]
        return 0.125 * (phi * (1.0 + 3.0 * sign * e) + sign * _f32(kw["sharp_c"]) * phi * (1.0 - phi) * n[axis])

    zeros = torch.zeros_like(rho)
    M = {k: zeros.clone() for k in ("d", "x", "y", "z", "xx", "xy", "xz", "yy", "yz", "zz", "n")}
    grid = _axes(nx, ny, nz)

    def behind(c):
        """Nodes whose source x - c lies behind a wall face, by face; and behind any."""
        faces, any_ = {}, None
        for a, size in enumerate((nx, ny, nz)):
            if c[a] and not per[a]:
                m = (grid[a] == (0 if c[a] > 0 else size - 1))
                faces[2 * a + (0 if c[a] > 0 else 1)] = m
                any_ = m if any_ is None else any_ | m
        return faces, any_

    solid = None if isfluid is None else isfluid == 0
    for c in _C:
        f, q = post(c)
        shift = (c[2], c[1], c[0])
        ft = torch.roll(f, shift, (0, 1, 2))
        qt = torch.roll(q, shift, (0, 1, 2)) if colour else None
        faces, out = behind(c)
        if solid is not None and any(c):
            src = torch.roll(solid, shift, (0, 1, 2))
            out = src if out is None else out | src
        if out is not None:
            back, qback = post(tuple(-k for k in c))
            ft = torch.where(out, back, ft)
            if colour:
                qt = torch.where(out, qback, qt)
            for face, m in faces.items():
                if kw["bc"][face] != capi.BC_VELOCITY:
                    continue
                wq = _W[sum(k * k for k in c)]
                U = [torch.full_like(rho, _f32(k)) for k in kw["bc_u"][face]]
                val = wq * (_feq(c, rho, *U, _eq_terms(*U)) - 1.0 + (1.0 - omega) * _fneq(c, P, third))
                ft = torch.where(m, val, ft)
                if colour:
                    qt = torch.where(m, (val + wq) * _f32(kw["bc_phi"][face]), qt)
        M["d"] += ft
        for k, a in (("x", 0), ("y", 1), ("z", 2)):
            if c[a]:
                M[k] += c[a] * ft
        for k, a, b in (("xx", 0, 0), ("xy", 0, 1), ("xz", 0, 2), ("yy", 1, 1), ("yz", 1, 2), ("zz", 2, 2)):
            if c[a] * c[b]:
                M[k] += c[a] * c[b] * (ft + _W[sum(j * j for j in c)])
        if colour:
            M["n"] += qt
    r1 = 1.0 + M["d"]
    U = [M[k] / r1 for k in "xyz"]
    out = [M["d"]] + U
    for k, a, b in (("xx", 0, 0), ("xy", 0, 1), ("xz", 0, 2), ("yy", 1, 1), ("yz", 1, 2), ("zz", 2, 2)):
        out.append(M[k] - (r1 / 3.0 if a == b else 0.0) - r1 * U[a] * U[b])
    if colour:
        out.append(M["n"] / r1)
    elif phase:
        new = 0.25 * phi
        for axis in range(3):
            for sign in (1, -1):
                c = tuple(sign if a == axis else 0 for a in range(3))
                shift = (c[2], c[1], c[0])
                gt = torch.roll(g_post(axis, sign), shift, (0, 1, 2))
                _, behind_any = behind(c)
                if solid is not None:
                    src = torch.roll(solid, shift, (0, 1, 2))
                    behind_any = src if behind_any is None else behind_any | src
                if behind_any is not None:
                    gt = torch.where(behind_any, g_post(axis, -sign), gt)
                new = new + gt
        out.append(new)
    else:
        out.append(phi)
    if solid is not None:
        out = [torch.where(solid, a, b) for a, b in zip(s, out)]
    return out


def _mix64(z):
    with np.errstate(over="ignore"):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


def _exact_train(case, seed):
    """The same samples, network and Adam steps in FP64."""
    f, t, w = (a.double() for a in _train_set(case, seed))
    x = f / torch.tensor([float(np.float32(k)) for k in [1e-4] * 6 + [1.0, 0.3, 0.05, 2e-4]], dtype=torch.float64, device=DEV)
    p = torch.tensor(init_params(0), dtype=torch.float64, device=DEV)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    steps, batch, n = case["steps"], case["batch"], case["samples"]
    hist = []
    for k in range(steps):
        with np.errstate(over="ignore"):
            key = np.uint64(int(seed) % (1 << 31)) * np.uint64(0x100000001B3) ^ (np.uint64(k) << np.uint64(40))
            idx = torch.from_numpy((_mix64(key ^ np.arange(batch, dtype=np.uint64)) % np.uint64(n)).astype(np.int64)).to(DEV)
        q = p.clone().requires_grad_(True)
        W1 = q[:1024].view(64, 16)[:, :10]
        h = torch.relu(x[idx] @ W1.T + q[1024:1088])
        h = torch.relu(h @ q[1088:5184].view(64, 64).T + q[5184:5248])
        y = _f32(0.02) * torch.sigmoid(h @ q[5248:5312] + q[5312])
        loss = (w[idx] * (y - t[idx]) ** 2).mean()
        loss.backward()
        hist.append(float(loss))
        lr = 2e-3 * (0.1 + 0.9 * 0.5 * (1.0 + math.cos(math.pi * k / steps)))
        m = 0.9 * m + 0.1 * q.grad
        v = 0.999 * v + 0.001 * q.grad ** 2
        p = p - lr * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return {"loss": torch.tensor(hist, dtype=torch.float64), "params": p}


def exact(case, seed):
    path = case["path"]
    if path == "train":
        return _exact_train(case, seed)
    if path == "jet":
        return None   # the closure's network is BF16 by definition: no 64-bit value
    if path == "ensemble":
        phi = []
        for kw, dims, radius in _members(case, seed):
            s = [a.double() for a in _member_state(dims, radius)]
            for _ in range(case["steps"]):
                s = _exact_step(s, kw)
            phi.append(s[10].reshape(-1))
        return {"phi": torch.cat(phi)}
    kw = _params(case)
    s = [a.double() for a in _state(case, seed)]
    if path == "run":   # the upload takes rho in FP32
        s[0] = (s[0].float() + 1.0).double() - 1.0
    fluid = _obstacle(case).double() if case["obstacle"] else None
    totals = []
    for _ in range(case["steps"]):
        s = _exact_step(s, kw, fluid)
        rho = 1.0 + s[0]
        a = float((0.5 * rho * (1.0 + s[10])).sum()) if case["mode"] == "colour" else float(s[10].sum())
        totals.append([float(rho.sum()), a, float((0.5 * rho * (s[1] ** 2 + s[2] ** 2 + s[3] ** 2)).sum())])
    n = s[0].numel()
    if path == "call":
        out = torch.zeros((NF, (n + 31) // 32 * 32), dtype=torch.float64, device=DEV)
        for k in range(NF):
            out[k, :n] = s[k].reshape(-1)
        if case["mode"] == "single":
            out[10] = 1.0
        return out
    flow = torch.stack([1.0 + s[0], s[1], s[2], s[3], s[10]]).view(len(STAMP), n)
    return {"stamp": flow, "totals": torch.tensor(totals, dtype=torch.float64)}
