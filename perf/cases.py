"""The work a user of this framework has it do, as timed cases.

Engine cases go through the C ABI as the Fortran driver's loop does (``projectracer_gb300.engine``):
a job starts from restart arrays on the host, solves for psi, advances one time step, writes its
stats row and takes the restart records back.  The library keeps one context per process, so
every pass uploads its state; host arrays are pinned.  Network cases call the U-Net of the learned
psi guess (include/ptgpu_unet.h), whose handles are per network and whose arrays are host arrays too.

A case holds plain values: ``kind`` (step, solve, unet_forward, unet_gradients), the sizes, and for
the engine the physics family, the precision and the solver options that the configurations of this
repository use.
"""

from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from projectracer_gb300 import engine as eng
from projectracer_gb300.config import (PT_CYCLE_REFERENCE, PT_CYCLE_V, PT_GUESS_EXTRAPOLATE, PT_GUESS_PREVIOUS,
                                       PT_MG_CORRECTION, PT_PREC_FP64, PT_PREC_MIXED, workload)
from projectracer_gb300.inputs import grid_coords
from projectracer_gb300.learned import UNet


def listed():
    return [
        # the small production run: isoviscous 128x128 at 1e-8, mixed precision with GCR; every
        # kernel lasts microseconds, so launches and latency count
        dict(name="step_mixed_128x128", kind="step", physics="C1", precision="mixed", nx=128, nz=128, aspect=1.0,
             tpc=20, krylov=8, direct=0),
        # the ordinary thermochemical run (eta(T), 1e-8, four levels)
        dict(name="step_mixed_256x128", kind="step", physics="C2", precision="mixed", nx=256, nz=128, aspect=2.0,
             tpc=30, krylov=8, direct=0),
        # the headline workload: 1024x512, 16.8M tracers, viscosity contrast 1e5 with depth, 1e-6
        dict(name="step_mixed_1024x512", kind="step", physics="C3", precision="mixed", nx=1024, nz=512, aspect=2.0,
             tpc=32, krylov=0, direct=0),
        # an odd grid: spacings that are neither powers of two nor equal, rows that fill no tile
        dict(name="step_mixed_208x144", kind="step", physics="chem", precision="mixed", nx=208, nz=144, aspect=1.5,
             tpc=11, krylov=0, direct=0),
        # the velocity solve of the largest grid (2048x1024); few tracers, on which it does not depend
        dict(name="solve_mixed_2048x1024", kind="solve", physics="C5", precision="mixed", nx=2048, nz=1024, aspect=2.0,
             tpc=4, krylov=0, direct=0),
        # the reference's own algorithm in FP64: parity runs of the small and the ordinary grid
        dict(name="step_fp64_128x128", kind="step", physics="C1", precision="fp64", nx=128, nz=128, aspect=1.0,
             tpc=20, krylov=0, direct=0),
        dict(name="step_fp64_256x128", kind="step", physics="C2", precision="fp64", nx=256, nz=128, aspect=2.0,
             tpc=30, krylov=0, direct=0),
        # the reference's shipped solver (iterate=0, banded direct solve) on its shipped grid
        dict(name="step_direct_100x100", kind="step", physics="C1", precision="fp64", nx=100, nz=100, aspect=1.0,
             tpc=60, krylov=0, direct=1),
        # the learned guess of a small run: the smallest call there is
        dict(name="unet_forward_64x32", kind="unet_forward", nx=64, nz=32, batch=1),
        # the learned guess of the 512x256 study, one state per solve
        dict(name="unet_forward_512x256", kind="unet_forward", nx=512, nz=256, batch=1),
        # its training batch (forward, loss and all parameter gradients)
        dict(name="unet_gradients_512x256", kind="unet_gradients", nx=512, nz=256, batch=8),
        # a ragged training batch: rows and pixel counts that fill no tile
        dict(name="unet_gradients_136x72", kind="unet_gradients", nx=136, nz=72, batch=3),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "solve", "fp64", "direct", "unet_forward", "unet_gradients"])
    if kind.startswith("unet"):
        nx = 8 * max(2, round(_log_uniform(rng, 16, 512) / 8))
        nz = 8 * max(2, min(32, round(nx * rng.choice([0.5, 0.6, 1.0]) / 8)))
        most = max(1, min(12, 8 * 512 * 256 // (nx * nz)))
        return dict(kind=kind, nx=nx, nz=nz, batch=rng.randint(1, most))
    if kind == "direct":
        nz = 2 * rng.randint(24, 50)
        return dict(kind="step", physics="C1", precision="fp64", nx=nz, nz=nz, aspect=1.0, tpc=rng.randint(8, 40),
                    krylov=0, direct=1)
    fp64 = kind == "fp64"
    levels = rng.randint(3, 4)  # halvings below the fine grid
    unit = 2 ** levels
    nz = unit * max(4, round(_log_uniform(rng, 32, 96 if fp64 else 512) / unit))
    nz = unit * min(nz // unit, 31)
    ratio = rng.choice([1.0, 1.25, 1.5, 2.0])
    nx = unit * max(nz // unit, round(nz * ratio / unit))
    # square cells as a rule, flattened ones now and then
    aspect = nx / nz if rng.random() < 0.7 else 1.1 * nx / nz
    physics = "chem" if nz > 256 else rng.choice(["C1", "chem"])
    krylov = 0 if fp64 else 8 if physics == "C1" else rng.choice([0, 8])
    return dict(kind="solve" if kind == "solve" else "step", physics=physics, precision="fp64" if fp64 else "mixed",
                nx=nx, nz=nz, aspect=aspect, tpc=rng.randint(8, 32), krylov=krylov, direct=0)


# ---------------------------------------------------------------------------------- engine cases
def _config(case):
    mixed = case["precision"] == "mixed"
    physics = case["physics"]
    c, w = workload("C2" if physics == "chem" else physics, precision=PT_PREC_MIXED if mixed else PT_PREC_FP64)
    c.tolerance = w.get("bench_tolerance", c.tolerance)
    if physics == "chem":  # eta(T) and a dense layer at a Rayleigh number that every grid here resolves
        c.RaT, c.RaC, c.visT, c.courant, c.CFL, c.grids = 1e5, 5e4, 1e3, 0.1, 1, 6
        c.mg_scheme = PT_MG_CORRECTION
    if physics == "chem" or case["nz"] > 160:  # as the configurations set it: 1e-8 on the small grids only
        c.tolerance = 1e-6
    c.nx, c.nz, c.aspect, c.tpc = case["nx"], case["nz"], case["aspect"], case["tpc"]
    c.ntr = c.nx * c.nz * c.tpc
    c.krylov, c.direct = case["krylov"], case["direct"]
    c.mg_cycle = PT_CYCLE_V if mixed else PT_CYCLE_REFERENCE
    c.guess_mode = PT_GUESS_EXTRAPOLATE if mixed else PT_GUESS_PREVIOUS
    c.max_cycles = 200
    return c


# the program's engine: one context per process, made again when the configuration changes
_engine: dict = {"key": None, "engine": None}


def _get_engine(cfg):
    key = bytes(cfg)
    if _engine["key"] != key:
        if _engine["engine"] is not None:
            _engine["engine"].close()
        _engine["key"], _engine["engine"] = None, None
        _engine["engine"] = eng.Engine(cfg)
        _engine["key"] = key
    return _engine["engine"]


def _close_engine():
    if _engine["engine"] is not None:
        _engine["engine"].close()
    _engine["key"], _engine["engine"] = None, None


def _pinned(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out.numpy()


def _restart_arrays(cfg, seed):
    """Restart arrays as a run's start-up makes them: a conductive profile with a few convective
    modes and noise, a dense bottom layer, and tracers placed at random within the sub-cells of each
    cell, carrying T and C of their place."""
    dev = "cuda"
    gen = torch.Generator(device=dev)
    gen.manual_seed(1000003 * (seed % 2000003) + 17)
    host = np.random.default_rng(seed % 2**63)
    nx, nz, a = cfg.nx, cfg.nz, cfg.aspect
    modes = [(1, 1, 0.008 + 0.004 * host.random())] + [(int(host.integers(1, 5)), int(host.integers(1, 3)),
                                                        0.003 * host.random()) for _ in range(3)]

    def temperature(x, z):
        t = 1.0 - z
        for kx, kz, amp in modes:
            t = t + amp * torch.cos(kx * math.pi / a * x) * torch.sin(kz * math.pi * z)
        if cfg.ivis:
            t = t + 1e-3 * (2.0 * torch.rand(t.shape, generator=gen, device=dev, dtype=torch.float64) - 1.0)
        return t

    xg, zg = grid_coords(cfg)
    X, Z = np.meshgrid(xg[3:nx + 10], zg[3:nz + 10])
    T = temperature(torch.from_numpy(X).to(dev), torch.from_numpy(Z).to(dev)).cpu().numpy()
    T[(Z < 0) | (Z > 1)] = 0.0
    _, Z5 = np.meshgrid(xg[1:nx + 12], zg[1:nz + 12])
    C = np.where(Z5 < 0.2, 1.0, 0.0) if cfg.comp else np.zeros_like(Z5)
    n, per = int(cfg.ntr), cfg.tpc
    sa = int(math.sqrt(per))
    while per % sa:
        sa -= 1
    sb = per // sa
    ids = torch.arange(n, device=dev)
    sub, cell = ids % per, ids // per
    r = (torch.div(cell, nz, rounding_mode="floor") + ((sub % sa) + torch.rand(n, generator=gen, device=dev, dtype=torch.float64)) / sa) * (a / nx)
    s = ((cell % nz) + (torch.div(sub, sa, rounding_mode="floor") + torch.rand(n, generator=gen, device=dev, dtype=torch.float64)) / sb) * (1.0 / nz)
    Ttr = temperature(r, s)
    Ctr = (s < 0.2).to(torch.float64) if cfg.comp else torch.zeros_like(s)
    st = dict(xg=xg, zg=zg, T=T, Cnew=C, SF=np.zeros((nz + 7, nx + 7)), rtr=_pinned(r), str=_pinned(s),
              Ctr=_pinned(Ctr), Ttr=_pinned(Ttr))
    return st


# arrays the program receives the restart records in, kept between calls
_records: dict = {}


def _record_arrays(cfg):
    key = (cfg.nx, cfg.nz, int(cfg.ntr))
    if key not in _records:
        _records.clear()
        nx, nz, n = key
        shapes = dict(T=(nz + 7, nx + 7), C=(nz + 11, nx + 11), SF=(nz + 7, nx + 7), r=(n,), s=(n,), Ttr=(n,))
        _records[key] = {k: torch.empty(v, dtype=torch.float64, pin_memory=True).numpy() for k, v in shapes.items()}
    return _records[key]


def _prepare_engine(case, seed):
    cfg = _config(case)
    st = _restart_arrays(cfg, seed)
    torch.cuda.synchronize()
    _get_engine(cfg)
    _record_arrays(cfg)
    return dict(kind=case["kind"], cfg=cfg, restart=st)


def _run_engine(state):
    cfg = state["cfg"]
    e, out = _get_engine(cfg), _record_arrays(cfg)
    e.upload(state["restart"])
    info = e.solve_psi()
    if state["kind"] == "solve":
        e._check(e.L.pt_get_field(eng.F_SF, out["SF"].ctypes.data))
        e._check(e.L.pt_get_field(eng.F_U, out["T"].ctypes.data))
        return dict(SF=out["SF"], u=out["T"], cycles=info["cycles"])
    row = e.stats()
    dt, _ = e.step()
    ptr = {k: ctypes.c_void_p(v.ctypes.data) for k, v in out.items()}
    e._check(e.L.pt_download_state(ptr["T"], ptr["C"], ptr["SF"], ptr["r"], ptr["s"], None, ptr["Ttr"], None))
    return dict(out, dt=dt, Nu=row["Nu"], vrms=row["vrms"], tracer_min=row["tracer_min"], tracer_max=row["tracer_max"])


def _work_engine(case):
    nodes, ntr = (case["nx"] + 1) * (case["nz"] + 1), case["nx"] * case["nz"] * case["tpc"]
    comp = case["physics"] != "C1"
    solves = 1 if case["kind"] == "solve" else 4
    # tracers in (r, s, T, C) and out (r, s, T), restart fields in and out
    b = 8.0 * ntr * (3 + comp + (0 if case["kind"] == "solve" else 3)) + 8.0 * nodes * (5 + comp)
    # a solve at its best: about ten sweeps of a 120-operation stencil on a hierarchy of 4/3 nodes; per
    # RK stage three 16-term interpolations and one 9-node projection of each tracer
    f = solves * nodes * (4.0 / 3.0) * 10 * 120 + (0 if case["kind"] == "solve" else 4 * ntr * 250.0)
    return dict(bytes=b, flops=f)


# ---------------------------------------------------------------------------------- network cases
# (source, skip source, view, cin, cout, level) of the 14 convolutions; view 1 pools 2x2, 2 upsamples
# and appends the skip tensor
_LAYERS = [(-1, -1, 0, 4, 32, 0), (0, -1, 0, 32, 32, 0), (1, -1, 1, 32, 64, 1), (2, -1, 0, 64, 64, 1),
           (3, -1, 1, 64, 128, 2), (4, -1, 0, 128, 128, 2), (5, -1, 1, 128, 256, 3), (6, -1, 0, 256, 256, 3),
           (7, 5, 2, 384, 128, 2), (8, -1, 0, 128, 128, 2), (9, 3, 2, 192, 64, 1), (10, -1, 0, 64, 64, 1),
           (11, 1, 2, 96, 32, 0), (12, -1, 0, 32, 32, 0)]


class _Net(UNet):
    """A network handle that goes with its state."""

    def __del__(self):
        self.close()


def _prepare_unet(case, seed):
    nz, nx, b = case["nz"], case["nx"], case["batch"]
    net = _Net(nz, nx, b, seed % 2**31 + 1)
    rng = np.random.default_rng(seed % 2**63)
    z, x = np.meshgrid(np.linspace(0, 1, nz, endpoint=False), np.linspace(0, 2, nx, endpoint=False), indexing="ij")
    xs = np.empty((b, 4, nz, nx), dtype=np.float32)
    ts = np.empty((b, nz, nx), dtype=np.float32)
    for q in range(b):
        # planes T, C, log10(eta)/5, RHS/max|RHS| of a state with a few convection cells, and its psi
        kx, kz, ph = int(rng.integers(1, 4)), int(rng.integers(1, 3)), rng.uniform(0, 6.0)
        cell = np.cos(kx * np.pi * x / 2 + ph) * np.sin(kz * np.pi * z)
        xs[q, 0] = 1 - z + 0.1 * cell + 1e-3 * rng.standard_normal((nz, nx))
        xs[q, 1] = z + 0.05 * cell < 0.2
        xs[q, 2] = -0.6 * xs[q, 0]
        xs[q, 3] = np.sin(kx * np.pi * x / 2 + ph) * np.sin(kz * np.pi * z) + 0.05 * rng.standard_normal((nz, nx))
        ts[q] = np.sin(kx * np.pi * x / 2 + ph) * np.sin(kz * np.pi * z) * (1 + 0.2 * cell)
    state = dict(kind=case["kind"], net=net, batch=b, x=_pinned(torch.from_numpy(xs)))
    if case["kind"] == "unet_forward":
        state["y"] = _pinned(torch.zeros(b, nz, nx))
    else:
        state["t"] = _pinned(torch.from_numpy(ts))
        state["grads"] = _pinned(torch.zeros(net.num_params()))
    return state


def _run_unet(state):
    net = state["net"]
    if state["kind"] == "unet_forward":
        net._ok(net.L.pt_unet_forward(net.h, state["x"].ctypes.data, state["batch"], state["y"].ctypes.data))
        return state["y"]
    loss = ctypes.c_float()
    net._ok(net.L.pt_unet_gradients(net.h, state["x"].ctypes.data, state["t"].ctypes.data, state["batch"],
                                    state["grads"].ctypes.data, ctypes.byref(loss)))
    return dict(grads=state["grads"], loss=np.float32(loss.value))


def _work_unet(case):
    pixels = case["batch"] * case["nx"] * case["nz"]
    conv = sum(2.0 * 9 * cin * cout * (pixels >> (2 * lev)) for _, _, _, cin, cout, lev in _LAYERS)
    params = sum(9 * cin * cout + cout for _, _, _, cin, cout, _ in _LAYERS) + 33
    if case["kind"] == "unet_forward":
        return dict(bytes=4.0 * pixels * 5 + 2.0 * params, flops=conv)
    # forward, gradients of every weight, and of every input but the network's own
    return dict(bytes=4.0 * pixels * 5 + 2.0 * params + 4.0 * params, flops=3 * conv - 2.0 * 9 * 4 * 32 * pixels)


def _exact_unet(case, seed):
    """The network in 64 bits with torch's own convolutions, without any rounding to 16 bits."""
    state = _prepare_unet(case, seed)
    flat = torch.from_numpy(state["net"].params().astype(np.float64)).cuda().requires_grad_(True)
    x = torch.from_numpy(state["x"]).cuda().double()
    F = torch.nn.functional
    acts, off = [], 0
    for src, skip, view, cin, cout, _ in _LAYERS:
        w = flat[off:off + cout * 9 * cin].view(cout, 3, 3, cin).permute(0, 3, 1, 2)
        off += cout * 9 * cin
        bias = flat[off:off + cout]
        off += cout
        h = x if src < 0 else acts[src]
        if view == 1:
            h = F.avg_pool2d(h, 2)
        elif view == 2:
            h = torch.cat([F.interpolate(h, scale_factor=2, mode="nearest"), acts[skip]], 1)
        # the convolution as nine shifted matrix products, which keeps its workspace small
        hp = F.pad(h, (1, 1, 1, 1))
        H, W = h.shape[2:]
        z = bias.view(1, -1, 1, 1)
        for t in range(9):
            z = z + torch.einsum("oc,bchw->bohw", w[:, :, t // 3, t % 3],
                                 hp[:, :, t // 3:t // 3 + H, t % 3:t % 3 + W])
        acts.append(torch.relu(z))
    y = torch.einsum("c,bchw->bhw", flat[off:off + 32], acts[-1]) + flat[off + 32]
    if case["kind"] == "unet_forward":
        out = y.detach().cpu().numpy()
    else:
        loss = ((y - torch.from_numpy(state["t"]).cuda().double()) ** 2).mean()
        loss.backward()
        out = dict(grads=flat.grad.cpu().numpy(), loss=float(loss))
    state["net"].close()
    return out


# ---------------------------------------------------------------------------------- the interface
def prepare(case, seed):
    if case["kind"].startswith("unet"):
        _close_engine()
        return _prepare_unet(case, seed)
    return _prepare_engine(case, seed)


def run(state):
    return _run_unet(state) if state["kind"].startswith("unet") else _run_engine(state)


def work(case):
    return _work_unet(case) if case["kind"].startswith("unet") else _work_engine(case)


def exact(case, seed):
    if not case["kind"].startswith("unet"):
        return None  # a whole solve and step: no short restatement
    if case["kind"] == "unet_gradients" and case["batch"] * case["nx"] * case["nz"] > 200000:
        return None  # over the time and memory of a quick 64-bit pass
    return _exact_unet(case, seed)
