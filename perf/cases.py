"""The work a user has this framework do, as measured cases.

A program that uses the framework steps channels (one, or a batch of uneven
ones) between two looks at their fields, and trains and evaluates the
warm-start network.  Each case is one such stretch through the public entry
points:

  channel  ek_step(steps) of one channel, then its fields copied to the
           caller's device buffers (u_x, u_y, c+, c-, psi; FP64 storage also
           the steady-state residual).  The state moves on from pass to pass,
           as it does in a run to steady state.
  batch    the same for many channels in lockstep (ek_batch_step).
  train    Adam iterations of the network; the updated weights and the losses.
  forward  the network on host rows, the profiles back on the host.

Fields of FP32 and FP16 storage come back in the type that they are good for.
exact() restates the physics in plain torch, FP64, without this package.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("ek-pnp_b200"))

STORE = {"f64": 0, "f32": 1, "f16": 2}
KEEP = {"f32": torch.float32, "f16": torch.float16}
OUT = ("ux", "uy", "cp", "cn", "psi")
ORDER = ("rho", "ux", "uy", "cp", "cn", "psi", "ex", "ey")
DIMS = ((16, 256), (256, 256), (256, 256), (256, 512))  # the network's layers (inputs padded 4 -> 16)


def _channel(name, nx, ny, steps, storage, **more):
    c = dict(name=name, kind="channel", nx=nx, ny=ny, steps=steps, storage=storage, kappa_h=8.0, zeta=-2.0, ex=1e-4,
             diff=0.05, eps=0.01, wave=0.0)
    c.update(more)
    return c


def listed():
    return [
        # the reference's own default shape (NX = 10, NY = 101): the smallest call
        _channel("f64-10x101", 10, 101, 100, "f64", kappa_h=6.0, zeta=-1.0, ex=5e-4),
        # the parity channel, FP64: what a user validates against the reference with
        _channel("f64-256x128", 256, 128, 100, "f64"),
        # a length that is not a power of two, and an odd number of rows
        _channel("f64-1000x257", 1000, 257, 20, "f64", kappa_h=16.0),
        # the large channel in FP64
        _channel("f64-4096x1024", 4096, 1024, 10, "f64", kappa_h=32.0, zeta=-4.0, ex=5e-5, eps=1.0),
        # an ordinary channel in FP32
        _channel("f32-512x203", 512, 203, 100, "f32", kappa_h=10.0),
        # the large channel in FP32 shifted storage: the headline workload
        _channel("f32-4096x1024", 4096, 1024, 20, "f32", kappa_h=32.0, zeta=-4.0, ex=5e-5, eps=1.0),
        # the same channel with FP16 storage
        _channel("f16-4096x1024", 4096, 1024, 20, "f16", kappa_h=32.0, zeta=-4.0, ex=5e-5, eps=1.0),
        # the heterogeneous wall, zeta(x) = -2 + 1.5 sin(2 pi x / 1024): the largest call
        _channel("f32-8192x2048-wave", 8192, 2048, 10, "f32", kappa_h=64.0, wave=1.5),
        # uneven channels of the batched workload, one cycle between two looks
        dict(name="batch-64-uneven", kind="batch", channels=64, nx=0, nx_max=1024, ny_min=32, ny_max=512, steps=200,
             storage="f32"),
        # the 16-column channels that the warm start's training set and its relaxation run on
        dict(name="batch-128-narrow", kind="batch", channels=128, nx=16, nx_max=16, ny_min=32, ny_max=512, steps=200,
             storage="f32"),
        # the warm-start network: training iterations, and profiles for the held-out channels
        dict(name="train-256", kind="train", batch=256, rows=8192, iters=32, lr=2e-3),
        dict(name="forward-1000", kind="forward", batch=256, rows=1000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["channel"] * 7 + ["batch"] * 2 + ["train", "forward"])
    if kind == "channel":
        storage = rng.choice(["f64", "f32", "f32", "f16"])
        ny = _log_int(rng, 12, 1200)
        if rng.random() < 0.3:
            nx = _log_int(rng, 9, 1500)
        else:
            nx = 1 << rng.randint(4, 12)
        steps = max(4, min(100, int(6e7 / (nx * ny))))
        kappa_h = math.exp(rng.uniform(0.0, math.log(min(50.0, 0.5 * (ny - 1)))))
        return dict(kind="channel", nx=nx, ny=ny, steps=steps, storage=storage, kappa_h=round(kappa_h, 3),
                    zeta=round(rng.uniform(-3.0, -0.5), 3), ex=round(math.exp(rng.uniform(math.log(2e-5), math.log(1e-3))), 8),
                    diff=round(rng.uniform(0.02, 0.1), 4), eps=0.01, wave=0.4 if storage != "f64" and rng.random() < 0.3 else 0.0)
    if kind == "batch":
        nx = rng.choice([0, 0, 16])
        ny_min = rng.randint(24, 64)
        return dict(kind="batch", channels=_log_int(rng, 4, 64), nx=nx, nx_max=16 if nx else rng.choice([128, 512, 1024]),
                    ny_min=ny_min, ny_max=rng.randint(ny_min + 10, 512), steps=200, storage=rng.choice(["f32", "f32", "f16"]))
    if kind == "train":
        b = rng.choice([128, 256, 512])
        return dict(kind="train", batch=b, rows=_log_int(rng, 2 * b, 8192), iters=rng.randint(16, 40), lr=2e-3)
    return dict(kind="forward", batch=rng.choice([128, 256, 512]), rows=_log_int(rng, 1, 8192))


# ---- inputs ------------------------------------------------------------------

def _params(c):
    """ek_params of a channel in lattice units (dx = dy = dt = cfl = 1)."""
    kappa = c["kappa_h"] / (c["ny"] - 1)
    z, d = c["zeta"], c["diff"]
    return dict(nx=c["nx"], ny=c["ny"], storage=STORE[c["storage"]], flags=1, dx=1.0, dy=1.0, dt=1.0, cfl=1.0,
                cs2=1.0 / 3.0, lx=float(c["nx"]), rho0=1.0, c0=1.0, nu=1.0 / 6.0, magic_f=0.25, diff_p=d, magic_p=0.25,
                mob_p=d, diff_n=d, magic_n=0.25, mob_n=-d, eps=c["eps"], f_charge=0.5 * c["eps"] * kappa * kappa,
                zeta_lo=z, zeta_hi=z, cp_lo=math.exp(-z), cp_hi=math.exp(-z), cn_lo=math.exp(z), cn_hi=math.exp(z),
                ext_x=c["ex"], exf=0.0, uw=0.0)


def _walls(c):
    x = np.arange(c["nx"])
    return c["zeta"] + c["wave"] * np.sin(2.0 * math.pi * x / min(c["nx"], 1024))


def _fields(c, seed, dev):
    """Start fields: the linear double layer, Boltzmann ions with 0.1 % noise, the electro-osmotic profile."""
    nx, ny = c["nx"], c["ny"]
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    kw = dict(device=dev, dtype=torch.float64)
    half = 0.5 * (ny - 1)
    a = c["kappa_h"] / (ny - 1) * (torch.arange(ny, **kw) - half).abs()
    b = 0.5 * c["kappa_h"]
    prof = torch.exp(a - b) * (1.0 + torch.exp(-2.0 * a)) / (1.0 + math.exp(-2.0 * b))
    zeta = torch.as_tensor(_walls(c), **kw)
    psi = prof[:, None] * zeta[None, :]
    cp = torch.exp(-psi) * (1.0 + 1e-3 * torch.randn(ny, nx, generator=g, **kw))
    cn = torch.exp(psi) * (1.0 + 1e-3 * torch.randn(ny, nx, generator=g, **kw))
    ux = 6.0 * c["eps"] * c["ex"] * (psi - zeta[None, :])
    return dict(rho=torch.ones(ny, nx, **kw), ux=ux, uy=torch.zeros(ny, nx, **kw), cp=cp, cn=cn, psi=psi)


def _batch_channels(c, seed):
    """Uneven channels of one batch.  The shapes belong to the case; the physics is the seed's."""
    shape = np.random.default_rng(2)
    r = np.random.default_rng(seed)
    widths = [w for w in (64, 128, 256, 512, 1024) if w <= c["nx_max"]]
    out = []
    for _ in range(c["channels"]):
        nx = c["nx"] or int(shape.choice(widths))
        ny = int(shape.integers(c["ny_min"], c["ny_max"] + 1))
        out.append(dict(nx=nx, ny=ny, storage=c["storage"], kappa_h=float(np.exp(r.uniform(0.0, math.log(50.0)))),
                        zeta=float(r.uniform(-4.0, -0.5)), ex=float(np.exp(r.uniform(math.log(1e-5), math.log(1e-3)))),
                        diff=float(r.uniform(0.02, 0.1)), eps=0.01, wave=0.0))
    return out


def _net_inputs(c, seed):
    """Descriptors in [-1, 1], smooth standardised profiles as targets, Glorot weights (flat: W then b per layer)."""
    r = np.random.default_rng(seed)
    x = r.uniform(-1.0, 1.0, (c["rows"], 4)).astype(np.float32)
    mix = r.standard_normal((4, 512))
    t = np.sin(x @ mix + r.uniform(0.0, 6.0, 512)).astype(np.float32)
    flat = []
    for l, (i, o) in enumerate(DIMS):
        a = math.sqrt(6.0 / ((4 if l == 0 else i) + o))
        w = r.uniform(-a, a, (o, i)).astype(np.float32)
        if l == 0:
            w[:, 4:] = 0.0
        flat += [w.reshape(-1), np.zeros(o, dtype=np.float32)]
    return x, t, np.concatenate(flat)


# ---- the measured calls --------------------------------------------------------

def _load(ch, c, seed):
    """The start fields of one channel, straight from device memory."""
    from ekpnp import lib
    f = _fields(c, seed, "cuda")
    torch.cuda.synchronize()
    rc = lib().ek_set_fields_device(ch._h, *[f[k].data_ptr() if k in f else None for k in ORDER])
    if rc:
        raise RuntimeError("ek_set_fields_device: %d" % rc)


def _buffers(c):
    return {k: torch.empty(c["ny"], c["nx"], device="cuda", dtype=torch.float64) for k in OUT}


def _read(ch, buf):
    from ekpnp import lib
    rc = lib().ek_get_fields_device(ch._h, *[ctypes.c_void_p(buf[k].data_ptr()) if k in buf else None for k in ORDER])
    if rc:
        raise RuntimeError("ek_get_fields_device: %d" % rc)


def prepare(case, seed):
    from ekpnp import Batch, Channel
    kind = case["kind"]
    if kind == "channel":
        ch = Channel(_params(case))
        if case["wave"]:
            z = _walls(case)
            ch.set_wall_profile(z, z, np.exp(-z), np.exp(-z), np.exp(z), np.exp(z))
        _load(ch, case, seed)
        ch.init_equilibrium()
        ch.sync()
        if case["storage"] == "f64":
            ch.residual(1)  # the snapshot that the first residual is taken from
        return dict(case=case, ch=ch, buf=_buffers(case))
    if kind == "batch":
        specs = _batch_channels(case, seed)
        b = Batch([_params(s) for s in specs])
        for i, s in enumerate(specs):
            _load(b[i], s, seed + 1000 * i)
        b.set_cycle(200)
        b.init_equilibrium()
        b.sync()
        return dict(case=case, b=b, buf=[_buffers(s) for s in specs])
    from ekpnp.mlp import Mlp
    x, t, flat = _net_inputs(case, seed)
    net = Mlp(batch=case["batch"], seed=seed)
    net.params = flat
    if kind == "train":
        net.set_data(x, t)
    return dict(case=case, net=net, x=x)


def run(state):
    c = state["case"]
    if c["kind"] == "channel":
        ch, buf = state["ch"], state["buf"]
        ch.step(c["steps"])
        _read(ch, buf)
        if c["storage"] == "f64":
            r = ch.residual(c["steps"])  # waits for the stream
            return dict(fields=buf, residual=r[:4])
        ch.sync()
        return dict(fields={k: v.to(KEEP[c["storage"]]) for k, v in buf.items()})
    if c["kind"] == "batch":
        b = state["b"]
        b.step(c["steps"])
        for ch, buf in zip(b.channels, state["buf"]):
            _read(ch, buf)
        b.sync()
        return {k: torch.cat([buf[k].reshape(-1) for buf in state["buf"]]).to(KEEP[c["storage"]]) for k in OUT}
    if c["kind"] == "train":
        loss = state["net"].train(c["iters"], c["lr"])
        return dict(params=state["net"].params, loss=loss.astype(np.float32))
    return state["net"].forward(state["x"])


def work(case):
    kind = case["kind"]
    if kind in ("channel", "batch"):
        s = {"f64": 8, "f32": 4, "f16": 2}[case["storage"]]
        chans = [case] if kind == "channel" else _batch_channels(case, 0)
        nodes = sum(c["nx"] * c["ny"] for c in chans)
        fft = sum(c["nx"] * c["ny"] * (5.0 * math.log2(c["nx"]) + 12.0) for c in chans)
        # per step: 27 populations read and written, the right-hand side and psi once each;
        # once: the five fields written out
        fld = 8 if case["storage"] == "f64" else 4
        return {"bytes": case["steps"] * nodes * (54.0 * s + 2.0 * fld) + nodes * 5 * 8.0,
                "flops": case["steps"] * (nodes * 420.0 + fft)}
    mac = float(sum(i * o for i, o in DIMS))
    n = sum(i * o + o for i, o in DIMS)
    if kind == "train":
        rows = case["batch"]
        # per iteration: the batch, the FP32 weights and both Adam moments read and written
        return {"bytes": case["iters"] * (rows * 516.0 * 4 + 6.0 * n * 4), "flops": case["iters"] * 6.0 * rows * mac}
    return {"bytes": case["rows"] * 516.0 * 4 + n * 4.0, "flops": 2.0 * case["rows"] * mac}


# ---- the same in plain FP64 ------------------------------------------------------

CX = (0, 1, 0, -1, 0, 1, -1, -1, 1)
CY = (0, 0, 1, 0, -1, 1, 1, -1, -1)
OPP = (0, 3, 4, 1, 2, 7, 8, 5, 6)
W = (4 / 9,) + (1 / 9,) * 4 + (1 / 36,) * 4


def _equilibrium(dens, ux, uy):
    usq = 1.5 * (ux * ux + uy * uy)
    out = []
    for d in range(9):
        cu = 3.0 * (CX[d] * ux + CY[d] * uy)
        out.append(W[d] * dens * (1.0 - usq + cu * (1.0 + 0.5 * cu)))
    return torch.stack(out)


def _trt(p, e, wp, wm):
    o = list(OPP)
    q = p[o]
    return p - wp * 0.5 * ((p + q) - (e + e[o])) - wm * 0.5 * ((p - q) - (e - e[o]))


def _guo(ux, uy, fx, fy, nu, magic):
    """Guo source with the TRT split of its even and odd parts."""
    out = []
    uf = 3.0 * (ux * fx + uy * fy)
    for d in range(9):
        cf = CX[d] * fx + CY[d] * fy
        cu = CX[d] * ux + CY[d] * uy
        out.append(W[d] * (3.0 * cf - uf + 9.0 * cu * cf))
    s = torch.stack(out)
    sb = s[list(OPP)]
    wp = 1.0 / (3.0 * nu + 0.5)
    wm = 1.0 / (magic / (3.0 * nu) + 0.5)
    return (1.0 - 0.5 * wp) * 0.5 * (s + sb) + (1.0 - 0.5 * wm) * 0.5 * (s - sb)


def _pull(p):
    return torch.stack([torch.roll(p[d], (CY[d], CX[d]), (0, 1)) for d in range(9)])


class _Poisson:
    """Spectral in x, three-point in y, Dirichlet walls: sine transform down the interior rows."""

    def __init__(self, c, zeta, dev):
        nx, n = c["nx"], c["ny"] - 2
        j = torch.arange(1, n + 1, device=dev, dtype=torch.float64)
        self.s = torch.sin(math.pi / (n + 1) * torch.outer(j, j))
        lam = 4.0 * torch.sin(0.5 * math.pi / (n + 1) * j) ** 2
        k = 2.0 * math.pi / nx * torch.arange(nx // 2 + 1, device=dev, dtype=torch.float64)
        self.mu = -(lam[:, None] + k[None, :] ** 2) * (0.5 * (n + 1))
        self.c, self.zeta, self.nx = c, zeta, nx

    def __call__(self, q, rq):
        rhs = rq * q[1:-1]
        rhs[0] -= self.zeta
        rhs[-1] -= self.zeta
        f = torch.fft.rfft(rhs, dim=1)
        f = torch.complex(self.s @ f.real, self.s @ f.imag) / self.mu
        f = torch.complex(self.s @ f.real, self.s @ f.imag)
        return torch.cat([self.zeta[None], torch.fft.irfft(f, n=self.nx, dim=1), self.zeta[None]])


def _efield(psi):
    ex = 0.5 * (torch.roll(psi, 1, 1) - torch.roll(psi, -1, 1))
    ey = torch.empty_like(psi)
    ey[1:-1] = 0.5 * (psi[:-2] - psi[2:])
    ey[0], ey[-1] = ey[1], ey[-2]
    return ex, ey


def _channel_steps(c, start, steps):
    """`steps` coupled steps in FP64: the fields after them."""
    dev = start["psi"].device
    p = _params(c)
    d = c["diff"]
    fwp, fwm = 1.0 / (3.0 * p["nu"] + 0.5), 1.0 / (0.25 / (3.0 * p["nu"]) + 0.5)
    iwm, iwp = 1.0 / (3.0 * d + 0.5), 1.0 / (0.25 / (3.0 * d) + 0.5)
    zeta = torch.as_tensor(_walls(c), device=dev, dtype=torch.float64)
    solve = _Poisson(c, zeta, dev)
    psi, ux, uy = start["psi"], start["ux"], start["uy"]
    ex, ey = _efield(psi)
    f = _equilibrium(start["rho"], ux, uy)
    h = _equilibrium(start["cp"], ux + d * ex, uy + d * ey)
    t = _equilibrium(start["cn"], ux - d * ex, uy - d * ey)
    o = list(OPP)
    w = torch.tensor(W, device=dev, dtype=torch.float64)[:, None]
    cw = (torch.exp(-zeta), torch.exp(zeta))
    for step in range(steps):
        if step:
            own = (h[:, [0, -1]].clone(), t[:, [0, -1]].clone())
            f, h, t = _pull(f), _pull(h), _pull(t)
            for q, s, cwall in ((h, own[0], cw[0]), (t, own[1], cw[1])):
                for row, k in ((0, 0), (-1, 1)):
                    q[:, row] = -s[o, k] + 2.0 * w * cwall
        ex, ey = _efield(psi)
        rho, cp, cn = f.sum(0), h.sum(0), t.sum(0)
        force = p["f_charge"] * (cp - cn)
        fx, fy = force * (ex + c["ex"]), force * ey
        mx, my = (f[1] + f[5] + f[8]) - (f[3] + f[6] + f[7]), (f[2] + f[5] + f[6]) - (f[4] + f[7] + f[8])
        ux, uy = (mx + 0.5 * fx) / rho, (my + 0.5 * fy) / rho
        ux[0], uy[0] = -(mx[1] + 0.5 * fx[0]) / rho[1], -(my[1] + 0.5 * fy[0]) / rho[1]
        psi = solve(cp - cn, -p["f_charge"] / p["eps"])
        h = _trt(h, _equilibrium(cp, ux + d * ex, uy + d * ey), iwp, iwm)
        t = _trt(t, _equilibrium(cn, ux - d * ex, uy - d * ey), iwp, iwm)
        g = _trt(f, _equilibrium(rho, ux, uy), fwp, fwm) + _guo(ux, uy, fx, fy, p["nu"], 0.25)
        g[:, 0], g[:, -1] = f[o, 0], f[o, -1]
        f = g
    return dict(rho=rho, ux=ux, uy=uy, cp=cp, cn=cn, psi=psi)


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "channel":
        start = _fields(case, seed, dev)
        end = _channel_steps(case, start, case["steps"])
        out = dict(fields={k: end[k] for k in OUT})
        if case["storage"] == "f64":
            res = []
            for k in ("ux", "cp", "cn", "psi"):
                norm = float(end[k].norm())
                if k == "ux":
                    norm = max(norm, abs(6.0 * case["eps"] * case["zeta"] * case["ex"]) * math.sqrt(case["nx"] * case["ny"]))
                res.append(float((end[k] - start[k]).norm()) / (case["steps"] * norm))
            out["residual"] = np.array(res)
        return out
    if case["kind"] == "forward":
        x, _, flat = _net_inputs(case, seed)
        h, at = np.concatenate([x, np.zeros((len(x), 12), dtype=np.float32)], 1).astype(np.float64), 0
        for l, (i, o) in enumerate(DIMS):
            wl = flat[at:at + i * o].reshape(o, i).astype(np.float64)
            b = flat[at + i * o:at + i * o + o].astype(np.float64)
            at += i * o + o
            h = h @ wl.T + b
            if l < 3:
                h = h / (1.0 + np.exp(-h))
        return h
    return None  # a batch is many channels' steps (minutes); training rounds its operands to BF16 by design
