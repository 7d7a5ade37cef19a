"""Workloads of the Bloch-Torrey solver: what its users run, through its public
entry points, from a single step on a small grid to tens of millions of voxels.

listed() names twelve of them, draw() gives others of the same ranges,
prepare() makes what a program has in hand before the call (geometry, flow,
handle, schedule, initial field), run() is one pass of the call, work() what
a pass cannot do without, exact() the same results in 64 bits from plain torch.

Every input is made from a seed: overlapping solid spheres or a thresholded
Gaussian random field as the pore space, the curl of smoothed noise as the
flow (zero on faces that touch solid or the domain's edge), unit transverse
magnetisation in the pore. dx = 1 um, D = 2.3e-9 m^2/s, T1 = 2.5 s, T2 = 2 s,
rho = 10 um/s, dt = 0.9 dx^2 / (6 D).
"""
import ctypes
import math
import os

import numpy as np
import torch

import initializator_gb300 as bt
from initializator_gb300 import closure, rate_closure

DX, D0, T1, T2, RHO, PEQ = 1.0e-6, 2.3e-9, 2.5, 2.0, 1.0e-5, 1.0
DT = 0.9 * DX * DX / (6.0 * D0)
GAMMA = 2.675e8
WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(bt.__file__)), "data", "rate_closure_g0.npz")


def _solve(name=None, **kw):
    c = dict(kind="solve", nx=64, ny=64, nz=64, f64=False, scheme="reference", pore="spheres", feature=6.0,
             porosity=0.65, flow=0.0, grad=0.0, sequence="none", batch=1, rates="bulk", host=False, steps=100)
    c.update(kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # A plugin host that may not allocate steps a small sample by itself:
        # the smallest call, its launches and their latency.
        dict(name="noalloc_48", kind="noalloc", nx=48, ny=48, nz=48, f64=False, porosity=0.65, flow=1e-3),
        # The compatibility configuration (64^3 sphere pack, no flow, no
        # gradient) in the reference's precision: parity runs.
        _solve("fid_f64_64", f64=True, steps=50),
        # The same in FP32: many short steps of a field that fits in L2.
        _solve("fid_f32_64", steps=200),
        # What a user of the reference's program gets by default: its GPU
        # scheme (MacCormack) in FP64 with flow and a static gradient, the
        # field handed in from and back to host memory; odd, non-cubic.
        _solve("gpu_scheme_f64", nx=90, ny=75, nz=66, f64=True, scheme="maccormack", flow=1e-3, grad=0.05, host=True,
               steps=20),
        # Two fluids: per-voxel T1, T2 and D, and the two components' sums.
        _solve("two_fluid_f32", nx=128, ny=112, nz=96, rates="two-fluid", flow=1e-3, steps=40),
        # The headline configuration: 256^3 sphere pack with flow under PGSE,
        # through its 180 degree pulse.
        _solve("pgse_256", nx=256, ny=256, nz=256, scheme="kspace", feature=10.0, porosity=0.6, flow=1e-3, grad=0.1,
               sequence="pgse", steps=200),
        # Multi-echo train (a 180 degree pulse every 10 steps under a constant
        # gradient) on an odd grid, the initial field from host memory.
        _solve("cpmg_odd", nx=201, ny=149, nz=131, scheme="kspace", grad=0.05, sequence="cpmg", host=True, steps=100),
        # q-sweep: one random-field geometry, eight gradient strengths
        # advanced together.
        _solve("qsweep_8", nx=192, ny=192, nz=128, scheme="kspace", pore="grf", feature=3.0, porosity=0.25, flow=1e-3,
               grad=0.3, sequence="pgse", batch=8, steps=40),
        # Many uneven samples advanced side by side (edges 48 to 192).
        dict(name="ragged_12", kind="ragged", samples=12, lo=48, hi=192, sizes=1, grad=0.1, steps=160),
        # The largest: a tight random-field rock with fast flow, a sixteenth of
        # the 1024 x 1024 x 768 problem.
        _solve("large_grf", nx=512, ny=384, nz=256, scheme="kspace", pore="grf", feature=5.0, porosity=0.2, flow=2e-3,
               grad=0.2, sequence="pgse", steps=30),
        # The learned closure end to end: the network once, then the coarse
        # solve with its rates, handle and all.
        dict(name="learned_128", kind="learned", nx=128, ny=128, nz=128, grad=0.0, steps=250),
        # One training step of the closure's network: forward, backward, AdamW.
        dict(name="train_8x32", kind="train", nb=8, nx=32, ny=32, nz=32),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _edges(rng, lo, hi, most):
    """Three edges, most of them odd or ragged, of at most `most` voxels."""
    while True:
        e = [int(round(_log(rng, lo, hi))) for _ in range(3)]
        if e[0] * e[1] * e[2] <= most:
            return dict(zip(("nx", "ny", "nz"), e))


def _rock(rng):
    if rng.random() < 0.6:
        return dict(pore="spheres", feature=rng.choice([4.0, 6.0, 10.0]), porosity=round(rng.uniform(0.5, 0.7), 3))
    return dict(pore="grf", feature=rng.choice([3.0, 5.0]), porosity=round(rng.uniform(0.2, 0.4), 3))


def draw(rng):
    """One more case: each listed one's kind, sizes over its whole range."""
    what = rng.choice(["noalloc", "fid", "fid", "gpu", "fluid", "pgse", "pgse", "cpmg", "qsweep", "ragged", "learned",
                       "train"])
    flow = rng.choice([0.0, round(_log(rng, 2e-4, 2e-3), 6)])
    if what == "noalloc":
        return dict(kind="noalloc", f64=rng.random() < 0.3, porosity=round(rng.uniform(0.5, 0.7), 3), flow=flow,
                    **_edges(rng, 16, 128, 1 << 20))
    if what == "fid":
        f64 = rng.random() < 0.5
        return _solve(f64=f64, flow=flow, grad=rng.choice([0.0, 0.05]), steps=rng.randint(10, 120),
                      **_rock(rng), **_edges(rng, 24, 160, (1 << 18) if f64 else (1 << 21)))
    if what == "gpu":
        return _solve(f64=True, scheme="maccormack", flow=flow, grad=rng.choice([0.0, 0.05]), host=True,
                      steps=rng.randint(5, 30), **_rock(rng), **_edges(rng, 24, 128, 1 << 19))
    if what == "fluid":
        f64 = rng.random() < 0.3
        return _solve(f64=f64, rates="two-fluid", flow=flow, steps=rng.randint(10, 50), **_rock(rng),
                      **_edges(rng, 32, 160, (1 << 18) if f64 else (1 << 21)))
    if what == "pgse":
        e = _edges(rng, 40, 512, 1 << 24)
        return _solve(scheme="kspace", flow=flow, grad=round(rng.uniform(0.02, 0.3), 3), sequence="pgse",
                      steps=rng.randint(20, 120), **_rock(rng), **e)
    if what == "cpmg":
        return _solve(scheme="kspace", flow=flow, grad=0.05, sequence="cpmg", host=True, steps=rng.randint(20, 120),
                      **_rock(rng), **_edges(rng, 40, 256, 1 << 22))
    if what == "qsweep":
        return _solve(scheme="kspace", flow=flow, grad=0.3, sequence="pgse", batch=rng.randint(2, 12),
                      steps=rng.randint(10, 40), **_rock(rng), **_edges(rng, 48, 224, 1 << 21))
    if what == "ragged":
        return dict(kind="ragged", samples=rng.randint(2, 12), lo=rng.randint(24, 64), hi=rng.randint(96, 192),
                    sizes=rng.randint(2, 1 << 20), grad=round(rng.uniform(0.02, 0.2), 3), steps=rng.randint(40, 120))
    if what == "learned":
        e = {k: v // 2 * 2 for k, v in _edges(rng, 32, 160, 1 << 21).items()}
        return dict(kind="learned", grad=rng.choice([0.0, 0.2]), steps=rng.randint(60, 250), **e)
    e = _edges(rng, 12, 64, 1 << 15)
    return dict(kind="train", nb=rng.randint(1, 8), **e)


# ---- inputs -----------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _spheres(shape, radius, porosity, g):
    """Overlapping solid spheres with uniform centres: 1 - porosity = 1 - exp(-n V)."""
    r = int(math.ceil(radius))
    a = torch.arange(-r, r + 1, device="cuda")
    o = torch.cartesian_prod(a, a, a)
    o = o[(o * o).sum(1) <= radius * radius]
    n = max(1, round(-math.log(porosity) * math.prod(shape) / len(o)))
    ctr = torch.stack([torch.randint(0, s, (n,), generator=g, device="cuda") for s in shape], 1)
    solid = torch.zeros(shape, dtype=torch.bool, device="cuda")
    size = torch.tensor(shape, device="cuda")
    for part in ctr.split(4096):
        p = (part[:, None, :] + o[None]).reshape(-1, 3)
        p = p[((p >= 0) & (p < size)).all(1)]
        solid[p[:, 0], p[:, 1], p[:, 2]] = True
    return ~solid


def _smooth(shape, sigma, g):
    x = torch.fft.rfftn(torch.randn(shape, generator=g, device="cuda"))
    for ax, n in enumerate(shape):
        f = torch.fft.rfftfreq(n, device="cuda") if ax == 2 else torch.fft.fftfreq(n, device="cuda")
        view = [1, 1, 1]
        view[ax] = -1
        x *= torch.exp(-2.0 * (math.pi * sigma * f) ** 2).view(view)
    return torch.fft.irfftn(x, s=shape)


def _pore(c, g, shape):
    if c.get("pore", "spheres") == "spheres":
        return _spheres(shape, c.get("feature", 6.0), c["porosity"], g)
    f = _smooth(shape, c["feature"], g)
    s = f.flatten()[:: max(1, f.numel() // 1_000_000)].sort().values
    return f <= s[int(c["porosity"] * (len(s) - 1))]


def _flow(pore, vmax, g):
    """Face velocities (float64, CUDA): curl of a smoothed potential on the edges."""
    nz, ny, nx = pore.shape
    ax, ay, az = (_smooth((nz + 1, ny + 1, nx + 1), 4.0, g) for _ in range(3))
    v = [(az[:nz, 1:] - az[:nz, :ny]) - (ay[1:, :ny] - ay[:nz, :ny]),
         (ax[1:, :, :nx] - ax[:nz, :, :nx]) - (az[:nz, :, 1:] - az[:nz, :, :nx]),
         (ay[:, :ny, 1:] - ay[:, :ny, :nx]) - (ax[:, 1:, :nx] - ax[:, :ny, :nx])]
    for q, dim in zip(v, (2, 1, 0)):
        n = pore.shape[dim]
        q.narrow(dim, 1, n - 1).mul_(pore.narrow(dim, 1, n - 1) & pore.narrow(dim, 0, n - 1))
        q.narrow(dim, 0, 1).zero_()
        q.narrow(dim, n, 1).zero_()
    top = max(float(q.abs().max()) for q in v)
    return [q.double() * (vmax / max(top, 1e-30)) for q in v]


def _samples(c):
    """The samples of a ragged batch: each edge uniform in [lo, hi], porosity in [0.5, 0.7]."""
    r = np.random.default_rng(c["sizes"])
    out = []
    for _ in range(c["samples"]):
        e = [int(v) for v in r.integers(c["lo"], c["hi"] + 1, 3)]
        out.append(_solve(nx=e[0], ny=e[1], nz=e[2], scheme="kspace", porosity=float(r.uniform(0.5, 0.7)),
                          grad=c["grad"], sequence="pgse", steps=c["steps"]))
    return out


def _two_fluids(pore, g):
    """(c1, T1, T2, D): the first fluid's fraction and the mixed coefficients."""
    c1 = torch.sigmoid(350.0 * _smooth(tuple(pore.shape), 6.0, g).double())
    t1 = 1.0 / (c1 / 2.5 + (1 - c1) / 1.2)
    t2 = 1.0 / (c1 / 2.0 + (1 - c1) / 0.8)
    d = D0 * c1 + 0.4 * D0 * (1 - c1)
    big = torch.full_like(c1, 1e50)
    return c1, torch.where(pore, t1, big), torch.where(pore, t2, big), torch.where(pore, d, 1.0 / big)


def _waveform(c, n):
    """Per-step gradients along z (T/m) and the RF pulses of a sequence."""
    t0 = np.arange(n) * DT
    if c["sequence"] == "pgse":  # two 2 ms lobes 20 ms apart, a 180 degree pulse between them
        f = sum(np.clip(np.minimum(t0 + DT, b + 2e-3) - np.maximum(t0, b), 0.0, None) / DT for b in (0.0, 20e-3))
        rf = [(max(0, math.ceil(10e-3 / DT) - 1), 2, math.pi, (1.0, 0.0, 0.0))]
    elif c["sequence"] == "cpmg":
        f = np.ones(n)
        rf = [(s, 2, math.pi, (1.0, 0.0, 0.0)) for s in range(4, n, 10)]
    else:
        return None, []
    return np.stack([0 * f, 0 * f, f * c["grad"]], 1), [p for p in rf if p[0] < n]


def _inputs(c, seed):
    """Everything a solve needs, on the GPU: pore, face velocities, fluids, waves, pulses."""
    g, shape = _gen(seed), (c["nz"], c["ny"], c["nx"])
    pore = _pore(c, g, shape)
    vel = _flow(pore, c["flow"], g) if c.get("flow") else None
    fluids = _two_fluids(pore, g) if c.get("rates") == "two-fluid" else None
    wave, rf = _waveform(c, c["steps"]) if c.get("sequence") else (None, [])
    if wave is not None:
        b = c.get("batch", 1)
        wave = wave[:, None, :] * (np.linspace(0.0, 1.0, b) if b > 1 else np.ones(1))[None, :, None]
    return pore, vel, fluids, wave, rf


def _config(c, shape):
    scheme = {"reference": bt.BT_SCHEME_REFERENCE, "kspace": bt.BT_SCHEME_KSPACE,
              "maccormack": bt.BT_SCHEME_MACCORMACK}[c.get("scheme", "reference")]
    static = c.get("grad", 0.0) if c.get("sequence", "none") == "none" else 0.0
    return bt.make_config(shape, precision=bt.BT_F64 if c.get("f64") else bt.BT_F32, scheme=scheme, dx=DX, dt=DT,
                          main_field=(0.0, 0.0, 1.0), gamma=GAMMA, grad=(0.0, 0.0, static),
                          vector_mult=1 if static else 0, d_pore=D0, t1=T1, t2=T2, rho1=RHO, rho2=RHO, p_eq=PEQ,
                          velocity=1 if c.get("flow") else 0, batch=c.get("batch", 1))


def _host(ts):
    return None if ts is None else [t.cpu().numpy() for t in ts]


class _Sample:
    """A solver with its geometry and schedule, and the field it starts from."""

    def __init__(self, c, seed):
        pore, vel, fluids, wave, rf = _inputs(c, seed)
        shape = tuple(pore.shape)
        self.c, self.solver = c, bt.Solver(_config(c, shape))
        s = self.solver
        s.upload_geometry(pore.to(torch.uint8).cpu().numpy(), _host(vel))
        if fluids is not None:
            c1, t1, t2, d = _host(fluids)
            s.upload_rates(t1, t2, d)
            s.set_phase_weights(c1, 1.0 - c1)
        if wave is not None:
            s.set_schedule(rf, grad_wave=wave)
        m = pore.to(torch.float64 if c.get("f64") else torch.float32)
        if c.get("host"):
            self.start = np.zeros((3,) + shape)
            self.start[0] = pore.cpu().numpy()
        else:
            b = (c["batch"],) if c.get("batch", 1) > 1 else ()
            mx = m.expand(b + shape).contiguous()
            self.start = [mx, torch.zeros_like(mx), torch.zeros_like(mx)]

    def rewind(self):
        self.solver.set_step(0)
        if self.c.get("host"):
            self.solver.set_state(self.start)
        else:
            self.solver.set_state_device(self.start)

    def sums(self, mt):
        """The sums in the precision of the fields that they are of."""
        return mt if self.c.get("f64") else mt.astype(np.float32)

    def fields(self):
        out = []
        for b in range(self.solver.batch):
            for v in self.solver.field_views(b):
                v.sample = self  # the view reads the handle's memory
                out.append(v)
        return out


def prepare(case, seed):
    c, k = dict(case), case["kind"]
    if k == "solve":
        return _Sample(c, seed)
    if k == "ragged":
        return [_Sample(one, seed * 100 + i) for i, one in enumerate(_samples(c))]
    if k == "noalloc":
        shape = (c["nz"], c["ny"], c["nx"])
        pore, vel, _, _, _ = _inputs(c, seed)
        t = torch.float64 if c["f64"] else torch.float32
        mx = pore.to(t)
        bufs = [pore.to(torch.uint8).contiguous()]
        bufs += [v.to(t).contiguous() for v in vel] if vel else [None] * 3
        bufs += [mx, torch.zeros_like(mx), torch.zeros_like(mx)] + [torch.empty_like(mx) for _ in range(3)]
        bufs.append(torch.zeros(3, dtype=torch.float64, device="cuda"))
        return dict(case=c, cfg=_config(c, shape), bufs=bufs)
    if k == "learned":
        return dict(case=c, rc=_rate_case(c, seed), net=rate_closure.RateClosure.load(WEIGHTS))
    g = _gen(seed)
    lay = closure.PaddedRows(c["nb"], c["nz"], c["ny"], c["nx"])
    x = torch.randn((c["nb"], c["nz"], c["ny"], c["nx"], 8), generator=g, device="cuda")
    y = torch.randn((c["nb"], c["nz"], c["ny"], c["nx"], 16), generator=g, device="cuda")
    full = torch.zeros((c["nb"], c["nz"] + 2, c["ny"] + 2, c["nx"] + 2, 16), device="cuda")
    full[:, 1:-1, 1:-1, 1:-1] = y
    net = closure.Net(seed=int(seed) % (1 << 30), zero_last=False)
    return dict(case=c, lay=lay, x=lay.pack(x, "cuda"), target=full.reshape(-1, 16), net=net)


def _rate_case(c, seed):
    g, shape = _gen(seed), (c["nz"], c["ny"], c["nx"])
    pore = _spheres(shape, 6.0, 0.65, g)
    vel = _flow(pore, 1e-3, g)
    n = 4 * c["steps"]
    wave = _learned_wave(c, n)
    kw = dict(dx=DX, dt=DT, d_pore=D0, t1=T1, t2=T2, rho1=RHO, rho2=RHO, p_eq=PEQ, velocity=1, diffusion=1,
              gamma=GAMMA)
    fine = closure.Case(pore.to(torch.uint8).cpu().numpy(), _host(vel), wave, _learned_pulses(n), kw)
    return rate_closure.RateCase(fine, c["steps"])


def _learned_wave(c, n):
    return _waveform(dict(sequence="pgse", grad=c["grad"]), n)[0]


def _learned_pulses(n):
    s = 4 * math.ceil(10e-3 / DT / 4) - 1  # at the end of a coarse step
    return [(s, 2, math.pi, (1.0, 0.0, 0.0))] if s < n else []


# ---- one pass ---------------------------------------------------------------


def run(state):
    if isinstance(state, _Sample):
        c, s = state.c, state.solver
        state.rewind()
        mt = s.run(c["steps"])
        out = {"mt": state.sums(mt)}
        if c["rates"] == "two-fluid":
            out["phases"] = state.sums(s.read_mt_phases(c["steps"]))
        if c["host"] and c["f64"]:
            out["m"] = list(s.get_state())  # back to the host, as the reference's program does
        else:
            out["m"] = state.fields()
        return out
    if isinstance(state, list):
        for one in state:
            one.rewind()
        mts = bt.run_many([one.solver for one in state], state[0].c["steps"])
        return [{"mt": one.sums(mt), "m": one.fields()} for one, mt in zip(state, mts)]
    c = state["case"]
    if c["kind"] == "noalloc":
        b = state["bufs"]
        rc = bt.lib().bt_step_noalloc(ctypes.byref(state["cfg"]), *[None if t is None else t.data_ptr() for t in b],
                                      torch.cuda.current_stream().cuda_stream)
        if rc:
            raise bt.BtError(rc, "bt_step_noalloc")
        return {"m": b[7:10], "mt": b[10] if c["f64"] else b[10].float()}
    if c["kind"] == "learned":
        rc = state["rc"]
        with torch.no_grad():
            corr, _, _ = state["net"].predict([rc])
        s = rc.solver(corr[0])
        mt = 8.0 * s.run(rc.n)
        s.close()
        return {"correction": corr[0], "mt": mt.astype(np.float32)}
    net, lay = state["net"], state["lay"]
    y = net.forward(lay, state["x"])
    dy = (y - state["target"]) * (2.0 / (c["nb"] * c["nx"] * c["ny"] * c["nz"]))
    net.backward(lay, dy)
    net.adamw(lr=1e-4)
    return {"y": y, "grad": net.grad, "flat": net.flat}


# ---- what a pass cannot do without --------------------------------------------


def _voxel_steps(c, voxels):
    """A time step reads the field and the flow and writes the field: 3 values
    each way, 3 velocities and the geometry byte a voxel (the batch shares the
    last two); about 13 operations a face and component, as one fused sum."""
    w = 8 if c.get("f64") else 4
    b = c.get("batch", 1)
    per = 6 * w * b + (3 * w if c.get("flow") else 0) + 1
    if c.get("rates") == "two-fluid":  # T1, T2 and D of each voxel, both fractions
        per += 5 * w
    ops = (70 + (12 if c.get("flow") else 0) + (30 if c.get("sequence", "none") != "none" else 0)) * b
    if c.get("scheme") == "maccormack":
        ops *= 2
    return {"bytes": per * voxels * c.get("steps", 1), "flops": ops * voxels * c.get("steps", 1)}


def work(case):
    c = case
    if c["kind"] == "ragged":
        return _voxel_steps(dict(sequence="pgse", steps=c["steps"]), sum(o["nx"] * o["ny"] * o["nz"] for o in _samples(c)))
    voxels = c["nx"] * c["ny"] * c["nz"]
    if c["kind"] in ("solve", "noalloc"):
        return _voxel_steps(c, voxels)
    conv = 2 * 27 * 16 * 16  # operations of one 3x3x3 convolution a voxel
    if c["kind"] == "learned":
        w = _voxel_steps(dict(flow=1, sequence="pgse", steps=c["steps"]), voxels / 8)
        return {"bytes": w["bytes"] + voxels / 8 * (32 + 4 + 3 * 64), "flops": w["flops"] + 4 * conv * voxels / 8}
    n = c["nb"] * voxels
    # forward: x, the three layers' activations and pre-activations written, y;
    # backward: those read again, dy, three layers' gradients written and read
    return {"bytes": n * (32 + 3 * 96 + 64 + 3 * 96 + 32 + 64 + 3 * 64), "flops": 11 * conv * n}


# ---- the same in 64 bits ------------------------------------------------------


def _lo(a, dim):
    return torch.cat([a.narrow(dim, 0, 1), a.narrow(dim, 0, a.shape[dim] - 1)], dim)


def _hi(a, dim):
    return torch.cat([a.narrow(dim, 1, a.shape[dim] - 1), a.narrow(dim, a.shape[dim] - 1, 1)], dim)


class _Exact:
    """The three updates in FP64 on whole arrays; copy ghosts on the domain's faces."""

    def __init__(self, pore, vel, d, dx, dt, fluids=None, rate=None, p_eq=PEQ):
        self.pore, self.dx, self.dt, self.peq = pore, dx, dt, p_eq
        diff = torch.where(pore, torch.full_like(pore, d, dtype=torch.float64), 1e-50) if fluids is None else fluids[3]
        if fluids is not None:
            self.r1, self.r2 = 1.0 / fluids[1], 1.0 / fluids[2]
        elif rate is not None:
            self.r1, self.r2 = rate
        else:
            faces = sum((~f(pore, ax)).double() for ax in range(3) for f in (_lo, _hi))
            self.r1, self.r2 = 1.0 / T1 + RHO / dx * faces, 1.0 / T2 + RHO / dx * faces
        # per axis x, y, z: (dimension, low and high face weights, face velocities, open faces)
        self.ax = []
        for a, dim in enumerate((2, 1, 0)):
            w = [dt / dx ** 2 * 2 * diff * f(diff, dim) / (diff + f(diff, dim) + 1e-50) for f in (_lo, _hi)]
            v = (None, None)
            if vel is not None:
                n = pore.shape[dim]
                v = (vel[a].narrow(dim, 0, n), vel[a].narrow(dim, 1, n))
            self.ax.append((dim, w, v))

    def near(self, m, dim, side, phase):
        """The neighbours at one side, in the frame of the voxel (KSPACE: phase = (c, s) of the face)."""
        f = _lo if side == 0 else _hi
        q = [f(t, dim) for t in m]
        if phase is not None and phase[1] != 0.0:
            c, s = phase[0], phase[1] if side == 0 else -phase[1]
            r = [c * q[0] - s * q[1], c * q[1] + s * q[0]]
            at = 0 if side == 0 else m[0].shape[dim] - 1
            for i in range(2):
                r[i].narrow(dim, at, 1).copy_(m[i].narrow(dim, at, 1))
            q[:2] = r
        return q

    def rates(self, m, form, n, grad=None, phases=None):
        """The change of m in one step: relaxation, precession, diffusion, advection."""
        dt = self.dt
        div = sum(n[i] * m[i] for i in range(3))
        out = [dt * self.r1 * (self.peq * n[i] - n[i] * div) + dt * self.r2 * (n[i] * div - m[i]) for i in range(3)]
        if grad is not None:
            nz, ny, nx = m[0].shape
            pos = [torch.arange(k, device="cuda", dtype=torch.float64) + 0.5 for k in (nx, ny, nz)]
            b = [dt * GAMMA * grad[a] * self.dx * pos[a].view([-1 if i == 2 - a else 1 for i in range(3)]) for a in range(3)]
            out[0] += b[2] * m[1] - b[1] * m[2]
            out[1] += b[0] * m[2] - b[2] * m[0]
            out[2] += b[1] * m[0] - b[0] * m[1]
        h = dt / self.dx
        for a, (dim, w, v) in enumerate(self.ax):
            ph = None if phases is None else phases[a]
            lo, hi = self.near(m, dim, 0, ph), self.near(m, dim, 1, ph)
            for i in range(3):
                out[i] += w[0] * (lo[i] - m[i]) + w[1] * (hi[i] - m[i])
            if v[0] is None:
                continue
            u = 0.5 * (v[0] + v[1])
            for i in range(3):
                if form == "upwind":
                    out[i] -= 0.5 * h * ((u - u.abs()) * (hi[i] - m[i]) * (v[1] != 0) + (u + u.abs()) * (m[i] - lo[i]) * (v[0] != 0))
                elif form == "backward":
                    out[i] -= u * h * (m[i] - lo[i]) * _lo(self.pore, dim)
                else:
                    out[i] -= u * h * (hi[i] - m[i]) * _hi(self.pore, dim)
        return [torch.where(self.pore, t, 0.0) for t in out]

    def run(self, scheme, m, steps, grad=None, wave=None, rf=()):
        """(M(t), final field); KSPACE: the field in the frame of the last step's wave vector."""
        n = (0.0, 0.0, 1.0)
        k = np.zeros(3)
        mt = []
        for s in range(steps):
            if scheme == "maccormack":
                p = [a + b for a, b in zip(m, self.rates(m, "backward", n, grad))]
                m = [0.5 * (a + b + r) for a, b, r in zip(m, p, self.rates(p, "forward", n, grad))]
            else:
                phases = None
                if scheme == "kspace":
                    gdt = GAMMA * (wave[s] if wave is not None else np.zeros(3)) * self.dt
                    th = (k + 0.5 * gdt) * self.dx
                    phases = [(math.cos(t), math.sin(t)) for t in th]
                    k = k + gdt
                m = [a + b for a, b in zip(m, self.rates(m, "upwind", n, grad, phases))]
            e = None
            if k.any():
                pos = [torch.arange(q, device="cuda", dtype=torch.float64) + 0.5 for q in reversed(m[0].shape)]
                ang = sum(float(k[a]) * self.dx * pos[a].view([-1 if i == 2 - a else 1 for i in range(3)]) for a in range(3))
                e = (torch.cos(ang), -torch.sin(ang))
            lab = m if e is None else [e[0] * m[0] - e[1] * m[1], e[0] * m[1] + e[1] * m[0], m[2]]
            for step, _, angle, ax in rf:
                if step != s:
                    continue
                cs, sn = math.cos(angle), math.sin(angle)
                dot = sum(ax[i] * lab[i] for i in range(3))
                cross = [ax[1] * lab[2] - ax[2] * lab[1], ax[2] * lab[0] - ax[0] * lab[2], ax[0] * lab[1] - ax[1] * lab[0]]
                lab = [lab[i] * cs + ax[i] * (1 - cs) * dot + sn * cross[i] for i in range(3)]
                m = lab if e is None else [e[0] * lab[0] + e[1] * lab[1], e[0] * lab[1] - e[1] * lab[0], lab[2]]
            mt.append(self.totals(lab))
        return mt, m

    def totals(self, lab):
        return torch.stack([t.sum() for t in lab])


def _exact_solve(c, seed):
    pore, vel, fluids, wave, rf = _inputs(c, seed)
    x = _Exact(pore, vel, D0, DX, DT, fluids)
    if fluids is not None:
        c1, c2 = fluids[0], 1.0 - fluids[0]
        w = [torch.where(((c1 > 0.8) | (c2 > 0.8)) & pore, q, 0.0) for q in (c1, c2)]
        x.totals = lambda lab: torch.stack([t.sum() for t in lab] + [(t * q).sum() for q in w for t in lab])
    grad = (0.0, 0.0, c["grad"]) if c["sequence"] == "none" and c["grad"] else None
    mts, fields = [], []
    for b in range(c["batch"]):
        m = [pore.double(), torch.zeros_like(pore, dtype=torch.float64), torch.zeros_like(pore, dtype=torch.float64)]
        mt, m = x.run(c["scheme"], m, c["steps"], grad, None if wave is None else wave[:, b], rf)
        mts.append(torch.stack(mt).cpu().numpy())
        fields += m
    mt = mts[0] if c["batch"] == 1 else np.stack(mts, 1)
    out = {"mt": mt[..., :3], "m": fields}
    if fluids is not None:
        out["phases"] = mt[:, 3:]
    return out


def _conv(x, w, b):
    """3x3x3 convolution of (n, z, y, x, 16) by w[27][ci][co], zero halo."""
    k = w.view(3, 3, 3, 16, 16).permute(4, 3, 0, 1, 2)
    return torch.nn.functional.conv3d(x.permute(0, 4, 1, 2, 3), k, b, padding=1).permute(0, 2, 3, 4, 1)


def _net(x, flat):
    w, b = flat[: 4 * 27 * 256].view(4, 27, 16, 16), flat[4 * 27 * 256:].view(4, 16)
    for i in range(4):
        x = _conv(x, w[i], b[i])
        if i < 3:
            x = torch.nn.functional.gelu(x)
    return x


def _exact_learned(c, seed):
    g, shape = _gen(seed), (c["nz"], c["ny"], c["nx"])
    pore = _spheres(shape, 6.0, 0.65, g)
    vel = _flow(pore, 1e-3, g)
    cs = [n // 2 for n in shape]

    def mean(t, dims):  # over pairs along the given dimensions
        for d in dims:
            t = t.unflatten(d, (-1, 2)).mean(d + 1)
        return t

    phi = mean(pore.double(), (0, 1, 2))
    pc = phi > 0
    v = [mean(vel[0][:, :, ::2], (0, 1)), mean(vel[1][:, ::2], (0, 2)), mean(vel[2][::2], (1, 2))]
    dx, dt = 2 * DX, 4 * DT

    def faces(p):
        return torch.where(p, sum((~f(p, ax)).double() for ax in range(3) for f in (_lo, _hi)), 0.0)

    nc = faces(pc)
    nf = torch.where(pc, mean(faces(pore), (0, 1, 2)) / phi.clamp(min=1 / 8), 0.0)
    u = [0.5 * (q.narrow(d, 0, n) + q.narrow(d, 1, n)) * dt / dx for q, d, n in zip(v, (2, 1, 0), reversed(cs))]
    feats = [phi, nc / 6, nf / 6, pc.double()] + u + [sum(q * q for q in u).sqrt()]
    x = torch.zeros([1] + cs + [16], dtype=torch.float64, device="cuda")
    x[0, ..., :8] = torch.stack(feats, -1)
    z = np.load(WEIGHTS)
    y = _net(x, torch.as_tensor(z["flat"], device="cuda").double())[0, ..., 0] * float(z["scale"]) * pc
    # rates on a grid of 1 / (2 k) of one fine face's, at most 255 levels
    surf = (0.5 * nc + y).clamp(min=0.0)
    top = float(surf[pc].max())
    k = max(1, int(127.0 / top)) if top > 0 else 1
    surf = torch.round(surf * (2 * k)) / (2 * k)
    xct = _Exact(pc, v, D0, dx, dt, rate=(1 / T1 + RHO / DX * surf, 1 / T2 + RHO / DX * surf))
    n = c["steps"]
    wave = _learned_wave(c, 4 * n).reshape(n, 4, 3).mean(1)
    rf = [((s - 3) // 4, f, p, ax) for s, f, p, ax in _learned_pulses(4 * n)]
    mt, _ = xct.run("kspace", [phi, torch.zeros_like(phi), torch.zeros_like(phi)], n, None, wave, rf)
    return {"correction": y, "mt": 8.0 * torch.stack(mt).cpu().numpy()}


def _exact_train(c, seed):
    s = prepare(c, seed)
    net, shape = s["net"], (c["nb"], c["nz"], c["ny"], c["nx"])
    flat = net.flat.double().requires_grad_(True)
    inside = (slice(None),) + (slice(1, -1),) * 3
    box = (c["nb"], c["nz"] + 2, c["ny"] + 2, c["nx"] + 2, 16)
    margin = (s["x"].shape[0] - math.prod(box[:4])) // 2
    x = s["x"][margin: margin + math.prod(box[:4])].double().view(box)[inside]
    y = _net(x, flat)
    scale = 1.0 / math.prod(shape)
    ((y - s["target"].double().view(box)[inside]) ** 2).sum().mul(scale).backward()
    g = flat.grad
    p = flat.detach() * (1 - 1e-4 * 0.01) - 1e-4 * g / (g.abs() + 1e-8)  # the first AdamW step
    full = torch.zeros(box, dtype=torch.float64, device="cuda")
    full[inside] = y.detach()
    return {"y": full.view(-1, 16), "grad": g, "flat": p}


def exact(case, seed):
    c, k = dict(case), case["kind"]
    if k == "solve":
        return _exact_solve(c, seed)
    if k == "ragged":
        return [_exact_solve(one, seed * 100 + i) for i, one in enumerate(_samples(c))]
    if k == "noalloc":
        o = _exact_solve(dict(_solve(), **c, steps=1), seed)
        return {"m": o["m"], "mt": o["mt"][0]}
    return _exact_learned(c, seed) if k == "learned" else _exact_train(c, seed)
