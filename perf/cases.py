"""Performance cases of the framework: what its users run, through its public entry points.

Kinds of case and the work each stands for:

* ``sim``      a stretch of a network simulation: RK4 Hodgkin-Huxley updates, delayed spike
               delivery and the implicit paracrine solve, from the 1,000-neuron network that a
               user starts with to the 1M-neuron benchmark network; push, pull and automatic
               delivery, fused electrode recording, batches of independent networks
* ``loop``     the reference's own step loop through the drop-in classes: coupling and leapfrog
               step several times, then one paracrine update
* ``pcg``      one field solve to 1e-6 with the Jacobi-PCG, constant or heterogeneous D
* ``mg``       the same system with the multigrid-preconditioned solver
* ``conv``     one 3x3x3 convolution layer of the learned preconditioner in training: forward,
               input gradient and weight gradient
* ``net``      loss and gradients of the learned preconditioner's whole network

Counts and iteration numbers that a last-bit difference can move by one (spike totals, firing
counts, solver iterations) are not returned: the fields they come from are.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

import neuronephys_clean_gb300 as nn

DT = float(np.float32(0.01))        # RK4 step, ms
MODES = {"push": nn.NN_DELIVERY_PUSH, "pull": nn.NN_DELIVERY_PULL, "auto": nn.NN_DELIVERY_AUTO}
STATE = ("V", "M", "H", "N", "GE", "GI")
CONV_SHAPES = ((16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (48, 16))


def listed():
    return [
        # the 1,000-neuron starter network with a 32^3 field: launches and latency
        dict(name="sim_1k", kind="sim", n=1000, k=10, dmax=1, grid=32, steps=100, delivery="push", regions=0, inst=0),
        # a mid-size network with pull delivery and electrodes recorded every tenth step
        dict(name="sim_50k_pull", kind="sim", n=49_999, k=100, dmax=20, grid=48, steps=200, delivery="pull",
             regions=64, inst=0),
        # the benchmark network: 1M neurons, 1e8 synapses, 128^3 field, automatic delivery
        dict(name="sim_1m", kind="sim", n=1_000_000, k=100, dmax=20, grid=128, steps=200, delivery="auto",
             regions=0, inst=0),
        # a batch of independent networks (a parameter sweep) with a field each
        dict(name="sim_batch", kind="sim", n=120_000, k=200, dmax=1, grid=0, steps=200, delivery="push",
             regions=0, inst=24),
        # the reference's loop at its largest chunked network size
        dict(name="loop_15k", kind="loop", n=14_638, k=100, grid=32, steps=10),
        # and at a million neurons
        dict(name="loop_1m", kind="loop", n=1_000_000, k=100, grid=64, steps=10),
        # the paracrine system of the benchmark network, solved by itself
        dict(name="pcg_128", kind="pcg", nx=128, ny=128, nz=128, het=False),
        # an odd-sided heterogeneous volume (a segmented tissue block)
        dict(name="pcg_odd", kind="pcg", nx=97, ny=83, nz=150, het=True),
        # the heterogeneous 256^3 solve, plain and with multigrid
        dict(name="pcg_256", kind="pcg", nx=256, ny=256, nz=256, het=True),
        dict(name="mg_256", kind="mg", nx=256, ny=256, nz=256, het=True),
        # a decoder layer of the preconditioner's network in training
        dict(name="conv_48_16", kind="conv", nx=72, ny=80, nz=96, cin=48, cout=16),
        # the network's loss and gradients on a 64^3 coarse grid
        dict(name="net_64", kind="net", side=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sim", "sim", "batch", "loop", "pcg", "pcg", "mg", "conv", "net"])
    if kind == "sim":
        mode = rng.choice(["push", "pull", "auto"])
        n = _log(rng, 500, 150_000 if mode == "pull" else 600_000)
        k = min(_log(rng, 10, 120), n // 20)
        return dict(kind="sim", n=n, k=k, dmax=rng.choice([1, 5, 20, 40]), grid=rng.randint(16, 100),
                    steps=100 * rng.randint(1, 2), delivery=mode, regions=rng.choice([0, 0, 64]), inst=0)
    if kind == "batch":
        inst = rng.randint(3, 32)
        return dict(kind="sim", n=inst * _log(rng, 1200, 5000), k=_log(rng, 20, 200), dmax=1, grid=0, steps=100,
                    delivery="push", regions=0, inst=inst)
    if kind == "loop":
        return dict(kind="loop", n=_log(rng, 2000, 900_000), k=rng.randint(10, 100), grid=rng.randint(20, 64),
                    steps=rng.randint(4, 10))
    if kind in ("pcg", "mg"):
        side = lambda m: m * rng.randint(max(1, 20 // m), 200 // m)  # noqa: E731
        m = rng.choice([1, 1, 2, 4, 8]) if kind == "pcg" else rng.choice([2, 4, 8, 16])
        return dict(kind=kind, nx=side(m), ny=side(m), nz=side(m), het=rng.random() < 0.5)
    if kind == "conv":
        cin, cout = rng.choice(CONV_SHAPES)
        side = lambda: rng.randint(8, 88 if cin < 64 else 48)  # noqa: E731
        return dict(kind="conv", nx=side(), ny=side(), nz=side(), cin=cin, cout=cout)
    return dict(kind="net", side=4 * rng.randint(2, 16))


# ------------------------------------------------------------------ helpers --

_CTX = None


def _ctx():
    global _CTX
    if _CTX is None:
        _CTX = nn.Context(0)
    return _CTX


class _Memory:
    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner  # torch holds this object, and so the memory, as long as the view lives
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape), "typestr": kind,
                                         "version": 3, "strides": None}


def _view(owner, shape, kind="<f4", ptr=None):
    """A torch view of device memory that `owner` (a DeviceArray, or the object that ptr belongs to) holds."""
    return torch.as_tensor(_Memory(owner, owner.value if ptr is None else ptr, shape, kind), device="cuda")


def _array(t):
    """A framework array with the values of a tensor."""
    a = nn.DeviceArray(_ctx(), tuple(t.shape), np.float32 if t.dtype == torch.float32 else np.int32)
    _view(a, t.shape, "<f4" if t.dtype == torch.float32 else "<i4").copy_(t)
    return a


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(g, *shape, dtype=torch.float32):
    return torch.rand(shape, generator=g, device="cuda", dtype=dtype)


_CYCLE = None


def _cycle():
    """One spike cycle of a single tonically firing neuron (drive 9 uA/cm^2), step by step: rows V, m, h, n."""
    global _CYCLE
    if _CYCLE is None:
        y, past, crossings, rows = [-65.0, 0.05, 0.6, 0.32], -65.0, [], []
        while len(crossings) < 3:
            k = []
            for c in (0.0, 0.5, 0.5, 1.0):
                z = [a + c * DT * b for a, b in zip(y, k[-1])] if k else y
                V, m, h, n = z
                am, an = (V + 40) / 10 / (1 - math.exp(-(V + 40) / 10)), (V + 55) / 100 / (1 - math.exp(-(V + 55) / 10))
                k.append([9.0 - 120 * m ** 3 * h * (V - 50) - 36 * n ** 4 * (V + 77) - 0.3 * (V + 54.4),
                          am * (1 - m) - 4 * math.exp(-(V + 65) / 18) * m,
                          0.07 * math.exp(-(V + 65) / 20) * (1 - h) - h / (1 + math.exp(-(V + 35) / 10)),
                          an * (1 - n) - 0.125 * math.exp(-(V + 65) / 80) * n])
            y = [a + DT / 6 * (p + 2 * q + 2 * r + s) for a, p, q, r, s in zip(y, *k)]
            if past < -20.0 <= y[0]:
                crossings.append(len(rows))
            past = y[0]
            rows.append(list(y))
        _CYCLE = torch.tensor(rows[crossings[1]:crossings[2]], device="cuda").T.contiguous()
    return _CYCLE


# --------------------------------------------------------------- simulation --

def _instances(c):
    """Neuron offsets and grid sides of a batch: sizes spread by a factor of 16, sides 32 to 51."""
    w = np.exp(np.log(16.0) * np.arange(c["inst"]) / max(1, c["inst"] - 1))
    sizes = np.maximum(300, np.floor(c["n"] * w / w.sum())).astype(np.int64)
    sizes[-1] += c["n"] - sizes.sum()
    sides = np.clip(np.rint(32 * (sizes / sizes.min()) ** (1 / 6)), 32, 64).astype(np.int32)
    return np.concatenate([[0], np.cumsum(sizes)]), sides


def _sim_inputs(c, seed):
    """Network, positions and state: neurons on a jittered lattice, targets within about a tenth of the cube,
    a quarter of the neurons firing tonically at random phases (about 15 Hz over the population)."""
    g, n, k = _gen(seed), c["n"], c["k"]
    off, sides = _instances(c) if c["inst"] else (np.array([0, n]), None)
    starts = torch.from_numpy(off).cuda()
    i = torch.arange(n, device="cuda")
    b = torch.searchsorted(starts, i, right=True) - 1
    size, first = (starts[1:] - starts[:-1])[b], starts[b]
    L = torch.ceil(size.double() ** (1 / 3) - 1e-9).long()
    li = i - first
    cell = torch.stack([li % L, (li // L) % L, li // (L * L)])
    pos = ((cell + _rand(g, 3, n)) / L).float().clamp_(0, 1 - 1e-6)
    if c["inst"]:
        tgt = (_rand(g, n, k, dtype=torch.float64) * size[:, None]).long()
    else:
        step = torch.randn((3, n, k), generator=g, device="cuda").mul_(0.1 * float(L[0])).round_().int()
        z, y, x = (torch.remainder(cell[q].int()[:, None] + step[q], int(L[0])) for q in (2, 1, 0))
        tgt = torch.remainder((z * int(L[0]) + y) * int(L[0]) + x, n)
        del step, z, y, x
    d = dict(col=(tgt + first[:, None] if c["inst"] else tgt).int().reshape(-1),
             weight=(_rand(g, n * k) * (2 * 2.5 / k)),               # 2.5 nS of input weight a neuron
             delay=torch.randint(1, c["dmax"] + 1, (n * k,), generator=g, device="cuda", dtype=torch.uint8),
             inh=(_rand(g, n) < 0.2).to(torch.uint8), pos=pos, drive=_rand(g, n) * 8.0,
             gna=(0.8 + 0.4 * _rand(g, len(off) - 1))[b] if c["inst"] else None)
    cyc = _cycle()
    tonic = d["drive"] > 6.0
    at = (_rand(g, n) * cyc.shape[1]).long().clamp_(max=cyc.shape[1] - 1)
    rest = torch.tensor([-65.0, 0.0529, 0.5961, 0.3177], device="cuda")[:, None]
    d["state"] = torch.cat([torch.where(tonic, cyc[:, at], rest + (_rand(g, 4, n) - 0.5) * rest.abs() * 0.02),
                            torch.zeros((2, n), device="cuda")]).float()
    d["regions"] = torch.randint(0, n, (c["regions"], 80), generator=g, device="cuda").int() if c["regions"] else None
    d["off"], d["sides"] = off, sides
    return d


def _prepare_sim(c, seed):
    d = _sim_inputs(c, seed)
    n, k = c["n"], c["k"]
    cfg = nn.default_config(n)
    cfg.seed, cfg.max_delay, cfg.grid, cfg.timescale = seed, c["dmax"], c["grid"], 100
    cfg.delivery, cfg.par_D, cfg.par_rtol, cfg.par_max_iter = MODES[c["delivery"]], 1.0, 1e-6, 5000
    s = nn.Simulation(_ctx(), cfg)
    if c["inst"]:
        s.set_instances(d["off"], d["sides"])
    host = lambda t: t.cpu().numpy()  # noqa: E731
    s.set_network(np.arange(n + 1, dtype=np.int64) * k, host(d["col"]), host(d["weight"]), host(d["delay"]),
                  host(d["inh"]))
    for name, v in zip(STATE + ("IDRIVE", "X", "Y", "Z"), torch.cat([d["state"], d["drive"][None], d["pos"]])):
        s.set_field(name, host(v))
    if c["inst"]:
        s.set_field("GNA_SCALE", host(d["gna"]))
    if c["regions"]:
        s.set_electrodes(host(d["regions"].reshape(-1)), 80 * np.arange(c["regions"] + 1), every=10,
                         capacity=c["steps"] // 10)
    views = {q: _view(s, (n,), ptr=nn.lib().nn_sim_field_ptr(s.handle, nn.FIELDS[q])) for q in STATE}
    return dict(sim=s, views=views)


def _run_sim(c, st):
    s = st["sim"]
    s.step(c["steps"])
    out = dict(st["views"], density=s.density())
    if c["regions"]:
        out["electrodes"] = s.read_electrodes()[1]
    return out


def _normals(seed, n, t):
    """The framework's documented noise stream: Philox2x32-10 and Box-Muller a neuron pair and step."""
    M = 0xFFFFFFFF
    c0 = torch.arange((n + 1) // 2, device="cuda")
    c1 = torch.full_like(c0, t & M)
    key = (seed + 0x9E3779B9 * (seed >> 32) + 0x85EBCA6B * (t >> 32)) & M
    for _ in range(10):
        p = c0 * 0xD256D193
        c0, c1 = ((p >> 32) & M) ^ key ^ c1, p & M
        key = (key + 0x9E3779B9) & M
    u1, u2 = ((c0 >> 8) + 1).double() / 2 ** 24, (c1 >> 8).double() / 2 ** 24
    r = torch.sqrt(-2 * torch.log(u1))
    return torch.stack([r * torch.cos(2 * math.pi * u2), r * torch.sin(2 * math.pi * u2)], 1).reshape(-1)[:n]


def _xr(u):
    return torch.where(u.abs() < 1e-6, 1 + u / 2, u / -torch.expm1(-u))


def _hh(y, drive, gna):
    V, m, h, n, ge, gi = y
    am, an = _xr((V + 40) / 10), 0.1 * _xr((V + 55) / 10)
    q = torch.exp(-(V + 65) / 80)
    cur = drive - gna * m ** 3 * h * (V - 50) - 36 * n ** 4 * (V + 77) - _GL * (V - _EL) - ge * V - gi * (V + 80)
    return torch.stack([cur, am - (am + 4 * torch.exp(-(V + 65) / 18)) * m,
                        0.07 * q ** 4 * (1 - h) - h / (1 + torch.exp(-(V + 35) / 10)),
                        an - (an + 0.125 * q) * n, -ge / 5, -gi / 5])


_GL, _EL = float(np.float32(0.3)), float(np.float32(-54.4))


def _cg(apply, diag, b, x, rtol):
    """Jacobi-PCG in 64 bits."""
    r = b - apply(x)
    z = r / diag
    p, rz, bb = z, (r * z).sum(), (b * b).sum()
    for i in range(20000):
        if i % 10 == 0 and float((r * r).sum()) <= rtol * rtol * float(bb):
            break
        Ap = apply(p)
        a = rz / (p * Ap).sum()
        x, r = x + a * p, r - a * Ap
        z = r / diag
        new = (r * z).sum()
        p, rz = z + (new / rz) * p, new
    return x


def _operator(shape, alpha, beta, D=None):
    """(apply, diagonal) of (1 + beta) I + alpha L_D, zero outside the grid."""
    D = torch.ones(shape, device="cuda", dtype=torch.float64) if D is None else D.double()
    diag = torch.full(shape, 1 + beta, device="cuda", dtype=torch.float64)
    faces = []
    for a in range(3):
        m = shape[a]
        lo, hi = D.narrow(a, 0, m - 1), D.narrow(a, 1, m - 1)
        f = alpha * 2 * lo * hi / (lo + hi)
        faces.append(f)
        diag.narrow(a, 0, m - 1).add_(f)
        diag.narrow(a, 1, m - 1).add_(f)
        for e in (0, m - 1):
            diag.select(a, e).add_(alpha * D.select(a, e))

    def apply(v):
        y = diag * v
        for a, f in enumerate(faces):
            m = shape[a]
            y.narrow(a, 0, m - 1).sub_(f * v.narrow(a, 1, m - 1))
            y.narrow(a, 1, m - 1).sub_(f * v.narrow(a, 0, m - 1))
        return y

    return apply, diag


def _exact_sim(c, seed):
    d = _sim_inputs(c, seed)
    n, k, D = c["n"], c["k"], c["dmax"] + 1
    y, drive = d["state"].double(), d["drive"].double()
    gna = 120.0 * (d["gna"].double() if c["inst"] else 1.0)
    sides = d["sides"] if c["inst"] else np.array([c["grid"]])
    goff = np.concatenate([[0], np.cumsum(sides.astype(np.int64) ** 3)])
    b = torch.searchsorted(torch.from_numpy(d["off"]).cuda(), torch.arange(n, device="cuda"), right=True) - 1
    side = torch.from_numpy(sides).cuda()[b].long()
    v = torch.minimum((d["pos"] * side.float()).long(), side - 1)
    vox = torch.from_numpy(goff).cuda()[b] + v[0] + side * (v[1] + side * v[2])
    u, src = (torch.zeros(int(goff[-1]), device="cuda", dtype=torch.float64) for _ in range(2))
    ring = torch.zeros((D, 2, n), device="cuda", dtype=torch.float64)
    col, w, dl = d["col"].long().view(n, k), d["weight"].double().view(n, k), d["delay"].long().view(n, k)
    samples = []
    for t in range(c["steps"]):
        slot = t % D
        y[4:] += ring[slot]
        ring[slot] = 0
        cur, old = drive + _normals(seed, n, t), y[0]
        k1 = _hh(y, cur, gna)
        k2 = _hh(y + DT / 2 * k1, cur, gna)
        k3 = _hh(y + DT / 2 * k2, cur, gna)
        y = y + DT / 6 * (k1 + 2 * (k2 + k3) + _hh(y + DT * k3, cur, gna))
        j = torch.nonzero((old < -20) & (y[0] >= -20))[:, 0]
        src.index_add_(0, vox[j], torch.ones_like(y[0, j]))
        at = (((t + dl[j]) % D) * 2 + d["inh"].long()[j][:, None]) * n + col[j]
        ring.view(-1).index_add_(0, at.reshape(-1), w[j].reshape(-1))
        if c["regions"] and t % 10 == 0:
            samples.append(y[0][d["regions"].long()].mean(1))
        if (t + 1) % 100 == 0:
            rhs, src = u + src, torch.zeros_like(src)
            for q, m in enumerate(sides):
                one = slice(int(goff[q]), int(goff[q + 1]))
                shape = (int(m),) * 3
                A = _operator(shape, 100 * DT * 1e-3 * int(m) ** 2, 0.0)
                u[one] = _cg(*A, rhs[one].view(shape), u[one].view(shape), 1e-12).reshape(-1)
    out = dict(zip(STATE, y), density=u)
    if c["regions"]:
        out["electrodes"] = torch.stack(samples)
    return out


# ------------------------------------------------------- the reference's loop --

LOOP_VARS = ("V", "M", "N", "H", "EY", "EIN", "EOUTPUT")


def _loop_inputs(c, seed):
    g, n, k = _gen(seed), c["n"], c["k"]
    half = 0.4995 * (c["grid"] - 1)
    return dict(col=torch.randint(0, n, (n, k), generator=g, device="cuda", dtype=torch.int32),
                pos=(2 * _rand(g, 3, n) - 1) * half, V=torch.randn(n, generator=g, device="cuda") * 20 - 55,
                M=_rand(g, n) * 0.2, N=0.2 + 0.3 * _rand(g, n), H=0.3 + 0.4 * _rand(g, n), APPCUR=2 * _rand(g, n))


def _prepare_loop(c, seed):
    ctx, d, n = _ctx(), _loop_inputs(c, seed), c["n"]
    e = nn.HHEphys(ctx, n, seed=seed)
    var = {name: a for name, a in zip(nn.SIM_PARAMS, e.vars)}
    for name in ("V", "M", "N", "H", "APPCUR"):
        _view(var[name], (n,)).copy_(d[name])
    _view(var["ECOUNT"], (n,)).copy_(torch.bincount(d["col"].view(-1), minlength=n))
    net = nn.AdjacencyList(_array(d["col"].view(-1)),
                           _array(torch.arange(n + 1, device="cuda", dtype=torch.int32) * c["k"]))
    p = nn.ParacrineModule.default_params()
    p.nx = p.ny = p.nz = c["grid"]
    p.quirk_firing_list = 0
    g, pos = ctx.empty((n,), np.float32), [_array(v) for v in d["pos"]]
    torch.cuda.synchronize()
    m = nn.ParacrineModule(ctx, g, n, p, *pos)
    views = {name: _view(var[name], (n,)) for name in LOOP_VARS}
    views["density"] = _view(m, (m.G,), ptr=nn.lib().nn_paracrine_density(m.handle))
    views["g_paracrine"] = _view(g, (n,))
    return dict(ephys=e, coupling=nn.AtomicCoupling(ctx, n), net=net, paracrine=m, var=var, views=views, keep=(g, pos))


def _run_loop(c, st):
    e, cp, m, var = st["ephys"], st["coupling"], st["paracrine"], st["var"]
    for _ in range(c["steps"]):
        cp(st["net"], var["EIN"], var["EOUTPUT"], read_count=False)
        m.update_on_fine_timescale(cp)
        e.simulate_ephys()
    m.update_on_own_timescale()
    return st["views"]


def _exact_loop(c, seed):
    d, n, G = _loop_inputs(c, seed), c["n"], c["grid"]
    f = lambda x: float(np.float32(x))  # noqa: E731
    dt, Ar, Ad, g = f(0.4), 5.0, f(0.18), f(0.1)
    V, M, N, H, app = (d[q].double() for q in ("V", "M", "N", "H", "APPCUR"))
    EY, out = torch.zeros_like(V), torch.zeros_like(V)
    count = torch.bincount(d["col"].view(-1), minlength=n).double()
    gen = torch.zeros_like(V)
    semi = lambda a, r, x: (a * dt + (1 - dt / 2 * r) * x) / (1 + dt / 2 * r)  # noqa: E731
    for t in range(c["steps"]):
        fire = out > f(0.1)
        EIN = torch.bincount(d["col"][fire].reshape(-1), minlength=n).double()
        gen += 0.5 * fire
        am, an = _xr((V + 35) / 10), 0.1 * _xr((V + 50) / 10)
        bm, bn = 4 * torch.exp(-(V + 60) / 18), 0.125 * torch.exp(-(V + 60) / 80)
        ah, bh = 0.07 * torch.exp(-V / 20 - 3), 1 / (torch.exp(-3 - 0.1 * V) + 1)
        T = torch.where(count > 0, Ar * EIN / count.clamp(min=1), torch.zeros_like(V))
        M, N, H, EY = semi(am, am + bm, M), semi(an, an + bn, N), semi(ah, ah + bh, H), semi(T, T + Ad, EY)
        na, kk, gl = 120 * M ** 3 * H, 36 * N ** 4, f(0.3)
        E = na * 55 - kk * 72 - gl * 50
        V = semi(E + 3 + 1.5 * _normals(seed, n, t) + app, na + kk + gl + g * EY, V)
        out = 1 / (1 + torch.exp(-(V + 20) / 3))
    # trilinear deposit, Crank-Nicolson solve on the 27-point Laplacian, interpolation
    s = (d["pos"].double() / (G - 1) + 0.5) * (G - 1)
    q = s.long()
    fr = s - q
    K = torch.tensor([1, 3, 1, 3, 14, 3, 1, 3, 1], dtype=torch.float64, device="cuda")
    K = torch.cat([K, torch.tensor([3, 14, 3, 14, -128, 14, 3, 14, 3.0], dtype=torch.float64, device="cuda"), K]) / 30
    lap = lambda v: F.conv3d(v.view(1, 1, G, G, G), K.view(1, 1, 3, 3, 3), padding=1).view(-1)  # noqa: E731
    corners = []
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                w = torch.ones_like(V)
                for a, o in enumerate((dx, dy, dz)):
                    w = w * (fr[a] if o else 1 - fr[a])
                corners.append(((q[0] + dx) + G * ((q[1] + dy) + G * (q[2] + dz)), w))
    u = torch.zeros(G ** 3, dtype=torch.float64, device="cuda")
    for at, w in corners:
        u.index_add_(0, at, w * gen)
    D, decay, pdt = f(2e-5), f(3e-4), 100 * f(0.4)
    A = lambda v: (1 + 0.5 * pdt * decay) * v - 0.5 * D * pdt * lap(v)  # noqa: E731
    L = lap(u)
    x, rhs = (1 - pdt * decay) * u + pdt * D * L, (1 - decay / 2) * u + D / 2 * L
    r = rhs - A(x)
    p, rr, it = r, float((r * r).sum()), 0
    if rr >= f(1e-6):
        while it < 20:
            Ap = A(p)
            a = rr / float((p * Ap).sum())
            x, r, it = x + a * p, r - a * Ap, it + 1
            new = float((r * r).sum())
            if new < f(1e-6):
                break
            p, rr = r + new / rr * p, new
        u = x
    par = sum(w * u[at] for at, w in corners)
    return dict(V=V, M=M, N=N, H=H, EY=EY, EIN=EIN, EOUTPUT=out, density=u, g_paracrine=par)


# ------------------------------------------------------------ field solvers --

def _diffusivity(g, shape):
    """exp of a Gaussian random field of unit variance, correlated over 8 cells."""
    f = torch.fft.rfftn(torch.randn(shape, generator=g, device="cuda"))
    e = [torch.fft.fftfreq(m, device="cuda") for m in shape[:2]] + [torch.fft.rfftfreq(shape[2], device="cuda")]
    r2 = e[0][:, None, None] ** 2 + e[1][None, :, None] ** 2 + e[2][None, None, :] ** 2
    v = torch.fft.irfftn(f * torch.exp(-64 * math.pi ** 2 * r2), s=shape)
    return torch.exp((v - v.mean()) / v.std()).float()


def _field_inputs(c, seed):
    """Operator of a 1 ms backward-Euler step on a unit-cube grid, right-hand side of spike deposits over a
    smooth earlier field."""
    g = _gen(seed)
    shape = (c["nz"], c["ny"], c["nx"])
    D = _diffusivity(g, shape) if c["het"] else None
    z, y, x = (torch.linspace(0, math.pi, m, device="cuda").sin() for m in shape)
    b = 0.05 * z[:, None, None] * y[None, :, None] * x[None, None, :] * _rand(g, 1)
    cells = b.numel()
    at = torch.randint(0, cells, (max(1, cells // 800),), generator=g, device="cuda")
    b.view(-1).index_add_(0, at, torch.poisson(2 * torch.ones(len(at), device="cuda"), generator=g))
    return shape, D, b, 1e-3 * max(shape) ** 2, 1e-4


def _prepare_field(c, seed):
    shape, D, b, alpha, beta = _field_inputs(c, seed)
    ctx = _ctx()
    field = None if D is None else _array(D)
    rhs, x = _array(b.reshape(-1)), ctx.empty((b.numel(),), np.float32)
    torch.cuda.synchronize()
    pcg = nn.PCG(ctx, shape[2], shape[1], shape[0], alpha, beta, field)
    solver = nn.MultigridPCG(pcg) if c["kind"] == "mg" else pcg
    return dict(solver=solver, pcg=pcg, b=rhs, x=x, out=_view(x, shape), keep=field)


def _run_field(c, st):
    st["x"].zero()
    st["solver"].solve(st["b"], st["x"], rtol=1e-6)
    return st["out"]


def _exact_field(c, seed):
    shape, D, b, alpha, beta = _field_inputs(c, seed)
    return _cg(*_operator(shape, alpha, beta, D), b.double(), torch.zeros_like(b, dtype=torch.float64), 1e-11)


# ------------------------------------------------------ learned preconditioner --

def _blocked(t):
    """A dense (C, nz, ny, nx) tensor in the framework's padded layout of eight-channel blocks."""
    C, nz, ny, nx = t.shape
    guard = (nx + 2) * (ny + 3) + 130
    p = F.pad(t, (1, 1, 1, 1, 1, 1)).reshape(C // 8, 8, -1).transpose(1, 2)
    return F.pad(p, (0, 0, guard, guard)).contiguous()


def _conv_inputs(c, seed):
    g = _gen(seed)
    grid = (c["nz"], c["ny"], c["nx"])
    normal = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    return (normal(c["cin"], *grid).relu(), normal(c["cout"], *grid) * 0.1,
            normal(27, c["cin"], c["cout"]) * math.sqrt(2 / (27 * c["cin"])), normal(c["cout"]) * 0.1)


def _prepare_conv(c, seed):
    ctx, grid = _ctx(), (c["nz"], c["ny"], c["nx"])
    x, gy, w, b = (_array(t) for t in _conv_inputs(c, seed))
    torch.cuda.synchronize()
    act = [nn.Activation(ctx, grid, q) for q in (c["cin"], c["cout"], c["cout"], c["cin"])]
    act[0].pack(x)
    act[1].pack(gy)
    dw, db = ctx.empty((27, c["cin"], c["cout"]), np.float32), ctx.empty((c["cout"],), np.float32)
    views = dict(zip(("y", "gx"), (_view(a, (a.channels // 8, a.nbytes // (2 * a.channels), 8), "<i2")
                                   .view(torch.bfloat16) for a in act[2:])))
    views.update(dw=_view(dw, dw.shape), db=_view(db, db.shape))
    ctx.synchronize()
    return dict(x=act[0], gy=act[1], y=act[2], gx=act[3], dw=dw, db=db, b=b, views=views,
                w=nn.conv3d_pack_weights(ctx, w, c["cin"], c["cout"]),
                wt=nn.conv3d_pack_weights(ctx, w, c["cin"], c["cout"], adjoint=True), keep=w)


def _run_conv(c, st):
    ctx = _ctx()
    nn.conv3d_forward(ctx, st["x"], st["w"], st["y"], bias=st["b"], relu=True)
    nn.conv3d_forward(ctx, st["gy"], st["wt"], st["gx"], mask=st["x"])
    st["dw"].zero()
    st["db"].zero()
    nn.conv3d_wgrad(ctx, st["x"], st["gy"], st["dw"], st["db"])
    return st["views"]


def _exact_conv(c, seed):
    x, gy, w, b = _conv_inputs(c, seed)
    x, gy, w = (t.bfloat16().double() for t in (x, gy, w))
    grid = x.shape[1:]
    y = torch.zeros((c["cout"], x[0].numel()), device="cuda", dtype=torch.float64)
    gx = torch.zeros((c["cin"], x[0].numel()), device="cuda", dtype=torch.float64)
    dw = torch.empty((27, c["cin"], c["cout"]), device="cuda", dtype=torch.float64)
    xp, gp, g2 = F.pad(x, (1,) * 6), F.pad(gy, (1,) * 6), gy.reshape(c["cout"], -1)
    for t in range(27):
        o = (t // 9, t // 3 % 3, t % 3)
        at = lambda v, f: v[:, f(o[0]):f(o[0]) + grid[0], f(o[1]):f(o[1]) + grid[1],  # noqa: E731
                            f(o[2]):f(o[2]) + grid[2]].reshape(v.shape[0], -1)
        shifted = at(xp, lambda q: q)
        y += w[t].T @ shifted
        gx += w[t] @ at(gp, lambda q: 2 - q)
        dw[t] = shifted @ g2.T
    y = (y + b.double()[:, None]).relu().view(-1, *grid)
    return dict(y=_blocked(y), gx=_blocked(gx.view(-1, *grid) * (x > 0)), dw=dw, db=g2.sum(1))


NET_LAYERS = ((16, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16),
              (16, 16))


def _net_inputs(c, seed):
    g, m = _gen(seed), c["side"]
    D = _diffusivity(g, (2 * m,) * 3)
    params = []
    for ci, co in NET_LAYERS:
        params += [torch.randn((27, ci, co), generator=g, device="cuda").mul_(math.sqrt(2 / (27 * ci))),
                   torch.randn(co, generator=g, device="cuda") * 0.05]
    rc = torch.randn((m,) * 3, generator=g, device="cuda") * 1e-3
    target = F.avg_pool3d(rc.view(1, 1, m, m, m), 3, 1, 1).view(m, m, m) * 2
    return D, params, rc, target


def _prepare_net(c, seed):
    ctx, m = _ctx(), c["side"]
    D, params, rc, target = _net_inputs(c, seed)
    field, r, t = _array(D), _array(rc), _array(target)
    torch.cuda.synchronize()
    pcg = nn.PCG(ctx, 2 * m, 2 * m, 2 * m, 1e-3 * (2 * m) ** 2, 1e-4, field)
    net = nn.LearnedPreconditioner(pcg, seed=seed)
    net.set_params(torch.cat([p.reshape(-1) for p in params]).cpu().numpy())
    return dict(net=net, pcg=pcg, rc=r, target=t, keep=field)


def _run_net(c, st):
    loss, grad, y = st["net"].net_gradient(st["rc"], st["target"])
    return dict(loss=loss, grad=grad, y=y)


def _exact_net(c, seed):
    D, params, rc, target = _net_inputs(c, seed)
    m = c["side"]
    params = [p.double().requires_grad_() for p in params]
    logd = torch.log(D.double()).view(m, 2, m, 2, m, 2).mean((1, 3, 5))
    s = rc.double().square().mean().sqrt()

    def conv(i, x, relu=True):
        w, b = params[2 * i], params[2 * i + 1]
        y = F.conv3d(x, w.permute(2, 1, 0).reshape(w.shape[2], w.shape[1], 3, 3, 3), b, padding=1)
        return y.relu() if relu else y

    up = lambda v: F.interpolate(v, scale_factor=2, mode="nearest")  # noqa: E731
    x = torch.zeros((1, 16, m, m, m), device="cuda", dtype=torch.float64)
    x[0, 0], x[0, 1] = rc.double() / s, logd
    k0 = conv(1, conv(0, x))
    k1 = conv(3, conv(2, F.avg_pool3d(k0, 2)))
    v = conv(5, conv(4, F.avg_pool3d(k1, 2)))
    v = conv(7, conv(6, torch.cat([up(v), k1], 1)))
    y = conv(10, conv(9, conv(8, torch.cat([up(v), k0], 1))), relu=False)[0, 0]
    loss = 0.5 * (y - target.double() / s).square().sum()
    grad = torch.autograd.grad(loss, params)
    return dict(loss=loss.detach(), grad=torch.cat([q.reshape(-1) for q in grad]), y=y.detach())


# -------------------------------------------------------------- entry points --

_PREPARE = dict(sim=_prepare_sim, loop=_prepare_loop, pcg=_prepare_field, mg=_prepare_field, conv=_prepare_conv,
                net=_prepare_net)
_RUN = dict(sim=_run_sim, loop=_run_loop, pcg=_run_field, mg=_run_field, conv=_run_conv, net=_run_net)
_EXACT = dict(sim=_exact_sim, loop=_exact_loop, pcg=_exact_field, mg=_exact_field, conv=_exact_conv, net=_exact_net)


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, int(seed))
    state["case"] = case
    torch.cuda.synchronize()
    return state


def run(state):
    return _RUN[state["case"]["kind"]](state["case"], state)


def exact(case, seed):
    return _EXACT[case["kind"]](case, int(seed))


def work(case):
    kind = case["kind"]
    if kind == "sim":
        n, steps = case["n"], case["steps"]
        cells = int((_instances(case)[1].astype(np.int64) ** 3).sum()) if case["inst"] else case["grid"] ** 3
        solves = steps // 100
        # state, drive and field in, state and field out, the synapses of the spikes of about 15 Hz; 340
        # operations a neuron update, about 20 iterations of 25 operations a cell a solve
        events = 1.5e-4 * n * steps * case["k"]
        return dict(bytes=52.0 * n + 8.0 * cells + 13.0 * events, flops=340.0 * n * steps + 500.0 * cells * solves)
    if kind == "loop":
        n = case["n"]
        events = 0.05 * n * case["steps"] * case["k"]
        cells = case["grid"] ** 3
        return dict(bytes=4.0 * events + 4.0 * n * 30 + 8.0 * cells, flops=200.0 * n * case["steps"] + 300.0 * cells)
    if kind in ("pcg", "mg"):
        cells = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=(12.0 if case["het"] else 8.0) * cells, flops=25.0 * 100 * cells)
    if kind == "conv":
        vox = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=4.0 * vox * (case["cin"] + case["cout"]), flops=3 * 2.0 * 27 * case["cin"] * case["cout"] * vox)
    m = case["side"] ** 3
    share = (1, 1, 1 / 8, 1 / 8, 1 / 64, 1 / 64, 1 / 8, 1 / 8, 1, 1, 1)
    return dict(bytes=16.0 * m + 8.0 * sum(27 * a * b + b for a, b in NET_LAYERS),
                flops=3 * sum(2.0 * 27 * a * b * m * f for (a, b), f in zip(NET_LAYERS, share)))
