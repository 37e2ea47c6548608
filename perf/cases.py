"""The calls that a user of this framework makes, as measured cases.

Each case names one call of the public API and its sizes; `prepare` builds
what a program holds before that call, `run` is the call, and `exact` gives
the same outputs from plain torch in 64 bits.  Kinds:

* step      one RK3 step of the finite-volume solver (periodic box, explicit
            or semi-implicit channel), optionally preceded by its CFL
            reduction and followed by the shell forcing, as `solve` runs it;
* solve     a short `solve` of a channel with its statistics, fields
            allocated and the initial state projected as part of the call;
* ensemble  a batched ensemble of forced periodic boxes of uneven sizes;
* infer     the closure network evaluated on a periodic staggered field;
* train     Adam steps of the closure on random crops of its dataset;
* les       a CFL-adaptive interval of the closed, forced LES;
* spectral  one step of the pseudo-spectral solver.
"""
import math

import numpy as np
import torch

import distributednavierstokes_b200 as dns
from distributednavierstokes_b200 import closure, les_closure, spectral

DEV = "cuda"
F64 = torch.float64
CHANNELS = (3, 32, 32, 32, 6)


# ------------------------------------------------------------------ cases

def listed():
    return [
        # the smallest box of an ensemble and of a parameter study: launches count
        dict(name="box32_step", kind="step", nx=32, ny=32, nz=32, wall=False, implicit=False,
             cfl=False, forced=False),
        # the explicit test channel, stepped as solve does: CFL number, then the step
        dict(name="channel64_cfl_step", kind="step", nx=64, ny=64, nz=64, wall=True,
             implicit=False, cfl=True, forced=False),
        # a channel of no special length: ragged lines, an odd row count
        dict(name="ragged_channel_step", kind="step", nx=100, ny=75, nz=90, wall=True,
             implicit=True, cfl=False, forced=False),
        # forced isotropic turbulence at an everyday resolution
        dict(name="box128_forced_step", kind="step", nx=128, ny=128, nz=128, wall=False,
             implicit=False, cfl=False, forced=True),
        # the DNS that the closure's data come from
        dict(name="box256_step", kind="step", nx=256, ny=256, nz=256, wall=False, implicit=False,
             cfl=False, forced=False),
        # the production channel
        dict(name="channel384_cfl_step", kind="step", nx=384, ny=256, nz=384, wall=True,
             implicit=True, cfl=True, forced=False),
        # a whole solve with statistics after every step
        dict(name="channel96_solve", kind="solve", nx=96, ny=72, nz=80, implicit=False, steps=8),
        # uneven boxes advanced together
        dict(name="ensemble16", kind="ensemble", members=16, sizes="32,48,64,96,128", steps=4,
             forced=True),
        # the closure alone, on the LES grid
        dict(name="infer64", kind="infer", n=64),
        # the closure's training, in the batches it is trained with
        dict(name="train8x32", kind="train", batch=8, crop=32, n=64, snapshots=4, steps=4),
        # the closed LES between two samples
        dict(name="les64", kind="les", n=64, interval=0.4),
        # the pseudo-spectral solver at production size
        dict(name="spectral256_step", kind="spectral", n=256),
    ]


def _smooth(lo, hi):
    """The 5-smooth integers of [lo, hi]."""
    out = []
    for m in range(lo, hi + 1):
        r = m
        for q in (2, 3, 5):
            while r % q == 0:
                r //= q
        if r == 1:
            out.append(m)
    return out


def _pick(rng, values):
    """One of the sorted values, spread over their logarithm."""
    t = math.exp(rng.uniform(math.log(values[0]), math.log(values[-1])))
    return min(values, key=lambda v: abs(math.log(v / t)))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "step", "step", "solve", "ensemble", "infer",
                       "train", "les", "spectral"))
    even = [2 * m for m in _smooth(10, 192)]
    if kind == "step":
        wall = rng.random() < 0.55
        while True:
            n = (_pick(rng, even), rng.randint(20, 256) if wall else _pick(rng, _smooth(20, 256)),
                 _pick(rng, _smooth(20, 384)))
            if n[0] * n[1] * n[2] <= 384 * 256 * 384:
                break
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], wall=wall,
                    implicit=wall and rng.random() < 0.5, cfl=rng.random() < 0.5,
                    forced=not wall and rng.random() < 0.3)
    if kind == "solve":
        return dict(kind=kind, nx=_pick(rng, even[:60]), ny=rng.randint(20, 144),
                    nz=_pick(rng, _smooth(20, 144)), implicit=rng.random() < 0.5,
                    steps=rng.randint(3, 12))
    if kind == "ensemble":
        sizes = sorted(rng.sample((24, 32, 40, 48, 60, 64, 80, 96, 108, 128), rng.randint(2, 5)))
        return dict(kind=kind, members=rng.randint(3, 16), sizes=",".join(map(str, sizes)),
                    steps=rng.randint(2, 6), forced=rng.random() < 0.5)
    if kind == "infer":
        return dict(kind=kind, n=_pick(rng, list(range(12, 89))))
    if kind == "train":
        crop = rng.choice((12, 14, 16, 18, 20, 22, 24, 26, 28, 30, 32, 36, 40))
        return dict(kind=kind, batch=rng.randint(1, max(1, min(16, 300000 // crop ** 3))),
                    crop=crop, n=rng.choice((45, 48, 54, 64)), snapshots=rng.randint(2, 6),
                    steps=rng.randint(2, 5))
    if kind == "les":
        return dict(kind=kind, n=_pick(rng, [2 * m for m in _smooth(10, 40)]),
                    interval=round(rng.uniform(0.15, 0.45), 3))
    return dict(kind=kind, n=_pick(rng, [2 * m for m in _smooth(10, 128)]))


# ------------------------------------------------------ inputs (from the seed)

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _stretch(t):
    return (math.tanh(1.5 * (2 * t - 1)) / math.tanh(1.5) + 1) / 2


def _flow(c):
    """Grid, viscosity, force and CFL number of a finite-volume case."""
    n = (c["nx"], c["ny"], c["nz"])
    if c.get("wall"):
        return dict(n=n, lims=((0.0, 4 * math.pi), (-1.0, 1.0), (0.0, 4 * math.pi / 3)),
                    bc=("periodic", "wall", "periodic"), stretch=_stretch,
                    visc=1 / 395 if c["implicit"] else 1 / 180, bodyforce=(1.0, 0.0, 0.0),
                    ydiffusion="implicit" if c["implicit"] else "explicit")
    return dict(n=n, visc=c.get("visc", 2e-3))


def _random_phase(n, gen, energy=0.5, kpeak=4.0):
    """[3, nz, ny, nx]: solenoidal random-phase field, E(k) ~ k^4 exp(-2 (k/kpeak)^2)."""
    nx, ny, nz = n
    v = torch.randn((3, nz, ny, nx), generator=gen, device=DEV, dtype=F64)
    k = [torch.fft.fftfreq(m, 1.0 / m, device=DEV, dtype=F64) for m in (nz, ny)]
    kx = torch.fft.rfftfreq(nx, 1.0 / nx, device=DEV, dtype=F64)
    kz, ky, kx = k[0][:, None, None], k[1][None, :, None], kx[None, None, :]
    k2 = kx ** 2 + ky ** 2 + kz ** 2
    kd = torch.where(k2 == 0, 1.0, k2)
    h = torch.fft.rfftn(v, dim=(1, 2, 3)) * (torch.sqrt(kd) * torch.exp(-k2 / kpeak ** 2))
    h[:, 0, 0, 0] = 0
    div = (kx * h[0] + ky * h[1] + kz * h[2]) / kd
    for i, kk in enumerate((kx, ky, kz)):
        h[i] -= kk * div
    v = torch.fft.irfftn(h, s=(nz, ny, nx), dim=(1, 2, 3))
    return v * math.sqrt(energy / (0.5 * float((v * v).mean()) * 3))


def _fv_start(c, gen):
    """[3, nz, ny, nx] initial values of the staggered velocity."""
    nx, ny, nz = n = (c["nx"], c["ny"], c["nz"])
    if not c.get("wall"):
        return _random_phase(n, gen)
    g = _grid(_flow(c))
    y = torch.as_tensor(g["yc"], device=DEV)
    if c["implicit"]:  # turbulent mean profile at Re_tau 395
        yp = (1 - y.abs()) * 395
        mean, amp = torch.log1p(0.41 * yp) / 0.41 + 7.8 * (
            1 - torch.exp(-yp / 11) - yp / 11 * torch.exp(-yp / 3)), 0.2
    else:
        mean, amp = 1.5 * (1 - y * y), 0.1
    v = amp * (2 * torch.rand((3, nz, ny, nx), generator=gen, device=DEV, dtype=F64) - 1)
    v[0] += mean[None, :, None]
    v[1, :, ny - 1] = 0  # the wall face
    return v


def _params(seed):
    """Closure parameters: uniform weights and biases of the usual bound."""
    rng = np.random.default_rng(seed)
    out = []
    for ci, co in zip(CHANNELS, CHANNELS[1:]):
        b = 1 / math.sqrt(27 * ci)
        out += [rng.uniform(-b, b, 27 * co * ci), rng.uniform(-b, b, co)]
    return np.concatenate(out).astype(np.float32)


def _dataset(c, seed):
    """[S, 9, n, n, n] float32: velocities and a stress that depends on them."""
    gen, n = _gen(seed), c["n"]
    out = torch.empty((c["snapshots"], 9, n, n, n), device=DEV, dtype=torch.float32)
    for i in range(c["snapshots"]):
        v = _random_phase((n, n, n), gen, energy=1.5)
        d = [torch.roll(v, -1, dims=3) - v, torch.roll(v, -1, dims=2) - v,
             torch.roll(v, -1, dims=1) - v]
        for j, (a, b) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (2, 0))):
            t = sum(e[a] * e[b] for e in d)
            out[i, 3 + j] = (t - t.mean()) / t.std()
        out[i, :3] = v
    return out


def _members(c, seed):
    rng = np.random.default_rng(seed)
    sizes = [int(v) for v in c["sizes"].split(",")]
    pick = [sizes[i % len(sizes)] for i in range(c["members"])]
    visc = np.exp(rng.uniform(math.log(1e-3), math.log(1e-2), c["members"]))
    return [dict(kind="step", nx=m, ny=m, nz=m, wall=False, implicit=False, forced=c["forced"],
                 visc=float(v)) for m, v in zip(pick, visc)]


def _spec_start(n, seed):
    """Compact solenoidal state [3, m, m, kcut + 1] of the pseudo-spectral solver."""
    k = n // 3
    v = _random_phase((n, n, n), _gen(seed))
    idx = torch.tensor([j if j <= k else j - 2 * k - 1 for j in range(2 * k + 1)], device=DEV) % n
    h = torch.fft.rfftn(v, dim=(1, 2, 3)) / n ** 3
    return h[:, idx][:, :, idx][..., :k + 1].contiguous()


# ------------------------------------------------------------ prepare and run

def _fv_state(c, gen):
    s = dns.setup(**_flow(c))
    u = dns.vectorfield(s)
    for name, v in zip("xyz", _fv_start(c, gen)):
        dns.interior(u[name])[:] = v
    dns.exchange_halo(u, s)
    p, q = dns.scalarfield(s), dns.vectorfield(s)
    delta = dns.scalarfield(s) if s.imexy else p
    if c["kind"] != "solve":
        dns.project(u, delta, s)
    return s, u, p, q, delta


def prepare(case, seed):
    k = case["kind"]
    if k in ("step", "solve"):
        c = dict(case, wall=case.get("wall", True))
        s, u, p, q, delta = _fv_state(c, _gen(seed))
        st = dict(kind=k, s=s, u=u, p=p, q=q, delta=delta, case=c, forcing=None)
        if k == "solve":
            st["stats"] = dns.channelstats(s)
            return st
        st["dt"] = None if c["cfl"] else dns.cfl_timestep(u, s, _cfl(c))
        if c["forced"]:
            st["forcing"] = dns.shellforcing(u, s)
        return st
    if k == "ensemble":
        gen, setups, states, dts, forcings = _gen(seed), [], [], [], []
        for c in _members(case, seed):
            s, u, p, q, _ = _fv_state(c, gen)
            setups.append(s)
            states.append((u, p, q, None))
            dts.append(dns.cfl_timestep(u, s, 0.5))
            forcings.append(dns.shellforcing(u, s) if case["forced"] else None)
        ens = dns.Ensemble(setups)
        for i, f in enumerate(forcings):
            if f is not None:
                ens.set_forcing(i, f)
        return dict(kind=k, ens=ens, states=states, dts=dts, steps=case["steps"],
                    forcings=forcings)
    if k in ("infer", "les"):
        n = case["n"]
        c = dict(kind="step", nx=n, ny=n, nz=n, wall=False, implicit=False, visc=5e-4)
        net = closure.Closure(batch=0, crop=0, nfield=n)
        net.set_params(_params(seed))
        net.set_scales([1.7] * 3, [0.01] * 6)
        st = dict(kind=k, net=net, tau=torch.empty((6, n, n, n), dtype=F64, device=DEV))
        if k == "infer":  # a ghosted field of any side; the network needs no setup
            g = _grid(_flow(c))
            st["u"] = dns.VectorField(
                {a: _ghost(v, g, a).contiguous() for a, v in zip("xyz", _fv_start(c, _gen(seed)))})
            return st
        s, u, p, q, _ = _fv_state(c, _gen(seed))
        return dict(st, s=s, u=u, p=p, q=q, interval=case["interval"],
                    forcing=dns.shellforcing(u, s))
    if k == "train":
        net = closure.Closure(batch=case["batch"], crop=case["crop"])
        net.set_params(_params(seed))
        net.set_dataset(_dataset(case, seed))
        return dict(kind=k, net=net, steps=case["steps"], seed=seed % 65536)
    s = spectral.spectral_setup(n=case["n"], visc=5e-4)
    uh = _spec_start(case["n"], seed)
    return dict(kind=k, s=s, uh=uh, dt=0.85 * (2 * math.pi / case["n"]) / spectral.vsummax(uh, s))


def _u(u):
    return [u["x"], u["y"], u["z"]]


def run(state):
    k = state["kind"]
    if k == "step":
        s, u, dt = state["s"], state["u"], state["dt"]
        if dt is None:
            dt = dns.cfl_timestep(u, s, _cfl(state["case"]), use_step_max=True)
        dns.step(u, state["p"], state["q"], state["delta"], s, dt)
        if state["forcing"] is not None:
            state["forcing"](u, s)
        return {"u": _u(u), "p": state["p"], "dt": dt}
    if k == "solve":
        c = state["case"]
        end = dns.solve(u=state["u"], setup=state["s"], tlims=(0.0, 100.0), cfl=_cfl(c),
                        processors={"stats": state["stats"]["sample"]}, max_steps=c["steps"])
        return {"u": _u(end.u), "p": end.p, "t": end.t, "stats": state["stats"]["acc"]}
    if k == "ensemble":
        state["ens"].run(state["states"], state["dts"], state["steps"])
        return [[*_u(u), p] for u, p, _, _ in state["states"]]
    if k == "infer":
        return state["net"].infer(state["u"], state["tau"])
    if k == "les":
        t, n = les_closure.advance(state["u"], state["p"], state["q"], state["s"], 0.0,
                                   state["interval"], 0.5, forcing=state["forcing"],
                                   closure=state["net"], tau=state["tau"])
        return {"u": _u(state["u"]), "p": state["p"], "t": t, "n": n}
    if k == "train":
        state["net"].train(state["steps"], lr=1e-3, seed=state["seed"])
        return state["net"].get_params()
    vmax = spectral.spectral_step(state["uh"], state["s"], state["dt"])
    return {"uh": state["uh"], "vmax": vmax}


# ------------------------------------------------------- work and tolerance

def _fv_flops(c):
    """Three stages: momentum, update, divergence and gradient per cell, and the transforms."""
    lines = [c["nx"], c["nz"]] + ([] if c.get("wall", True) else [c["ny"]])
    per = 200 + 2 * 2.5 * sum(math.log2(m) for m in lines) + (60 if c["implicit"] else 20)
    return 3.0 * per * c["nx"] * c["ny"] * c["nz"]


def _net_flops(voxels):
    return 2.0 * 27 * sum(a * b for a, b in zip(CHANNELS, CHANNELS[1:])) * voxels


def work(case):
    k = case["kind"]
    if k in ("step", "solve"):
        cells = case["nx"] * case["ny"] * case["nz"]
        steps = case.get("steps", 1)
        # u in and out, p out (and in where it is lagged)
        return {"bytes": 8.0 * cells * (7 + case["implicit"]), "flops": steps * _fv_flops(case)}
    if k == "ensemble":
        m = _members(case, 0)
        return {"bytes": sum(56.0 * c["nx"] ** 3 for c in m),
                "flops": case["steps"] * sum(_fv_flops(c) for c in m)}
    if k == "infer":
        return {"bytes": 72.0 * case["n"] ** 3, "flops": _net_flops(case["n"] ** 3)}
    if k == "les":
        n = case["n"]
        steps = max(1, round(case["interval"] / (0.5 * (2 * math.pi / n) / 2.2)))
        fv = _fv_flops(dict(nx=n, ny=n, nz=n, wall=False, implicit=False))
        return {"bytes": 56.0 * n ** 3, "flops": steps * (fv + 3 * _net_flops(n ** 3))}
    if k == "train":
        vox = case["batch"] * case["crop"] ** 3
        return {"bytes": case["steps"] * 36.0 * vox + 12.0 * 63174,
                "flops": case["steps"] * 3 * _net_flops(vox)}
    n, m = case["n"], 2 * (case["n"] // 3) + 1
    return {"bytes": 2 * 48.0 * m * m * (case["n"] // 3 + 1),
            "flops": 3.0 * 9 * 2.5 * n ** 3 * 3 * math.log2(n)}


def tolerance(case):
    # measured against exact(); four times the largest seen over the ranges
    return {"step": {"rel": 2e-11}, "solve": {"rel": 1e-10}, "ensemble": {"rel": 1e-10},
            "infer": {"rel": 1.3e-2, "max": 0.13}, "train": {"rel": 1.5e-2, "max": 0.3},
            "les": {"rel": 1.2e-3}, "spectral": {"rel": 1e-12}}[case["kind"]]


# --------------------------------------------------- plain torch, in 64 bits

RK_A, RK_B, RK_AL = (0.0, -5 / 9, -153 / 128), (1 / 3, 15 / 16, 8 / 15), (1 / 3, 5 / 12, 1 / 4)


def _cfl(c):
    return 0.8 if c.get("implicit") else 0.5


def _grid(f):
    """Spacings of the staggered grid: dy, dyu over the ghosted rows."""
    nx, ny, nz = f["n"]
    (x0, x1), (y0, y1), (z0, z1) = f.get("lims", ((0.0, 2 * math.pi),) * 3)
    wall = f.get("bc", "ppp")[1] == "wall"
    st = f.get("stretch", lambda t: t)
    yf = np.array([y0 + (y1 - y0) * st(j / ny) for j in range(ny + 1)])
    lo, hi = (yf[1] - yf[0], yf[ny] - yf[ny - 1]) if wall else (yf[ny] - yf[ny - 1], yf[1] - yf[0])
    e = np.concatenate([[yf[0] - lo], yf, [yf[ny] + hi]])
    dy, yc = e[1:] - e[:-1], (e[1:] + e[:-1]) / 2
    dyu = np.concatenate([yc[1:] - yc[:-1], dy[-1:]])
    return dict(nx=nx, ny=ny, nz=nz, wall=wall, dx=(x1 - x0) / nx, dz=(z1 - z0) / nz, dy=dy,
                dyu=dyu, yc=yc[1:ny + 1], visc=f["visc"], f=f.get("bodyforce", (0.0, 0.0, 0.0)),
                implicit=f.get("ydiffusion") == "implicit")


def _ghost(v, g, c):
    """[nz, ny, nx] -> ghosted [nz + 2, ny + 2, nx + 2]; c in xyzp."""
    v = torch.cat([v[..., -1:], v, v[..., :1]], -1)
    if not g["wall"]:
        v = torch.cat([v[:, -1:], v, v[:, :1]], 1)
    elif c == "y":
        zero = torch.zeros_like(v[:, :1])
        v = torch.cat([zero, v[:, :-1], zero, -v[:, -2:-1]], 1)
    else:
        sg = 1 if c == "p" else -1
        v = torch.cat([sg * v[:, :1], v, sg * v[:, -1:]], 1)
    return torch.cat([v[-1:], v, v[:1]], 0)


def _sh(a, i=0, j=0, k=0):
    """The interior of a ghosted array, shifted by whole cells."""
    n = a.shape
    return a[1 + k:n[0] - 1 + k, 1 + j:n[1] - 1 + j, 1 + i:n[2] - 1 + i]


def _rows(a, g, d=0):
    return torch.as_tensor(a[1 + d:g["ny"] + 1 + d], device=DEV)[None, :, None]


def _momentum(u, g):
    """Convection, diffusion (without the y part where it is implicit) and force."""
    ax = (0, 1, 2)
    off = lambda c, d: {"ijk"[c]: d}
    dn, dN, un, us = (_rows(g["dy"], g), _rows(g["dy"], g, 1), _rows(g["dyu"], g),
                      _rows(g["dyu"], g, -1))
    h = (g["dx"], None, g["dz"])
    out = []
    for c in ax:
        U, tot = u[c], 0.0
        for d in ax:
            V = u[d]
            for sg in (1, -1):
                # face of the control volume of u_c towards sg along d
                o = off(d, 0 if sg > 0 else -1)
                near, far = _sh(U, **off(d, 0 if sg > 0 else -1)), _sh(U, **off(d, 1 if sg > 0 else 0))
                val = (near + far) / 2
                if c == d:
                    vel = val
                else:
                    a, b = dict(o), dict(o)
                    b["ijk"[c]] = 1
                    if c == 1:
                        vel = (_sh(V, **a) * dn + _sh(V, **b) * dN) / (2 * un)
                    else:
                        vel = (_sh(V, **a) + _sh(V, **b)) / 2
                width = h[d] if d != 1 else (un if c == 1 else dn)
                tot = tot - sg * vel * val / width
                if d != 1:
                    tot = tot + sg * g["visc"] * (far - near) / (h[d] * h[d])
                elif not g["implicit"]:
                    if c == 1:
                        tot = tot + sg * g["visc"] * (far - near) / (dN if sg > 0 else dn) / un
                    else:
                        tot = tot + sg * g["visc"] * (far - near) / (un if sg > 0 else us) / dn
        tot = tot + g["f"][c]
        if c == 1 and g["wall"]:
            tot[:, -1] = 0
        out.append(tot)
    return out


def _eig(n, h, half=False):
    k = torch.arange(n // 2 + 1 if half else n, device=DEV, dtype=F64)
    s = torch.sin(math.pi * k / n)
    return -4 * s * s / (h * h)


def _poisson(r, g):
    nx, ny, nz = g["nx"], g["ny"], g["nz"]
    lam = _eig(nx, g["dx"], True)[None, None, :] + _eig(nz, g["dz"])[:, None, None]
    if not g["wall"]:
        h = torch.fft.rfftn(r, dim=(0, 1, 2))
        lam = lam + _eig(ny, g["dy"][1])[None, :, None]
        lam[0, 0, 0] = 1
        h /= lam
        h[0, 0, 0] = 0
        return torch.fft.irfftn(h, s=(nz, ny, nx), dim=(0, 1, 2))
    h, lam = torch.fft.rfftn(r, dim=(0, 2)), lam[:, 0]
    a = [0.0] + [1 / (g["dy"][j] * g["dyu"][j - 1]) for j in range(2, ny + 1)]
    b = [1 / (g["dy"][j] * g["dyu"][j]) for j in range(1, ny)] + [0.0]
    zero = lam == 0
    x, cp = [], []
    for j in range(ny):  # Thomas sweeps; the mean mode is pinned by its first row
        beta = lam - (a[j] + b[j])
        row = h[:, j]
        if j:
            beta = beta - a[j] * cp[-1]
            x.append((row - a[j] * x[-1]) / beta)
            cp.append(b[j] / beta)
        else:
            x.append(torch.where(zero, 0.0, row / beta))
            cp.append(torch.where(zero, 0.0, b[j] / beta))
    for j in range(ny - 2, -1, -1):
        x[j] = x[j] - cp[j] * x[j + 1]
    return torch.fft.irfftn(torch.stack(x, 1), s=(nz, nx), dim=(0, 2))


def _grad(p, g):
    P = _ghost(p, g, "p")
    out = [(_sh(P, i=1) - p) / g["dx"], (_sh(P, j=1) - p) / _rows(g["dyu"], g),
           (_sh(P, k=1) - p) / g["dz"]]
    if g["wall"]:
        out[1][:, -1] = 0
    return out


def _project(u, g):
    G = [_ghost(v, g, c) for v, c in zip(u, "xyz")]
    r = ((u[0] - _sh(G[0], i=-1)) / g["dx"] + (u[1] - _sh(G[1], j=-1)) / _rows(g["dy"], g)
         + (u[2] - _sh(G[2], k=-1)) / g["dz"])
    p = _poisson(r, g)
    return [v - d for v, d in zip(u, _grad(p, g))], p


def _ydiff(g, c):
    """Dense wall-normal second difference of component c on its active rows."""
    ny, dy, dyu = g["ny"], g["dy"], g["dyu"]
    m = ny - 1 if c == 1 else ny
    D = np.zeros((m, m))
    for j in range(1, m + 1):
        if c == 1:
            a, b = 1 / (dyu[j] * dy[j]), 1 / (dyu[j] * dy[j + 1])
            d = -(a + b)
        else:
            a, b = 1 / (dy[j] * dyu[j - 1]), 1 / (dy[j] * dyu[j])
            d = -(a + b) - (a if j == 1 else 0) - (b if j == ny else 0)
        D[j - 1, j - 1] = d
        if j > 1:
            D[j - 1, j - 2] = a
        if j < m:
            D[j - 1, j] = b
    return torch.as_tensor(D, device=DEV)


def _rk_step(u, p, g, dt, stress=None):
    q = [0.0] * 3
    for A, B, al in zip(RK_A, RK_B, RK_AL):
        F = _momentum([_ghost(v, g, c) for v, c in zip(u, "xyz")], g)
        if stress is not None:
            F = [a + b for a, b in zip(F, stress(u))]
        q = [A * a + dt * b for a, b in zip(q, F)]
        v = [a + B * b for a, b in zip(u, q)]
        if g["implicit"]:
            th = al * dt * g["visc"] / 2
            v = [a - al * dt * b for a, b in zip(v, _grad(p, g))]
            for c in range(3):
                D = _ydiff(g, c)
                m = D.shape[0]
                eye = torch.eye(m, device=DEV, dtype=F64)
                rhs = v[c][:, :m] + th * torch.matmul(D, u[c][:, :m])
                v[c] = v[c].clone()
                v[c][:, :m] = torch.matmul(torch.linalg.inv(eye - th * D), rhs)
            u, d = _project(v, g)
            p = p + d / (al * dt)
        else:
            u, p = _project(v, g)
    return u, p


def _cfl_dt(u, g, cfl):
    eps = 2.220446049250313e-16
    m = [float(v.abs().max()) for v in u]
    dym = float(g["dy"][1:g["ny"] + 1].min())
    conv = min(g["dx"] / (m[0] + eps), dym / (m[1] + eps), g["dz"] / (m[2] + eps))
    inv = 1 / g["dx"] ** 2 + 1 / g["dz"] ** 2 + (0 if g["implicit"] else 1 / dym ** 2)
    return min(cfl * conv, cfl / (2 * g["visc"] * inv + eps))


def _shells(u):
    """Weights, floor shells and spectra of the three components."""
    nz, ny, nx = u[0].shape
    k = [torch.fft.fftfreq(m, 1.0 / m, device=DEV, dtype=F64).round() for m in (nz, ny)]
    kx = torch.arange(nx // 2 + 1, device=DEV, dtype=F64)
    k2 = kx[None, None, :] ** 2 + k[1][None, :, None] ** 2 + k[0][:, None, None] ** 2
    w = torch.where((kx > 0) & (2 * kx < nx), 2.0, 1.0)[None, None, :]
    return w, torch.floor(torch.sqrt(k2) + 1e-9), [torch.fft.rfftn(v) / v.numel() for v in u]


def _shell_energy(u, sh):
    w, ks, H = _shells(u)
    return sum(float((w * (ks == sh) * h.abs() ** 2).sum()) for h in H) / 2


def _clamp(u, eref):
    w, ks, H = _shells(u)
    f = torch.ones_like(ks)
    for sh, e in eref.items():
        now = sum(float((w * (ks == sh) * h.abs() ** 2).sum()) for h in H) / 2
        f = torch.where(ks == sh, math.sqrt(e / now), f)
    return [torch.fft.irfftn(h * f * v.numel(), s=v.shape) for h, v in zip(H, u)]


def _conv(x, W, b):
    """Valid 3x3x3 convolution of [B, ci, z, y, x] with W[27, co, ci], by taps."""
    d = [m - 2 for m in x.shape[2:]]
    out = b[None, :, None, None, None]
    for t in range(27):
        z, y, i = t // 9, t // 3 % 3, t % 3
        out = out + torch.einsum("oc,bczyx->bozyx", W[t],
                                 x[:, :, z:z + d[0], y:y + d[1], i:i + d[2]])
    return out


def _unflatten(p):
    out, o = [], 0
    for ci, co in zip(CHANNELS, CHANNELS[1:]):
        out.append((p[o:o + 27 * co * ci].reshape(27, co, ci),
                    p[o + 27 * co * ci:o + 27 * co * ci + co]))
        o += 27 * co * ci + co
    return out


def _network(x, p):
    for i, (W, b) in enumerate(_unflatten(p)):
        x = _conv(x, W, b)
        if i < 3:
            x = torch.nn.functional.gelu(x, approximate="tanh")
    return x


def _tau(u, p, scale_in=1.7, scale_out=0.01):
    """Stress at the cell centres from the staggered periodic velocity."""
    v = torch.stack([(torch.roll(a, 1, 2 - c) + a) / 2 for c, a in enumerate(u)])
    for d in (1, 2, 3):
        v = torch.cat([v.narrow(d, v.shape[d] - 4, 4), v, v.narrow(d, 0, 4)], d)
    return scale_out * _network(scale_in * v[None], p)[0]


def _stress(tau, g):
    """-div(tau) on the faces: normal stresses across them, shear from the edges."""
    xx, yy, zz, xy, yz, zx = tau
    h = (g["dx"], float(g["dy"][1]), g["dz"])
    mid = lambda a, c: (a + torch.roll(a, -1, 2 - c)) / 2
    up = lambda a, c: (torch.roll(a, -1, 2 - c) - a) / h[c]
    cen = lambda a, c: (torch.roll(a, -1, 2 - c) - torch.roll(a, 1, 2 - c)) / (2 * h[c])
    return [-(up(xx, 0) + cen(mid(xy, 0), 1) + cen(mid(zx, 0), 2)),
            -(cen(mid(xy, 1), 0) + up(yy, 1) + cen(mid(yz, 1), 2)),
            -(cen(mid(zx, 2), 0) + cen(mid(yz, 2), 1) + up(zz, 2))]


def _mix(x):
    m = (1 << 64) - 1
    z = (x + 0x9E3779B97F4A7C15) & m
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return z ^ (z >> 31)


def _crops(data, c, seed, step):
    """The batch of a training step: crops with a halo of 4, and their targets."""
    n, xs, ts = c["n"], [], []
    for b in range(c["batch"]):
        h = _mix(seed ^ _mix(4 * (step * 64 + b)))
        snap = data[h % c["snapshots"]].double()
        o = [_mix((h + i) & ((1 << 64) - 1)) % n for i in (3, 2, 1)]
        at = lambda pad: [(torch.arange(-pad, c["crop"] + pad, device=DEV) + v) % n for v in o]
        z, y, x = at(4)
        xs.append(snap[:3][:, z][:, :, y][..., x])
        z, y, x = at(0)
        ts.append(snap[3:][:, z][:, :, y][..., x])
    return torch.stack(xs), torch.stack(ts)


def _train(c, seed):
    data, s0 = _dataset(c, seed), seed % 65536
    p = torch.as_tensor(_params(seed), device=DEV, dtype=F64)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    for step in range(c["steps"]):
        x, t = _crops(data, c, s0, step)
        p.requires_grad_(True)
        grad = torch.zeros_like(p)
        for b in range(c["batch"]):  # one crop at a time: 64-bit activations are large
            loss = ((_network(x[b:b + 1], p) - t[b:b + 1]) ** 2).sum() / t.numel()
            grad += torch.autograd.grad(loss, p)[0]
        p = p.detach()
        m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
        p = p - 1e-3 * (m / (1 - 0.9 ** (step + 1))) / (
            torch.sqrt(v / (1 - 0.999 ** (step + 1))) + 1e-8)
    return p.cpu().numpy()


def _spectral(n, seed):
    k = n // 3
    m = 2 * k + 1
    cf = torch.tensor([j if j <= k else j - m for j in range(m)], device=DEV)
    idx = cf % n
    K = (torch.arange(k + 1, device=DEV, dtype=F64)[None, None, :], cf.double()[None, :, None],
         cf.double()[:, None, None])
    kk = K[0] ** 2 + K[1] ** 2 + K[2] ** 2

    def phys(h):
        full = torch.zeros((n, n, n // 2 + 1), device=DEV, dtype=torch.complex128)
        full[idx[:, None], idx[None, :], :k + 1] = h
        return torch.fft.irfftn(full, s=(n, n, n)) * n ** 3

    def spec(r):
        return torch.fft.rfftn(r)[idx][:, idx][..., :k + 1] / n ** 3

    u = _spec_start(n, seed)
    vel = [phys(h) for h in u]
    dt = 0.85 * (2 * math.pi / n) / float(sum(v.abs() for v in vel).max())
    w, vmax = u.clone(), None
    for a, b, dc in zip((8 / 15, 5 / 12, 3 / 4), (1 / 4, 0.0, 0.0), (8 / 15, 2 / 15, 1 / 3)):
        vel = [phys(h) for h in u]
        if vmax is None:
            vmax = float(sum(v.abs() for v in vel).max())
        S = {(i, j): spec(vel[i] * vel[j]) for i in range(3) for j in range(i, 3)}
        rhs = torch.stack([-1j * sum(K[j] * S[min(i, j), max(i, j)] for j in range(3))
                           for i in range(3)])
        phi = torch.exp(-5e-4 * dc * dt * kk)
        u, w = phi * (w + a * dt * rhs), phi * (w + b * dt * rhs)
        div = (K[0] * u[0] + K[1] * u[1] + K[2] * u[2]) / torch.where(kk == 0, 1.0, kk)
        u = torch.stack([u[i] - K[i] * div for i in range(3)])
    return {"uh": u, "vmax": vmax}


def _channel_sums(u, g):
    G = [_ghost(v, g, c) for v, c in zip(u, "xyz")]
    f = slice(0, g["ny"] - 1)
    uf, vf = (u[0] + _sh(G[0], j=1)) / 2, (u[1] + _sh(G[1], i=1)) / 2
    full = [u[0], u[2], u[0] ** 2, u[2] ** 2]
    face = [u[1], u[1] ** 2, uf, uf * vf]
    return torch.cat([v.sum((0, 2)) for v in full] + [v.sum((0, 2))[f] for v in face])


def _fv_out(u, p, g, **more):
    return {"u": [_ghost(v, g, c) for v, c in zip(u, "xyz")], "p": _ghost(p, g, "p"), **more}


def _fv_exact_start(c, gen):
    g = _grid(_flow(c))
    u = list(_fv_start(c, gen))
    u, _ = _project(u, g)
    return g, u, torch.zeros_like(u[0])


def exact(case, seed):
    k = case["kind"]
    if k in ("step", "solve"):
        c = dict(case, wall=case.get("wall", True))
        g, u, p = _fv_exact_start(c, _gen(seed))
        if k == "step":
            eref = {s: _shell_energy(u, s) for s in (1, 2)} if c["forced"] else None
            dt = _cfl_dt(u, g, _cfl(c))
            u, p = _rk_step(u, p, g, dt)
            if eref:
                u = _clamp(u, eref)
            return _fv_out(u, p, g, dt=dt)
        t, acc = 0.0, _channel_sums(u, g)
        for _ in range(c["steps"]):
            dt = _cfl_dt(u, g, _cfl(c))
            u, p = _rk_step(u, p, g, dt)
            t += dt
            acc = acc + _channel_sums(u, g)
        return _fv_out(u, p, g, t=t, stats=acc)
    if k == "ensemble":
        gen, out = _gen(seed), []
        for c in _members(case, seed):
            g, u, p = _fv_exact_start(c, gen)
            eref = {s: _shell_energy(u, s) for s in (1, 2)}
            dt = _cfl_dt(u, g, 0.5)
            for _ in range(case["steps"]):
                u, p = _rk_step(u, p, g, dt)
                if case["forced"]:
                    u = _clamp(u, eref)
            o = _fv_out(u, p, g)
            out.append([*o["u"], o["p"]])
        return out
    if k in ("infer", "les"):
        n = case["n"]
        c = dict(nx=n, ny=n, nz=n, wall=False, implicit=False, visc=5e-4)
        par = torch.as_tensor(_params(seed), device=DEV, dtype=F64)
        if k == "infer":
            return _tau(list(_fv_start(c, _gen(seed))), par)
        g, u, p = _fv_exact_start(c, _gen(seed))
        eref = {s: _shell_energy(u, s) for s in (1, 2)}
        t, steps, end = 0.0, 0, case["interval"]
        while t < end - 1e-10 * (abs(end) + 1):
            dt = min(_cfl_dt(u, g, 0.5), end - t)
            u, p = _rk_step(u, p, g, dt, stress=lambda v: _stress(_tau(v, par), g))
            u = _clamp(u, eref)
            t, steps = t + dt, steps + 1
        return _fv_out(u, p, g, t=end, n=steps)
    if k == "train":
        return _train(case, seed)
    return _spectral(case["n"], seed)
