"""The work that users of this framework have it do, as cases to be timed.

A case is one pass through the public entry points on device-resident data:

  run       a window of a simulation: upload a state, advance it by RK3 steps,
            read its scalars (and profiles where asked), download it.  FP64
            with FMA (`fast`), FP64 in the reference's rounding (`exact`) and
            the FP32 form, with or without the learned closure
  ensemble  a window of a batched ensemble of FP32 members of uneven sizes
  train     one training step of the closure network: forward, loss,
            backward, Adam
  pairs     one training snapshot: a fine state box-filtered to coarse
            features and subgrid targets

listed() names the cases, draw() gives more of the same ranges, prepare()
makes what a program holds before the pass, run() is the pass, work() its
compulsory bytes and operations, and exact() its result in 64 bits, as plain
torch gives it.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "rast-3dmhd_b200"))

import closure  # noqa: E402
import mhd3d  # noqa: E402

MODES = {"fast": mhd3d.MODE_FAST, "exact": mhd3d.MODE_EXACT, "fp32": mhd3d.MODE_FP32}
LARGEST = 512 * 512 * 256 * 8   # cell-steps of the largest listed window


def _window(name, mode, nx, ny, nz, steps, per_call, **kw):
    c = {"name": name, "kind": "run", "mode": mode, "nx": nx, "ny": ny, "nz": nz, "mag": 1, "rot": 1, "steps": steps,
         "per_call": per_call, "profiles": 0, "closure": 0, "ra": 1e6, "ta": 1e6, "contrast": 10.0, "stretch": 1.5}
    c.update(kw)
    return c


def listed():
    return [
        # the Fortran driver's loop on its smallest case: one CALL STEP a call,
        # DT read back after each
        _window("driver_64", "fast", 64, 64, 48, 50, 1, ra=1e5, ta=1e4),
        # the middle size with its horizontal profiles sampled once a window
        _window("profiled_256", "fast", 256, 256, 128, 20, 20, profiles=1),
        # the fine run of the closure case: the headline workload
        _window("fine_512", "fast", 512, 512, 256, 8, 8),
        # a hydrodynamic run without rotation, ragged in every direction
        _window("hydro_ragged", "fast", 203, 150, 75, 20, 5, mag=0, rot=0, ra=1e5),
        # a run that has to reproduce the reference bit for bit, stepped by its driver
        _window("reference_96", "exact", 96, 96, 64, 10, 1, ra=1e5, ta=1e4),
        # the coarse FP32 run of the closure case
        _window("coarse_fp32", "fp32", 128, 128, 64, 20, 20),
        # the same with the closure network evaluated on every step
        _window("coarse_closure", "fp32", 128, 128, 64, 20, 20, closure=1),
        # a large FP32 run at the large case's physics
        _window("large_fp32", "fp32", 512, 512, 256, 8, 8, ra=1e7, ta=1e7, contrast=30.0, stretch=2.0),
        # seeded members of the ensemble case's three grids
        {"name": "ensemble", "kind": "ensemble", "members": 12, "sizes": "64x64x48,96x96x64,128x128x96", "steps": 30},
        # a training step on one pair of the full-size coarse grid
        {"name": "train_128", "kind": "train", "nx": 128, "ny": 128, "nz": 64},
        # and on a coarse grid of the ensemble's members (24-wide rows)
        {"name": "train_24", "kind": "train", "nx": 24, "ny": 24, "nz": 16},
        # a pair from the fine run of the recorded closure case
        {"name": "pairs_384", "kind": "pairs", "nx": 384, "ny": 384, "nz": 192},
    ]


def _members(c):
    """Grid sizes of an ensemble's members."""
    sizes = [tuple(int(v) for v in s.split("x")) for s in c["sizes"].split(",")]
    return [sizes[i % len(sizes)] for i in range(c["members"])]


def _size(rng, lo, hi, odd=True):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n if odd and rng.random() < 0.4 else max(lo, n // 8 * 8)


def draw(rng):
    kind = rng.choice(["run"] * 7 + ["ensemble", "train", "pairs"])
    if kind == "ensemble":
        sizes = ["%dx%dx%d" % (_size(rng, 32, 128), _size(rng, 32, 128), _size(rng, 24, 96)) for _ in range(3)]
        c = {"kind": "ensemble", "members": rng.randint(4, 16), "sizes": ",".join(sizes), "steps": 1}
        c["steps"] = max(1, min(rng.randint(10, 30), LARGEST // sum(math.prod(m) for m in _members(c))))
        return c
    if kind == "train":
        return {"kind": "train", "nx": _size(rng, 16, 192), "ny": _size(rng, 16, 128), "nz": _size(rng, 8, 64)}
    if kind == "pairs":
        return {"kind": "pairs", "nx": 4 * _size(rng, 16, 96), "ny": 4 * _size(rng, 16, 96), "nz": 4 * _size(rng, 8, 48)}
    mode = rng.choice(["fast", "fast", "fp32", "fp32", "exact"])
    nx, ny, nz = _size(rng, 32, 512), _size(rng, 32, 512), _size(rng, 24, 256)
    clo = 1 if mode == "fp32" and rng.random() < 0.4 else 0
    mag = 1 if clo or rng.random() < 0.8 else 0
    steps = max(1, min(rng.randint(4, 40), LARGEST // (nx * ny * nz) // (4 if clo or mode == "exact" else 2)))
    c = _window("", mode, nx, ny, nz, steps, rng.choice([1, steps]), mag=mag, rot=rng.randint(0, 1), closure=clo,
                profiles=rng.randint(0, 1), ra=10.0 ** rng.uniform(4, 7), ta=10.0 ** rng.uniform(3, 7),
                contrast=rng.uniform(3, 30), stretch=rng.uniform(1.2, 2.0))
    del c["name"]
    return c


# ---- inputs -----------------------------------------------------------------
def _setup(nx, ny, nz, mag=1, rot=1, ra=1e6, ta=1e6, contrast=10.0, stretch=1.5):
    """Run set-up without a host state, and the layer's profiles over z."""
    def cfg_of(a, b):
        cfg = mhd3d.convection_config(a, b, nz, ra=ra, ta=ta, contrast=contrast, stretch=stretch)
        cfg.lmag, cfg.lrot = mag, rot
        return cfg
    thin = mhd3d.make_setup(cfg_of(4, 4))
    cx, cy = mhd3d.make_setup(cfg_of(nx, 2)), mhd3d.make_setup(cfg_of(2, ny))
    p = mhd3d.Params.from_buffer_copy(cx.params)
    p.npy, p.hy, p.h2y = ny, cy.params.hy, cy.params.h2y
    grid = dict(cx.grid)
    for n in ("wyy", "dyydy", "d2yydy2", "ddy"):
        grid[n] = cy.grid[n]
    prof = {f: thin.state[f][1, 1, :].copy() for f in ("tt", "ro")}
    prof["b"] = float(np.sqrt((thin.state["by"][1, 1, 1:-1] ** 2).mean())) if mag else 0.0
    cfg = cfg_of(nx, ny)
    return mhd3d.Setup(cfg, p, grid, {}), prof


def _smooth(gen, nz, ny, nx, modes=4):
    """A smooth random field, periodic in x and y, of order one."""
    dev = "cuda"
    z, y, x = (torch.arange(n, dtype=torch.float64, device=dev) / max(n - k, 1) for n, k in ((nz, 1), (ny, 0), (nx, 0)))
    out = torch.zeros(nz, ny, nx, dtype=torch.float64, device=dev)
    r = torch.rand(modes, 6, generator=gen).tolist()
    for a, b, c, p, q, s in r:
        fx = torch.sin(2 * math.pi * (1 + int(3 * a)) * x + 6.28 * p)
        fy = torch.cos(2 * math.pi * (1 + int(3 * b)) * y + 6.28 * q)
        fz = torch.cos(math.pi * (1 + int(4 * c)) * z + 1.5 * s)
        out += (0.5 + 0.5 * s) * fz[:, None, None] * fy[None, :, None] * fx[None, None, :]
    return out / math.sqrt(modes)


def _state(su, prof, seed):
    """A convecting state [nf, NZ, NY, NX] (Fortran (NX,NY,NZ) arrays): the
    layer with smooth perturbations of a few percent, flow at a few percent
    of the sound speed, and a bent magnetic field."""
    gen = torch.Generator().manual_seed(int(seed))
    noise = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    nx, ny, nz = su.params.npx, su.params.npy, su.params.npz
    nf = 8 if su.params.lmag else 5
    u = torch.empty(nf, nz + 2, ny + 2, nx + 2, dtype=torch.float64, device="cuda")
    wall = torch.sin(math.pi * torch.linspace(0, 1, nz, dtype=torch.float64, device="cuda"))[:, None, None]
    t0, r0 = (torch.from_numpy(prof[f][1:-1]).cuda()[:, None, None] for f in ("tt", "ro"))

    def put(f, v):
        u[f, 1:-1, 1:-1, 1:-1] = v
    ro = r0 * (1 + 0.02 * wall * _smooth(gen, nz, ny, nx))
    put(4, ro)
    put(3, t0 * (1 + 0.02 * wall * _smooth(gen, nz, ny, nx)
                 + 1e-4 * wall * (torch.rand(nz, ny, nx, generator=noise, dtype=torch.float64, device="cuda") - 0.5)))
    for f in range(3):
        put(f, 0.05 * ro * (wall if f == 2 else 1.0) * _smooth(gen, nz, ny, nx))
    for f in range(5, nf):
        put(f, prof["b"] * ((1.0 if f == 6 else 0.0) + 0.3 * (wall if f == 7 else 1.0) * _smooth(gen, nz, ny, nx)))
    u[:, 0], u[:, -1] = u[:, 1], u[:, -2]
    u[:, :, 0], u[:, :, -1] = u[:, :, -2], u[:, :, 1]
    u[:, :, :, 0], u[:, :, :, -1] = u[:, :, :, -2], u[:, :, :, 1]
    return u


def _net(seed):
    """A small closure network as training leaves it: scaled inputs, subgrid terms of a percent."""
    net = closure.ClosureNet(seed=int(seed) % 1000)
    net.in_scale.copy_(torch.tensor([20.0, 20.0, 20.0, 2.0, 2.0, 100.0, 100.0, 100.0]))
    net.out_scale.copy_(torch.tensor([1e-3] * 6 + [1e-3] * 3 + [1e-5] * 3))
    return net


def _physics(i):
    """Ra, Ta and density contrast of member i, spread over the ensemble case's ranges."""
    g = (i * 0.6180339887) % 1.0, (i * 0.7548776662 + 0.3) % 1.0, (i * 0.5698402909 + 0.6) % 1.0
    return {"ra": 10.0 ** (4 + 2 * g[0]), "ta": 10.0 ** (3 + 3 * g[1]), "contrast": 3.0 + 27.0 * g[2]}


def _run_setup(c):
    return _setup(c["nx"], c["ny"], c["nz"], c["mag"], c["rot"], c["ra"], c["ta"], c["contrast"], c["stretch"])


def _member_setups(c):
    return [_setup(*m, **_physics(i)) for i, m in enumerate(_members(c))]


def _train_data(c, seed):
    """Features (8 scaled channels of 16, BF16) and normalised targets of one coarse snapshot."""
    gen = torch.Generator().manual_seed(int(seed))
    noise = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    nz, ny, nx = c["nz"], c["ny"], c["nx"]
    feat = torch.zeros(nz, ny, nx, 16, dtype=torch.bfloat16, device="cuda")
    base = [_smooth(gen, nz, ny, nx) for _ in range(8)]
    for i, b in enumerate(base):
        feat[..., i] = b.to(torch.bfloat16)
    tgt = torch.empty(nz, ny, nx, 12, dtype=torch.float32, device="cuda")
    for i in range(12):
        tgt[..., i] = (base[i % 8] * base[(3 * i + 1) % 8]).float()
    tgt += 0.1 * torch.randn(nz, ny, nx, 12, generator=noise, device="cuda")
    return feat, tgt


def _upload(sim, u):
    ptrs = [closure._p(u[f]) for f in range(u.shape[0])]
    st = sim.lib.mhd3d_upload(sim.h, *(ptrs + [None] * (8 - len(ptrs))))
    if st:
        raise mhd3d.Mhd3dError(st, "mhd3d_upload")


def _download(sim, u):
    ptrs = [closure._p(u[f]) for f in range(u.shape[0])]
    st = sim.lib.mhd3d_download(sim.h, *(ptrs + [None] * (8 - len(ptrs))))
    if st:
        raise mhd3d.Mhd3dError(st, "mhd3d_download")


def prepare(case, seed):
    c = case
    if c["kind"] == "run":
        su, prof = _run_setup(c)
        s = {"case": c, "sim": mhd3d.GpuSim(su, mode=MODES[c["mode"]]), "u": _state(su, prof, seed)}
        s["out"] = torch.empty_like(s["u"])
        if c["closure"]:
            s["net"] = _net(seed)
            s["net"].attach(s["sim"], trip=1.0)
    elif c["kind"] == "ensemble":
        sus = _member_setups(c)
        ens = mhd3d.Ensemble([su for su, _ in sus])
        s = {"case": c, "ens": ens, "u": [_state(su, prof, seed + 7 * i) for i, (su, prof) in enumerate(sus)]}
        s["out"] = [torch.empty_like(u) for u in s["u"]]
        torch.cuda.synchronize()
        for m, u in zip(ens.members, s["u"]):
            _upload(m, u)
        ens.tune(2)   # as the ensemble workload does before its steps
    elif c["kind"] == "train":
        s = {"case": c, "net": _net(seed)}
        s["feat"], s["tgt"] = _train_data(c, seed)
    else:
        su, prof = _setup(c["nx"], c["ny"], c["nz"])
        coarse, _ = _setup(c["nx"] // 4, c["ny"] // 4, c["nz"] // 4)
        s = {"case": c, "sim": mhd3d.GpuSim(su, mode=mhd3d.MODE_FAST), "pairs": closure.PairCollector(su, coarse),
             "in_scale": _net(0).in_scale}
        u = _state(su, prof, seed)
        torch.cuda.synchronize()
        _upload(s["sim"], u)
    torch.cuda.synchronize()   # the library works on streams of its own
    return s


def run(state):
    s, c = state, state["case"]
    if c["kind"] == "run":
        sim = s["sim"]
        _upload(sim, s["u"])
        for _ in range(c["steps"] // c["per_call"]):
            r = sim.step(c["per_call"])
        out = {"dt": r["dt"], "umach": r["umach"]}
        if c["profiles"]:
            out["profiles"] = sim.profiles()
        _download(sim, s["out"])
        # an FP32 run's snapshots are kept in FP32
        keep = s["out"].float() if c["mode"] == "fp32" else s["out"]
        out.update({f: keep[i] for i, f in enumerate(mhd3d.FIELDS[:keep.shape[0]])})
        return out
    if c["kind"] == "ensemble":
        for m, u in zip(s["ens"].members, s["u"]):
            _upload(m, u)
        r = s["ens"].step(c["steps"])
        for m, o in zip(s["ens"].members, s["out"]):
            _download(m, o)
        return {"dt": r["dt"].astype(np.float32), "state": [o.float() for o in s["out"]]}
    if c["kind"] == "train":
        net, shape = s["net"], (c["nz"], c["ny"], c["nx"])
        stream = torch.cuda.current_stream().cuda_stream
        net.zero_grad()
        acts, pred = net.forward(s["feat"], shape, stream)
        loss, dy = net.loss_and_grad(pred, s["tgt"], stream)
        net.backward(acts, dy, shape, stream)
        net.adam_step(1e-3, stream)
        return {"loss": loss, "pred": pred, "dw": net.dw, "db": net.db, "w": net.w, "b": net.b}
    feat, tgt = s["pairs"].snapshot(s["sim"], s["in_scale"])
    return {"feat": feat, "targets": tgt, "coarse": s["pairs"].cstate}


# ---- compulsory work ----------------------------------------------------------
def work(case):
    """Bytes: the state in and out of a window (FP64), and per step the
    state read and written once in the precision it is held in.  FLOPs: the
    right-hand side and update of three stages (530 a cell and stage with a
    magnetic field), the convolutions, the filter's sums."""
    c = case
    if c["kind"] == "run":
        cells = c["nx"] * c["ny"] * c["nz"]
        nf = 8 if c["mag"] else 5
        w = 4 if c["mode"] == "fp32" else 8
        fl = 3 * (530 if c["mag"] else 330) * cells * c["steps"]
        by = cells * nf * (16 + 2 * w * c["steps"])
        if c["closure"]:
            fl += cells * c["steps"] * 2 * 27 * (8 * 32 + 32 * 32 + 32 * 12)
        return {"bytes": by, "flops": fl}
    if c["kind"] == "ensemble":
        cells = sum(math.prod(m) for m in _members(c))
        return {"bytes": cells * 8 * (16 + 8 * c["steps"]), "flops": 3 * 530 * cells * c["steps"]}
    v = c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "train":
        # forward and weight gradient of every layer, input gradient of two
        fl = 2 * 27 * v * (2 * (8 * 32 + 32 * 32 + 32 * 12) + 32 * 32 + 32 * 12)
        return {"bytes": v * (16 * 2 + 12 * 4 + 16 * 4), "flops": fl}
    return {"bytes": v * 64 + v // 64 * (32 + 48 + 64), "flops": 60 * v}


# ---- the same in 64 bits --------------------------------------------------------
class _Model:
    """The equations of one run in plain torch FP64: right-hand side, RK3
    update, walls and time step, on arrays [NZ, NPY, NPX] with the z ghost planes."""

    def __init__(self, su):
        self.p = p = su.params
        t = {n: torch.from_numpy(np.ascontiguousarray(a)).cuda() for n, a in su.grid.items()}
        x, y, z = (lambda a: a[1:-1][None, None, :]), (lambda a: a[1:-1][None, :, None]), (lambda a: a[1:-1][:, None, None])
        self.ax, self.bx, self.cx = p.hx * x(t["dxxdx"]), p.hx * x(t["d2xxdx2"]), p.h2x * x(t["dxxdx"]) ** 2
        self.ay, self.by, self.cy = p.hy * y(t["dyydy"]), p.hy * y(t["d2yydy2"]), p.h2y * y(t["dyydy"]) ** 2
        self.az, self.bz, self.cz = p.hz * z(t["dzzdz"]), p.hz * z(t["d2zzdz2"]), p.h2z * z(t["dzzdz"]) ** 2
        self.rka, self.dka = z(t["rkapa"]), z(t["dkapa"])
        self.dd = torch.minimum(torch.minimum(x(t["ddx"]), y(t["ddy"])), z(t["ddz"]))
        dz = float(np.float32(1.0) / np.float32(p.npz - 1)) / float(t["dzzdz"][-2])   # a REAL(4) quotient there
        self.bot_flux = p.c23 * dz * p.theta / float(t["rkapa"][-2])

    def dx(self, f): return (torch.roll(f, -1, 2) - torch.roll(f, 1, 2)) * self.ax
    def dy(self, f): return (torch.roll(f, -1, 1) - torch.roll(f, 1, 1)) * self.ay
    def dz(self, f): return (f[2:] - f[:-2]) * self.az

    def d2x(self, f):
        a, b = torch.roll(f, -1, 2), torch.roll(f, 1, 2)
        return (a - b) * self.bx + (a + b - 2 * f) * self.cx

    def d2y(self, f):
        a, b = torch.roll(f, -1, 1), torch.roll(f, 1, 1)
        return (a - b) * self.by + (a + b - 2 * f) * self.cy

    def d2z(self, f): return (f[2:] - f[:-2]) * self.bz + (f[2:] + f[:-2] - 2 * f[1:-1]) * self.cz

    def d2z_wall(self, f):
        """d2z with one-sided differences on the walls (planes 1 and -2)."""
        d = self.d2z(f)
        d[0] = (-3 * f[1] + 4 * f[2] - f[3]) * self.bz[0] + (2 * f[1] - 5 * f[2] + 4 * f[3] - f[4]) * self.cz[0]
        d[-1] = (3 * f[-2] - 4 * f[-3] + f[-4]) * self.bz[-1] + (2 * f[-2] - 5 * f[-3] + 4 * f[-4] - f[-5]) * self.cz[-1]
        return d

    def dz_wall(self, f):
        """dz of a quantity that vanishes on the walls, one-sided there."""
        d = self.dz(f)
        d[0] = (4 * f[2] - f[3]) * self.az[0]
        d[-1] = (f[-4] - 4 * f[-3]) * self.az[-1]
        return d

    def rhs(self, s):
        p = self.p
        ru, rv, rw, tt, ro = s[:5]
        ri = 1.0 / ro
        U, V, W = ru * ri, rv * ri, rw * ri
        P = ro * tt
        c = slice(1, -1)
        u, v, w, T, r = U[c], V[c], W[c], tt[c], ri[c]
        fr = -(self.dx(ru[c]) + self.dy(rv[c])) - self.dz_wall(rw)
        t13, ore = p.c13 * p.ore, p.ore

        def adv(m): return self.dx(m[c] * u) + self.dy(m[c] * v) + self.dz(m * W)
        fu = -self.dx(P[c]) - adv(ru) + ore * (p.c43 * self.d2x(u) + self.d2y(u) + self.d2z(U))
        fv = -self.dy(P[c]) - adv(rv) + ore * (self.d2x(v) + p.c43 * self.d2y(v) + self.d2z(V))
        fw = p.grav * ro[c] - self.dz(P) - adv(rw) + ore * (self.d2x(w) + self.d2y(w) + p.c43 * self.d2z(W))
        ux, vx, wx = self.dx(u), self.dx(v), self.dx(w)
        uy, vy, wy = self.dy(u), self.dy(v), self.dy(w)
        uz, vz, wz = self.dz(U), self.dz(V), self.dz(W)
        fu += t13 * (self.dx(vy) + self.dx(wz))
        fv += t13 * (self.dy(ux) + self.dy(wz))
        fw += t13 * (self.dx(uz) + self.dy(vz))
        tz = self.dz(tt)
        ft = -(u * self.dx(T) + v * self.dy(T) + w * tz)
        ft += r * (p.ocv / p.repr) * (self.rka * (self.d2x(T) + self.d2y(T) + self.d2z(tt)) + self.dka * tz)
        heat = p.ocv * ore * (p.c43 * ux * ux + vx * vx + wx * wx + uy * uy + 2 * uy * vx + uz * uz + vz * vz + wy * wy
                              + 2 * vz * wy + 2 * uz * wx)
        heat += p.c43 * p.ocv * ore * (vy * vy + wz * wz - ux * wz - ux * vy - vy * wz)
        ft -= p.ocv * T * (ux + vy + wz)
        if p.lrot:
            fu += p.omz * rv[c]
            fv += p.omx * rw[c] - p.omz * ru[c]
            fw -= p.omx * rv[c]
        out = [fu, fv, fw, ft, fr]
        if p.lmag:
            BX, BY, BZ = s[5:]
            bx, by, bz = BX[c], BY[c], BZ[c]
            bxy, bxz, byx, byz = self.dy(bx), self.dz(BX), self.dx(by), self.dz(BY)
            bzx, bzy = self.dx(bz), self.dy(bz)
            wzm = self.dz_wall(W)
            out.append(by * uy - bx * vy + bz * uz - bx * wzm - (u * self.dx(bx) + v * bxy + w * bxz)
                       + p.orm * (self.d2x(bx) + self.d2y(bx) + self.d2z_wall(BX)))
            out.append(bx * vx - by * ux + bz * vz - by * wzm - (u * byx + v * self.dy(by) + w * byz)
                       + p.orm * (self.d2x(by) + self.d2y(by) + self.d2z_wall(BY)))
            out.append(bx * wx - bz * ux + by * wy - bz * vy - (u * bzx + v * bzy + w * self.dz(BZ))
                       + p.orm * (self.d2x(bz) + self.d2y(bz) + self.d2z(BZ)))
            jz, jy, jx = bxy - byx, bxz - bzx, byz - bzy
            fu += p.obeta * (by * jz + bz * jy)
            fv += p.obeta * (bz * jx - bx * jz)
            fw -= p.obeta * (bx * jy + by * jx)
            heat += p.obeta * p.orm * p.ocv * (jx * jx + jy * jy + jz * jz)
        ft += r * heat
        return out

    def walls(self, s):
        p = self.p
        for a, b, c in ((1, 2, 3), (-2, -3, -4)):
            for f in (0, 1):
                s[f][a] = s[4][a] * (p.c43 * s[f][b] / s[4][b] - p.c13 * s[f][c] / s[4][c])
            s[2][a] = 0.0
            if p.lmag:
                s[7][a] = 0.0
        s[3][1] = 1.0
        s[3][-2] = p.c43 * s[3][-3] - p.c13 * s[3][-4] + self.bot_flux

    def cfl(self, s):
        p, c = self.p, slice(1, -1)
        ro, tt = s[4][c], s[3][c]
        uu = (s[0][c] ** 2 + s[1][c] ** 2 + s[2][c] ** 2) / ro ** 2
        a2 = p.gamma * tt
        if p.lmag:
            a2 = a2 + (s[5][c] ** 2 + s[6][c] ** 2 + s[7][c] ** 2) * p.obeta / ro
        lim = [(self.dd / (uu.sqrt() + a2.sqrt())).min(), (0.5 * self.dd ** 2 * p.repr * p.cv * ro / self.rka).min(),
               (0.375 * self.dd ** 2 * p.re * ro).min()]
        if p.lmag:
            lim.append((0.5 * self.dd ** 2 * p.rm).min())
        return p.sf * float(torch.stack(lim).min()), float((uu / tt / p.gamma).max().sqrt())

    def step(self, s, tend=None):
        """One RK3 step in place; returns its DT and Mach number."""
        p = self.p
        dt, mach = self.cfl(s)
        z = [f[1:-1].clone() for f in s]
        order = (0, 1, 2, 3, None, 4, 5, 6)   # tendencies have no density row
        for gam, zeta in ((p.gam1, p.zeta1), (p.gam2, p.zeta2), (p.gam3, None)):
            rhs = self.rhs(s)
            ghost = 1.0 / s[4][0], 1.0 / s[4][-1]
            for f, r in enumerate(rhs):
                if tend is not None and order[f] is not None:
                    r += tend[order[f]]
                s[f][1:-1] = z[f] + gam * dt * r
                if zeta is not None:
                    z[f] = s[f][1:-1] + zeta * dt * r
            del rhs
            s[4][0], s[4][-1] = ghost
            self.walls(s)
        return dt, mach

    def profiles(self, s):
        p, c = self.p, slice(1, -1)
        ro, tt, rw = s[4][c], s[3][c], s[2][c]
        ke = (s[0][c] ** 2 + s[1][c] ** 2 + rw ** 2) / ro ** 2
        m = lambda f: f.mean(dim=(1, 2))  # noqa: E731
        ttm = m(tt)
        d = torch.empty_like(ttm)
        d[1:-1] = ttm[2:] - ttm[:-2]
        d[0] = -3 * ttm[0] + 4 * ttm[1] - ttm[2]
        d[-1] = 3 * ttm[-1] - 4 * ttm[-2] + ttm[-3]
        me = m(0.5 * (s[5][c] ** 2 + s[6][c] ** 2 + s[7][c] ** 2)) if p.lmag else torch.zeros_like(ttm)
        return torch.stack([m(ro), ttm, m(0.5 * ro * ke), m(2.5 * ro * tt),
                            m(-rw * (2.5 * (tt - ttm[:, None, None]) + 0.5 * ke)),
                            d * self.az[:, 0, 0] * self.rka[:, 0, 0] / p.repr, me])


def _taps(x):
    """The 27 shifted copies of [nz, ny, nx, C]: periodic in x and y, zero outside in z."""
    for tap in range(27):
        dx, dy, dz = tap % 3 - 1, tap // 3 % 3 - 1, tap // 9 - 1
        s = torch.roll(x, (-dy, -dx), (1, 2))
        if dz:
            o = torch.zeros_like(s)
            if dz > 0:
                o[:-1] = s[1:]
            else:
                o[1:] = s[:-1]
            s = o
        yield tap, s


def _conv(x, w, b):
    cin, out = x.shape[3], b.expand(x.shape[:3] + b.shape).clone()
    for tap, s in _taps(x):
        out += s @ w[:, tap * cin:(tap + 1) * cin].T
    return out


def _forward(net, feat):
    acts, x = [feat], feat
    for li, (_, _, relu) in enumerate(closure.LAYERS):
        x = _conv(x, net.w16[li].double(), net.b[li].double())
        x = x.clamp_min(0) if relu else x
        acts.append(x)
    return acts


def _features(s, in_scale):
    c = slice(1, -1)
    dev = lambda f: f - f.mean(dim=(1, 2), keepdim=True)  # noqa: E731
    ro = s[4][c]
    f = [s[0][c] / ro, s[1][c] / ro, s[2][c] / ro, dev(s[3][c]), dev(ro), s[5][c], dev(s[6][c]), s[7][c]]
    out = torch.zeros(ro.shape + (16,), dtype=torch.float64, device="cuda")
    out[..., :8] = torch.stack(f, -1) * in_scale.double()
    return out


def _tendencies(model, s, net):
    q = _forward(net, _features(s, net.in_scale))[-1][..., :12] * net.out_scale.double()
    P = [q[..., i] for i in range(12)]
    x, y = model.dx, model.dy

    def z(f):
        d = torch.zeros_like(f)
        d[1:-1] = (f[2:] - f[:-2]) * model.az[1:-1]
        return d
    t = [-(x(P[0]) + y(P[3]) + z(P[4])), -(x(P[3]) + y(P[1]) + z(P[5])), -(x(P[4]) + y(P[5]) + z(P[2])),
         -(x(P[6]) + y(P[7]) + z(P[8])) / s[4][1:-1], y(P[11]) - z(P[10]), z(P[9]) - x(P[11]), x(P[10]) - y(P[9])]
    for f in t:
        f[0], f[-1] = 0.0, 0.0
    return t


def _whole(s):
    """[NZ, NPY, NPX] fields with their periodic halos."""
    out = torch.empty(len(s), s[0].shape[0], s[0].shape[1] + 2, s[0].shape[2] + 2, dtype=torch.float64, device="cuda")
    for i, f in enumerate(s):
        out[i, :, 1:-1, 1:-1] = f
    out[:, :, 0], out[:, :, -1] = out[:, :, -2], out[:, :, 1]
    out[:, :, :, 0], out[:, :, :, -1] = out[:, :, :, -2], out[:, :, :, 1]
    return out


def _integrate(su, u, steps, net=None):
    m = _Model(su)
    s = [f[:, 1:-1, 1:-1].clone() for f in u]
    del u
    for _ in range(steps):
        dt, mach = m.step(s, _tendencies(m, s, net) if net else None)
    return m, s, (dt, mach)


def exact(case, seed):
    c = case
    if c["kind"] == "run":
        su, prof = _run_setup(c)
        m, s, sc = _integrate(su, _state(su, prof, seed), c["steps"] // c["per_call"] * c["per_call"],
                              _net(seed) if c["closure"] else None)
        out = {"dt": sc[0], "umach": sc[1]}
        if c["profiles"]:
            out["profiles"] = m.profiles(s)
        w = _whole(s)
        out.update({f: w[i] for i, f in enumerate(mhd3d.FIELDS[:len(s)])})
        return out
    if c["kind"] == "ensemble":
        got = [_integrate(su, _state(su, prof, seed + 7 * i), c["steps"]) for i, (su, prof) in enumerate(_member_setups(c))]
        return {"dt": np.array([sc[0] for _, _, sc in got]), "state": [_whole(s) for _, s, _ in got]}
    if c["kind"] == "train":
        net = _net(seed)
        feat, tgt = _train_data(c, seed)
        acts = _forward(net, feat.double())
        n = feat.shape[0] * feat.shape[1] * feat.shape[2]
        d = acts[-1][..., :12] - tgt.double()
        out = {"loss": (d * d).sum().reshape(1) / (12 * n), "pred": acts[-1], "dw": [], "db": [], "w": [], "b": []}
        dy = torch.zeros_like(acts[-1])
        dy[..., :12] = 2 * d / (12 * n)
        for li in (2, 1, 0):
            x, cin = acts[li], acts[li].shape[3]
            w = net.w16[li].double()
            g, dx = torch.zeros_like(w), torch.zeros_like(x)
            for tap, sh in _taps(x):
                g[:, tap * cin:(tap + 1) * cin] = dy.reshape(n, -1).T @ sh.reshape(n, -1)
            for tap, sh in _taps(dy):   # the mirrored tap hands dy back
                dx += sh @ w[:, (26 - tap) * cin:(27 - tap) * cin]
            gb = dy.reshape(n, -1).sum(0)
            out["dw"].insert(0, g)
            out["db"].insert(0, gb)
            for key, par, gr in (("w", net.w[li], g), ("b", net.b[li], gb)):
                # Adam's first step: m/(1-b1) = g, v/(1-b2) = g*g
                out[key].insert(0, par.double() - 1e-3 * gr / (gr.abs() + 1e-8))
            dy = dx * (x > 0)
        return out
    su, prof = _setup(c["nx"], c["ny"], c["nz"])
    s = [f[1:-1, 1:-1, 1:-1] for f in _state(su, prof, seed)]
    nz, ny, nx = (v // 4 for v in (c["nz"], c["ny"], c["nx"]))

    def box(f): return f.reshape(nz, 4, ny, 4, nx, 4).mean(dim=(1, 3, 5))
    mom, tt, ro, b = s[:3], s[3], s[4], s[5:]
    v = [m / ro for m in mom]
    R, M, E, B = box(ro), [box(m) for m in mom], box(ro * tt), [box(f) for f in b]
    cv = [m / R for m in M]
    tg = [box(mom[i] * v[j]) - M[i] * cv[j] for i, j in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
    tg += [box(m * tt) - M[i] * E / R for i, m in enumerate(mom)]
    for i, j in ((1, 2), (2, 0), (0, 1)):
        tg.append(box(v[i] * b[j] - v[j] * b[i]) - (cv[i] * B[j] - cv[j] * B[i]))
    cs = [torch.cat([f[:1], f, f[-1:]]) for f in M + [E / R, R] + B]
    return {"feat": _features(cs, _net(0).in_scale), "targets": torch.stack(tg, -1), "coarse": _whole(cs).reshape(-1)}
