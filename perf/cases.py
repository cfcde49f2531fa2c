"""Workloads the engine is timed on: what a waveform-inversion program has it do.

A case is a dict of plain values. `listed()` gives the named ones, `draw(rng)` more
of the same ranges. `prepare` makes what the program holds before the call (model,
wavelets, observed traces, the engine); `run` is one pass through the public Python
calls; `work` the bytes and operations a pass cannot do without; `exact` the same
outputs from a plain torch propagator in 64 bits.

Kinds: "forward" (synthetic seismograms), "gradient" (one iteration's shot
gradients), "trial" (a step-length test: new model, forward, misfit), "td" (the
time-domain gradient kernels), "vjp" (the exact discrete gradient), "hessian" (the
approximate Hessian's diagonal), "update" (search direction and model update).
"""
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as tnf

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ifos3d-dev_b200"))
import ifosb  # noqa: E402

FC = {1: 80.0, 0: 100.0}  # source centre frequency in Hz at 1 m cells (viscoelastic, elastic)
BASE = dict(fw=10, nmech=0, free_surf=1, fdcoeff=2, h=1.0, shots=1, nrec=25, nf=0, ntast=1, taufield=False,
            interval=0, rec_hess=0, moduli=False, lbfgs=False, numpar=1, device_out=False)


def _case(name, kind, nx, ny, nz, nt, **kw):
    return dict(BASE, name=name, kind=kind, nx=nx, ny=ny, nz=nz, nt=nt, **kw)


def listed():
    return [
        # a small forward model of a teaching or test problem: launches and latency count
        _case("forward_small", "forward", 48, 44, 40, 60, fw=8, nrec=9),
        # a small inversion problem on ragged sizes: no free surface, spacing not a power of two, DFT every 4th step
        _case("gradient_small_visco", "gradient", 53, 45, 61, 100, fw=8, nmech=1, free_surf=0, h=2.5, shots=2, nrec=16,
              nf=3, ntast=4),
        # the elastic shot-gradient benchmark's grid, receivers and frequencies, one shot
        _case("gradient_elastic_128", "gradient", 128, 128, 128, 400, nf=2),
        # many small shots in one batch
        _case("gradient_batch_64", "gradient", 64, 64, 64, 150, shots=16, nf=2, nrec=36),
        # the viscoelastic forward-modelling benchmark's grid
        _case("forward_visco_256", "forward", 256, 256, 256, 150, nmech=3, nrec=400),
        # one shot of the batched viscoelastic gradient benchmark
        _case("gradient_visco_384", "gradient", 384, 256, 384, 30, nmech=3, nf=4, nrec=1024, device_out=True),
        # a step-length test of a viscoelastic inversion with a Q field, odd grid, spacing not a power of two
        _case("trial_visco_odd", "trial", 131, 101, 150, 100, nmech=2, h=3.0, shots=2, nrec=100, taufield=True),
        # the time-domain gradient with checkpoints kept by the forward
        _case("td_elastic_112", "td", 128, 96, 112, 120, interval=40),
        # the exact discrete gradient, elastic
        _case("vjp_exact_60", "vjp", 64, 56, 60, 80, nrec=36, interval=20),
        # the approximate Hessian: Green's functions of some receivers, one shot
        _case("hessian_96", "hessian", 96, 80, 88, 100, nf=2, nrec=16, rec_hess=6, shots=3),
        # conjugate-gradient direction and two test models
        _case("update_cg_128", "update", 128, 128, 128, 0),
        # L-BFGS direction and a test model, an odd grid
        _case("update_lbfgs_160", "update", 160, 131, 150, 0, lbfgs=True, numpar=2),
    ]


def draw(rng):
    kind = rng.choice(["forward", "forward", "gradient", "gradient", "gradient", "trial", "td", "vjp", "hessian", "update"])
    top = {"forward": 200, "gradient": 200, "trial": 140, "td": 120, "vjp": 56, "hessian": 90, "update": 150}[kind]
    size = lambda: int(round(math.exp(rng.uniform(math.log(36), math.log(top)))))  # noqa: E731
    c = dict(BASE, kind=kind, nx=size(), ny=size(), nz=size(), fw=rng.choice([6, 8, 10]))
    cells = c["nx"] * c["ny"] * c["nz"]
    c["nmech"] = rng.choice([0, 0, 1, 2, 3]) if kind in ("forward", "gradient", "trial", "td", "vjp") else 0
    c["taufield"] = bool(c["nmech"]) and rng.random() < 0.3
    c["free_surf"] = rng.choice([1, 1, 0])
    c["fdcoeff"] = rng.choice([1, 2])
    c["h"] = rng.choice([1.0, 1.0, 2.0, 2.5, 0.7])
    c["nrec"] = rng.choice([4, 9, 25, 100])
    budget = {"forward": 6e8, "gradient": 3e8, "trial": 2e8, "td": 1e8, "vjp": 1.2e7, "hessian": 6e7, "update": 1e9}[kind]
    steps = max(24, min(400, int(budget / cells)))
    c["nt"] = int(round(math.exp(rng.uniform(math.log(24), math.log(max(25, steps))))))
    c["shots"] = max(1, min(rng.choice([1, 1, 2, 3, 5, 8]), int(budget / cells / c["nt"])))
    if kind in ("gradient", "hessian"):
        c["nf"] = rng.choice([1, 2, 3, 4, 5])
        c["ntast"] = rng.choice([1, 1, 1, 2, 5])
    if kind in ("td", "vjp"):
        c["interval"] = rng.choice([10, 17, 25, 50])
    if kind == "vjp":
        c["moduli"] = c["nmech"] > 0 or rng.random() < 0.5
    if kind == "hessian":
        c["rec_hess"] = min(c["nrec"], rng.choice([2, 4, 5]))
    if kind == "update":
        c["lbfgs"] = rng.random() < 0.5
        c["numpar"] = rng.choice([1, 2])
        c["nt"] = 0
    return c


# ---------------------------------------------------------------------------
# inputs

def _dt(c):
    return float(np.float32(1e-4 * c["h"]))


def _fc(c):
    return FC[min(1, c["nmech"])] / c["h"]


def _freqs(c):
    return [20.0 * (l + 1) / c["h"] for l in range(c["nf"])]


def _profile(c):
    """CPML profiles of one axis (Komatitsch & Martin 2007, cubic grading), the same on
    all three axes: K, a, b on full and half nodes, [6][2 fw]."""
    fw, h, dt = c["fw"], c["h"], _dt(c)
    d0 = -4 * 4000.0 * math.log(8e-4) / (2 * fw * h)
    amax = math.pi * _fc(c)
    rows = np.zeros((6, 2 * fw))
    for half in (0, 1):
        pos = (fw - np.arange(fw) - 0.5 * half) / fw
        d = d0 * (0.25 * pos + 0.75 * pos ** 3)
        k = 1 + pos ** 3
        al = amax * (1 - pos)
        b = np.exp(-(d / k + al) * dt)
        a = d * (b - 1) / (k * (d + k * al))
        for q, v in enumerate((k, a, b)):
            rows[3 * half + q, :fw] = v
            rows[3 * half + q, fw:] = v[::-1] if half else np.concatenate(([v[-1]], v[:0:-1]))
    return rows.astype(np.float32)


def _model(c, seed):
    """Depth gradient with Gaussian blobs, as float32 numpy arrays [NY][NX][NZ]."""
    rng = np.random.default_rng(seed)
    dev = "cuda"
    ny, nx, nz = c["ny"], c["nx"], c["nz"]
    ax = [torch.arange(n, device=dev, dtype=torch.float32) for n in (ny, nx, nz)]
    vp = (2500 + 1000 * ax[0] / ny)[:, None, None].expand(ny, nx, nz).clone()
    tf = torch.ones_like(vp) if c["taufield"] else None
    for _ in range(4):
        g = [torch.exp(-((a - float(rng.uniform(0.2, 0.8)) * n) ** 2) / (2 * (0.1 * n) ** 2)) for a, n in zip(ax, (ny, nx, nz))]
        blob = g[0][:, None, None] * g[1][None, :, None] * g[2][None, None, :]
        vp *= 1 + float(rng.uniform(-0.1, 0.1)) * blob
        if tf is not None:
            tf += float(rng.uniform(0.2, 0.8)) * blob
    rho = 1700 + 0.2 * vp
    vs = vp / (1.75 + 0.1 * float(rng.random()))
    m = dict(taus=None, taup=None, eta=None)
    den = torch.ones((), device=dev)
    L = c["nmech"]
    if L:
        fl = np.exp(np.linspace(math.log(20.0), math.log(200.0), L)) / c["h"] if L > 1 else np.array([63.0 / c["h"]])
        tau = (tf if tf is not None else torch.ones_like(vp)) * (0.045 / (0.6 + 0.4 * L))
        w2 = (fl[0] / fl) ** 2
        den = 1 + tau * float((w2 / (1 + w2)).sum())
        m["taus"] = m["taup"] = tau
        m["eta"] = (_dt(c) * 2 * math.pi * fl).astype(np.float32)
    m.update(rho=rho, pi=vp * vp * rho / den, u=vs * vs * rho / den)
    return {k: (v.float().cpu().numpy() if torch.is_tensor(v) else v) for k, v in m.items()}


def _grid_points(c, n, j, margin):
    side = math.ceil(math.sqrt(n))
    xs = np.linspace(margin, c["nx"] - margin + 1, side).round().astype(int)
    zs = np.linspace(margin, c["nz"] - margin + 1, math.ceil(n / side)).round().astype(int)
    return np.array([[x, j, z] for x in xs for z in zs], np.int32)[:n]


def _inputs(c, seed):
    """Shots (srcpos, signals), receivers, observed traces."""
    rng = np.random.default_rng(seed + 77)
    p = _params(c)
    fc, dt, nt = _fc(c), _dt(c), c["nt"]
    t = np.arange(1, nt + 1) * dt
    j_rec = 1 if c["free_surf"] else c["fw"] + 2
    rec = _grid_points(c, c["nrec"], j_rec, c["fw"] + 3)
    shots, obs = [], np.zeros((c["shots"], 3, len(rec), p.nt), np.float32)
    for s in range(c["shots"]):
        pos = [int(rng.integers(c["fw"] + 2, n - c["fw"])) for n in (c["nx"], c["nz"])]
        i, j, k = pos[0], min(c["ny"] - c["fw"] - 1, c["fw"] + 3), pos[1]
        amp = float(rng.uniform(0.8, 1.2))
        wave = np.where(t <= 1 / fc, 0.75 * math.pi * fc * np.sin(math.pi * t * fc) ** 3, 0.0) * amp
        shots.append((np.array([[i, j, k, 0.0, fc, amp, 1.0]], np.float32), wave.astype(np.float32)[None]))
        dist = c["h"] * np.sqrt(((rec - np.array([i, j, k])) ** 2).sum(1))
        arg = math.pi * fc * (t[None, :] - 1 / fc - (dist / 2800.0)[:, None])
        obs[s] = (rng.uniform(0.5, 1.5, (3, 1, 1)) * 2e-8 * ((1 - 2 * arg ** 2) * np.exp(-arg ** 2))[None]
                  / (3 + dist / c["h"])[None, :, None]).astype(np.float32)
    return shots, rec, obs


def _params(c):
    return ifosb.make_params(c["nx"], c["ny"], c["nz"], dh=c["h"], dt=_dt(c), nt=max(2, c["nt"]), fdcoeff=c["fdcoeff"],
                             free_surf=c["free_surf"], fw=c["fw"], nmech=c["nmech"])


def _update_inputs(c, seed):
    """Gradients of successive iterations and the ghosted model an optimiser sees."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (3, c["ny"], c["nx"], c["nz"])
    base = torch.randn(shape, generator=g, device="cuda")
    grads = [(1e-20 * (base + 0.5 * torch.randn(shape, generator=g, device="cuda"))).cpu().numpy()
             for _ in range(5 if c["lbfgs"] else 2)]
    if c["lbfgs"]:
        grads = [a * np.float32(1e20) for a in grads]
    m = _model(c, seed)
    return grads, [ifosb.ghost_wrap(m[k]) for k in ("rho", "pi", "u")]


V0 = (3000.0, 1700.0, 2300.0)
STEP = 0.01


def prepare(case, seed):
    c = dict(BASE, **case)
    st = dict(c=c)
    if c["kind"] == "update":
        grads, model = _update_inputs(c, seed)
        opt = ifosb.Optimizer(c["nx"], c["ny"], c["nz"], numpar=c["numpar"], bfgsnum=5 if c["lbfgs"] else 0)
        if c["lbfgs"]:  # the history of four earlier iterations
            w = _weight(c)
            m = [a.copy() for a in model]
            for it in range(1, 5):
                g = grads[it - 1].copy()
                opt.lbfgs_savegrad(g) if it == 1 else opt.lbfgs(g, it)
                opt.modelupdate(g, *m, STEP, w, *V0, lbfgs=True, it_group=it)
            model = m
        else:
            opt.conjugate(grads[0].copy(), 1)
        return dict(st, opt=opt, grad=grads[-1], model=model)
    shots, rec, obs = _inputs(c, seed)
    m = _model(c, seed)
    eng = ifosb.Engine(_params(c), max_shots=c["shots"], max_nf=c["nf"])
    eng.set_cpml(np.tile(_profile(c), (3, 1)))
    eng.set_receivers(rec)
    if c["nf"]:
        eng.set_frequencies(_freqs(c), c["ntast"])
    if c["kind"] == "td":
        eng.set_td_checkpoints(c["interval"])
    if c["kind"] != "trial":
        eng.set_model(**m)
    if c["device_out"]:
        st["out"] = torch.zeros((3, c["ny"], c["nx"], c["nz"]), dtype=torch.float64, device="cuda")
    if c["kind"] == "hessian":
        st["sig"] = shots[0][1][0]
    return dict(st, eng=eng, shots=shots, obs=obs, model=m)


def _weight(c):
    return np.array([1.0, 0.5 if c["numpar"] > 1 else 0.0, 0.0], np.float32)


def run(st):
    c, kind = st["c"], st["c"]["kind"]
    if kind == "update":
        opt, w = st["opt"], _weight(c)
        g = st["grad"].copy()
        test = [a.copy() for a in st["model"]]
        if c["lbfgs"]:
            opt.lbfgs(g, 5)
            opt.modelupdate(g, *test, STEP, w, *V0, lbfgs=True, it_group=5)
            return dict(g=g[:c["numpar"]], rho=test[0], pi=test[1], u=test[2])
        opt.conjugate(g, 0)
        opt.modelupdate(g, *test, STEP, w, *V0)
        two = [a.copy() for a in st["model"]]
        opt.modelupdate(g, *two, 2 * STEP, w, *V0)
        return dict(g=g, pi1=test[1], u1=test[2], pi2=two[1], u2=two[2])
    e = st["eng"]
    if kind == "forward":
        return dict(sections=e.forward(st["shots"]))
    if kind == "gradient":
        e.zero_gradient()
        mis = e.shot_gradient(st["shots"], st["obs"])
        if c["device_out"]:
            return dict(misfit=mis, grad=e.get_gradient(fp64=True, out=st["out"]))
        return dict(misfit=mis, grad=e.get_gradient())
    if kind == "trial":
        e.set_model(**st["model"])
        sec = e.forward(st["shots"])
        return dict(sections=sec, misfit=e.residual(st["obs"]))
    if kind == "td":
        e.forward(st["shots"], want_sections=False)
        mis = e.residual(st["obs"])
        return dict(misfit=mis, kernels=e.gradient_td(c["interval"]))
    if kind == "vjp":
        e.forward(st["shots"], want_sections=False)
        e.residual(st["obs"])
        grad, mis = e.vjp_exact(c["interval"], moduli=c["moduli"])
        return dict(misfit=mis, grad=grad)
    if kind == "hessian":
        e.hessian_green(list(range(c["rec_hess"])), st["sig"])
        e.zero_hessian()
        e.forward(st["shots"], want_sections=False)
        e.hessian()
        return dict(hess=e.get_hessian())
    raise KeyError(kind)


def work(case):
    """One pass's necessary traffic and operations: per cell and step the state read and
    written once, the model read once, the PML memories of the frame read and written
    once, the DFT accumulators once per DFT step."""
    c = dict(BASE, **case)
    n = c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "update":
        if c["lbfgs"]:
            return dict(bytes=c["numpar"] * n * 8.0 * 4 * 5 + n * 4.0 * 9, flops=n * c["numpar"] * 40.0)
        return dict(bytes=n * 4.0 * (12 + 9 + 9), flops=n * 120.0)
    L, fw = c["nmech"], c["fw"]
    dims = (c["nx"], c["ny"], c["nz"])
    slabs = sum((1 if a == 1 and c["free_surf"] else 2) * fw * n / d for a, d in enumerate(dims))
    cells = n * c["shots"] * c["nt"]
    step = (84.0 + (48 * L + 8 if L else 0)) * cells + 48.0 * slabs * c["shots"] * c["nt"]
    fl = (150.0 + 60 * L) * cells
    dft = 48.0 * c["nf"] * cells / c["ntast"]
    k = c["kind"]
    if k in ("forward", "trial"):
        return dict(bytes=step + (5 * 4.0 * n if k == "trial" else 0), flops=fl)
    if k == "gradient":
        return dict(bytes=2 * (step + dft) + 48.0 * c["nf"] * n * c["shots"], flops=2 * (fl + 24.0 * c["nf"] * cells / c["ntast"]))
    if k == "td":
        return dict(bytes=3 * step + 48.0 * cells, flops=3 * fl + 100.0 * cells)
    if k == "vjp":
        return dict(bytes=8 * step, flops=4 * fl)
    return dict(bytes=(step + dft) * (1 + c["rec_hess"] / c["shots"]) + 48.0 * c["nf"] * n * (c["shots"] + c["rec_hess"]),
                flops=fl * (1 + c["rec_hess"] / c["shots"]) + 250.0 * n * c["nf"] * c["shots"] * c["rec_hess"])


# ---------------------------------------------------------------------------
# the same in 64 bits with plain torch: staggered-grid velocity-stress with CPML,
# relaxation mechanisms and a free surface at the first row (Levander's images)

class _Wave:
    """Fields as [NY][NX][NZ] float64 CUDA tensors; every step makes new tensors, so
    autograd can follow the whole loop."""

    def __init__(self, c, m):
        self.c, self.dt, self.h = c, _dt(c), float(np.float32(c["h"]))
        b = (1.1382, -0.046414) if c["fdcoeff"] == 2 else (9.0 / 8.0, -1.0 / 24.0)
        self.b = [float(np.float32(x)) for x in b]
        self.m = m
        self.prof = torch.tensor(_profile(c), dtype=torch.float64, device="cuda")
        rho, u = m["rho"], m["u"]
        up = lambda a, *ax: torch.roll(a, [-1] * len(ax), ax)  # noqa: E731  +1 neighbour, periodic
        self.rx, self.ry, self.rz = (0.5 * (rho + up(rho, ax)) for ax in (1, 0, 2))
        har = lambda p, q: 4 / (1 / u + 1 / up(u, p) + 1 / up(u, p, q) + 1 / up(u, q))  # noqa: E731
        self.uxy, self.uyz, self.uxz = har(1, 0), har(2, 0), har(2, 1)
        if c["nmech"]:
            ts = m["taus"]
            mean = lambda p, q: 0.25 * (ts + up(ts, p) + up(ts, p, q) + up(ts, q))  # noqa: E731
            self.txy, self.tyz, self.txz = mean(1, 0), mean(2, 0), mean(2, 1)
            self.eta = [float(x) for x in m["eta"]]
        z = torch.zeros((c["ny"], c["nx"], c["nz"]), dtype=torch.float64, device="cuda")
        self.v = [z, z, z]
        self.s = dict(xx=z, yy=z, zz=z, xy=z, yz=z, xz=z)
        self.r = [dict(self.s) for _ in range(c["nmech"])]
        self.psi = {}

    def _d(self, f, axis, up, scale, head=None):
        """Fourth-order difference, at +1/2 (up) or -1/2, zero outside; head: the two rows
        before the first along y."""
        n = f.shape[axis]
        pad = [0] * 6
        pad[2 * (2 - axis)] = 0 if head is not None else 2
        pad[2 * (2 - axis) + 1] = 2
        g = tnf.pad(f, pad)
        if head is not None:
            g = torch.cat([head, g], 0)
        at = lambda o: g.narrow(axis, 2 + o, n)  # noqa: E731
        o = 1 if up else 0
        return scale * (self.b[0] * (at(o) - at(o - 1)) + self.b[1] * (at(o + 1) - at(o - 2)))

    def _pml(self, d, key, axis, half):
        fw = self.c["fw"]
        k, a, b = self.prof[3 * half:3 * half + 3]
        shape = [1, 1, 1]
        shape[axis] = fw
        for far in (0, 1):
            if axis == 0 and not far and self.c["free_surf"]:
                continue
            w = slice(fw * far, fw * far + fw)
            sl = d.narrow(axis, d.shape[axis] - fw if far else 0, fw)
            old = self.psi.get((key, far))
            q = a[w].view(shape) * sl
            q = q if old is None else b[w].view(shape) * old + q
            self.psi[key, far] = q
            sl.copy_(sl / k[w].view(shape) + q)
        return d

    def velocity(self, add=None):
        s, w = self.s, self.dt / self.h
        hd = {k: None for k in ("yy", "xy", "yz")}
        if self.c["free_surf"]:
            hd["yy"] = -torch.stack([s["yy"][2], s["yy"][1]])
            for k in ("xy", "yz"):
                hd[k] = -torch.stack([s[k][1], s[k][0]])
        D = lambda k, ax, up: self._pml(self._d(s[k], ax, up, w, hd.get(k) if ax == 0 else None), ("s", k, ax), ax, int(up))  # noqa: E731
        vx, vy, vz = self.v
        vx = vx + (D("xx", 1, True) + D("xy", 0, False) + D("xz", 2, False)) / self.rx
        vy = vy + (D("yy", 0, True) + D("xy", 1, False) + D("yz", 2, False)) / self.ry
        vz = vz + (D("zz", 2, True) + D("xz", 1, False) + D("yz", 0, False)) / self.rz
        if add is not None:
            (jj, ii, kk), val = add
            vx, vy, vz = (f.index_put((jj, ii, kk), x, accumulate=True) for f, x in zip((vx, vy, vz), val))
        self.v = [vx, vy, vz]

    def stress(self, src=None):
        c, dt, w, m = self.c, self.dt, 1 / self.h, self.m
        L = c["nmech"]
        vx, vy, vz = self.v
        plain = {}

        def D(f, q, ax, up):
            d = self._d(f, ax, up, w)
            if q == ax and c["free_surf"]:
                plain[ax] = d[0].clone()
            return self._pml(d, ("v", q, ax), ax, int(up))
        xx, yy, zz = D(vx, 1, 1, False), D(vy, 0, 0, False), D(vz, 2, 2, False)
        e = dict(xy=D(vx, 1, 0, True) + D(vy, 0, 1, True), yz=D(vy, 0, 2, True) + D(vz, 2, 0, True),
                 xz=D(vx, 1, 2, True) + D(vz, 2, 1, True))
        tr = xx + yy + zz
        pair = dict(xx=yy + zz, yy=xx + zz, zz=xx + yy)
        mu = dict(xy=self.uxy, yz=self.uyz, xz=self.uxz)
        pi, u = m["pi"], m["u"]
        if L:
            tm = dict(xy=self.txy, yz=self.tyz, xz=self.txz)
            gg, ff = pi * (1 + L * m["taup"]), 2 * u * (1 + L * m["taus"])
            s, rn = {}, [dict() for _ in range(L)]
            for q in self.s:
                rate = gg * tr - ff * pair[q] if q in pair else mu[q] * (1 + L * tm[q]) * e[q]
                acc = self.s[q] + dt * rate
                for l in range(L):
                    eta, old = self.eta[l], self.r[l][q]
                    drive = pi * m["taup"] * tr - 2 * u * m["taus"] * pair[q] if q in pair else mu[q] * tm[q] * e[q]
                    new = ((1 - 0.5 * eta) * old - eta * drive) / (1 + 0.5 * eta)
                    acc = acc + 0.5 * dt * (old + new)
                    rn[l][q] = new
                s[q] = acc
            self.r = rn
        else:
            s = {q: self.s[q] + dt * (pi * tr - 2 * u * pair[q] if q in pair else mu[q] * e[q]) for q in self.s}
        if src is not None:
            (j, i, k), a = src
            one = tuple(torch.tensor([x], device="cuda") for x in (j, i, k))
            val = torch.tensor([a], dtype=torch.float64, device="cuda")
            for q in ("xx", "yy", "zz"):
                s[q] = s[q].index_put(one, val, accumulate=True)
        if c["free_surf"]:
            p0, u0 = pi[0], u[0]
            g0 = p0 * (1 + L * m["taup"][0]) if L else p0
            f0 = 2 * u0 * (1 + L * m["taus"][0]) if L else 2 * u0
            hor = plain[1] + plain[2]
            hh = -dt * (g0 - f0) ** 2 * hor / g0 - dt * (g0 - f0) * plain[0]
            row = {"xx": hh, "zz": hh}
            for l in range(L):
                eta = self.eta[l]
                d, ee = 2 * u0 * m["taus"][0], p0 * m["taup"][0]
                t = eta / (1 + 0.5 * eta) * ((d - ee) * (f0 / g0 - 1) * hor - (d - ee) * plain[0])
                for q in ("xx", "zz"):
                    self.r[l][q] = torch.cat([(self.r[l][q][0] + t)[None], self.r[l][q][1:]], 0)
                    row[q] = row[q] + 0.5 * dt * t
                self.r[l]["yy"] = torch.cat([torch.zeros_like(t)[None], self.r[l]["yy"][1:]], 0)
            for q in ("xx", "zz"):
                s[q] = torch.cat([(s[q][0] + row[q])[None], s[q][1:]], 0)
            s["yy"] = torch.cat([torch.zeros_like(hor)[None], s["yy"][1:]], 0)
        self.s = s


def _psource(sig, h):
    s = np.concatenate([[0.0], sig.astype(np.float64), [0.0]])
    return (s[2:] - s[:-2]) / (2 * h ** 3)


def _march(c, m, shot=None, inject=None, rec=None, back=False, keep=None):
    """One shot's time loop. Returns (traces [3][ntr][nt], DFT fields [nf][6]) and calls
    keep(n, velocities) after each step."""
    w = _Wave(c, m)
    nt, dt = c["nt"], _dt(c)
    fr = [float(np.float32(f)) for f in _freqs(c)]
    F = [[None] * 6 for _ in fr]
    total = float(np.float32(np.float32(nt - 1) * np.float32(dt)))
    idx = None if rec is None else tuple(torch.tensor(rec[:, q] - 1, device="cuda").long() for q in (1, 0, 2))
    amp = None if shot is None else _psource(shot[1][0], float(np.float32(c["h"])))
    at = None if shot is None else tuple(int(shot[0][0][q]) - 1 for q in (1, 0, 2))
    tr = []
    for n in range(1, nt + 1):
        w.velocity(None if inject is None else (idx, [2 * inject[q][:, n - 1] for q in range(3)]))
        w.stress(None if shot is None else (at, float(amp[n - 1])))
        if rec is not None and not back:
            tr.append(torch.stack([f[idx] for f in w.v]))
        if fr and n % c["ntast"] == 0:
            t = total - n * dt if back else n * dt
            for l, f in enumerate(fr):
                cs = (math.cos(2 * math.pi * t * f) * dt * c["ntast"], math.sin(2 * math.pi * t * f) * dt * c["ntast"])
                for q in range(6):
                    F[l][q] = w.v[q % 3] * cs[q // 3] if F[l][q] is None else F[l][q].add_(w.v[q % 3], alpha=cs[q // 3])
        if keep is not None:
            keep(n, w.v)
    return torch.stack(tr, -1) if tr else None, F


def _strain(c, f):
    w = _Wave.__new__(_Wave)
    w.b = [float(np.float32(x)) for x in ((1.1382, -0.046414) if c["fdcoeff"] == 2 else (9.0 / 8.0, -1.0 / 24.0))]
    s = 1 / float(np.float32(c["h"]))
    return [w._d(f[q], ax, up, s) for q, ax, up in ((0, 1, False), (0, 0, True), (0, 2, True), (1, 1, True), (1, 0, False),
                                                    (1, 2, True), (2, 1, True), (2, 0, True), (2, 2, False))]


def _lam_mu(f, b):
    lam = (f[0] + f[4] + f[8]) * (b[0] + b[4] + b[8])
    mu = 2 * (f[0] * b[0] + f[4] * b[4] + f[8] * b[8])
    for p, q in ((1, 3), (2, 6), (5, 7)):
        mu = mu + (f[p] + f[q]) * (b[p] + b[q])
    return lam, mu


def _residual(c, tr, obs):
    d = _dt(c) * torch.cumsum(tr - obs, -1)
    return torch.flip(d, [-1]), float((d * d).sum())


def exact(case, seed):
    c = dict(BASE, **case)
    if c["kind"] == "update":
        return _exact_update(c, seed)
    shots, rec, obs = _inputs(c, seed)
    m = {k: (torch.tensor(v, dtype=torch.float64, device="cuda") if isinstance(v, np.ndarray) and v.ndim == 3 else v)
         for k, v in _model(c, seed).items()}
    obs = torch.tensor(obs, dtype=torch.float64, device="cuda")
    if c["kind"] == "vjp":
        return _exact_vjp(c, m, shots, rec, obs)
    with torch.no_grad():
        if c["kind"] in ("forward", "trial"):
            tr = [_march(c, m, sh, rec=rec)[0] for sh in shots]
            out = dict(sections=torch.stack(tr).cpu().numpy())
            if c["kind"] == "trial":
                out["misfit"] = np.array([_residual(c, t, o)[1] for t, o in zip(tr, obs)])
            return out
        if c["kind"] == "gradient":
            return _exact_gradient(c, m, shots, rec, obs)
        if c["kind"] == "td":
            return _exact_td(c, m, shots, rec, obs)
        return _exact_hessian(c, m, shots, rec)


def _exact_gradient(c, m, shots, rec, obs):
    rho, pi, u = m["rho"], m["pi"], m["u"]
    g = torch.zeros((3,) + tuple(rho.shape), dtype=torch.float64, device="cuda")
    mis = []
    for sh, o in zip(shots, obs):
        tr, Ff = _march(c, m, sh, rec=rec)
        diff, j = _residual(c, tr, o)
        mis.append(j)
        _, Fb = _march(c, m, inject=diff, rec=rec, back=True)
        for l, f in enumerate(_freqs(c)):
            w = -1 / (4 * math.pi ** 2 * f * f)
            lam = mu = r = 0.0
            for q in (0, 3):
                a, b = _lam_mu(_strain(c, Ff[l][q:q + 3]), _strain(c, Fb[l][q:q + 3]))
                lam, mu = lam + w * a, mu + w * b
                r = r + sum(x * y for x, y in zip(Ff[l][q:q + 3], Fb[l][q:q + 3]))
            g[0] += 2 * torch.sqrt(rho * pi) * lam
            g[1] += torch.sqrt(rho * u) * (2 * mu - 4 * lam)
            g[2] += r + u / rho * mu + (pi - 2 * u) / rho * lam
    return dict(misfit=np.array(mis), grad=g)


def _exact_td(c, m, shots, rec, obs):
    n = c["nt"] - 1  # step pairs n + m = TIME / DT
    k = torch.zeros((4,) + tuple(m["rho"].shape), dtype=torch.float64, device="cuda")
    mis, dt = [], _dt(c)
    for sh, o in zip(shots, obs):
        hist, U = [], [torch.zeros(3, *m["rho"].shape, dtype=torch.float64, device="cuda")]

        def keep(step, v):
            hist.append(torch.stack(v))
        tr, _ = _march(c, m, sh, rec=rec, keep=keep)
        diff, j = _residual(c, tr, o)
        mis.append(j)
        run_f = torch.cumsum(torch.stack(hist), 0) * dt

        def corr(step, v):
            vb = torch.stack(v)
            U[0] = U[0] + vb * dt
            f = n - step
            if 1 <= f <= n - 1:
                k[0] += (hist[f - 1] * vb).sum(0)
                lam, mu = _lam_mu(_strain(c, run_f[f - 1]), _strain(c, U[0]))
                k[1] += lam
                k[2] += mu
        _march(c, m, inject=diff, rec=rec, back=True, keep=corr)
        k[3] += (run_f[-1] * U[0]).sum(0)
    return dict(misfit=np.array(mis), kernels=k)


def _exact_vjp(c, m, shots, rec, obs):
    names = ("rho", "pi", "u") + (("taus", "taup") if c["nmech"] else ())
    total, mis = None, []
    for sh, o in zip(shots, obs):
        par = {k: m[k].clone().requires_grad_(True) for k in names}
        tr, _ = _march(c, dict(m, **par), sh, rec=rec)
        d = _dt(c) * torch.cumsum(tr - o, -1)
        j = (d * d).sum()
        gr = torch.autograd.grad(j, [par[k] for k in names])
        mis.append(float(j))
        total = gr if total is None else [a + b for a, b in zip(total, gr)]
        del par, tr, d, j, gr
    total = [t.detach() for t in total]
    mis = np.array(mis)
    if c["moduli"]:
        z = torch.zeros_like(total[0])
        return dict(misfit=mis, grad=torch.stack(list(total) + [z] * (5 - len(total))))
    rho, vp, vs = m["rho"], torch.sqrt(m["pi"] / m["rho"]), torch.sqrt(m["u"] / m["rho"])
    return dict(misfit=mis, grad=torch.stack([total[1] * 2 * rho * vp, total[2] * 2 * rho * vs,
                                              total[0] + total[1] * vp * vp + total[2] * vs * vs]))


def _exact_hessian(c, m, shots, rec):
    rho, pi, u = m["rho"], m["pi"], m["u"]
    sig = torch.tensor(shots[0][1][0], dtype=torch.float64, device="cuda")[None]
    zero = torch.zeros_like(sig)
    green = [_march(c, m, inject=[zero, sig, zero], rec=rec[q:q + 1], back=True)[1] for q in range(c["rec_hess"])]
    h = torch.zeros((3,) + tuple(rho.shape), dtype=torch.float64, device="cuda")
    for sh in shots:
        _, Ff = _march(c, m, sh, rec=rec)
        for G in green:
            for l, fr in enumerate(_freqs(c)):
                w = 1 / (2 * math.pi * fr)
                f, fi = _strain(c, Ff[l][:3]), _strain(c, Ff[l][3:])
                b, bi = _strain(c, G[l][:3]), _strain(c, G[l][3:])
                dot = lambda x, y: sum(p * q for p, q in zip(x, y))  # noqa: E731
                (l1, m1), (l2, m2), (l3, m3), (l4, m4) = _lam_mu(fi, b), _lam_mu(f, bi), _lam_mu(fi, bi), _lam_mu(f, b)
                relam, imlam, remu, immu = w * (l1 + l2), w * (l3 - l4), w * (m1 + m2), w * (m3 - m4)
                rer = dot(Ff[l][:3], G[l][:3]) - dot(Ff[l][3:], G[l][3:])
                imr = dot(Ff[l][:3], G[l][3:]) + dot(Ff[l][3:], G[l][:3])
                h[0] += 4 * (relam ** 2 + imlam ** 2) * rho * pi
                h[1] += 4 * ((remu - 2 * relam) ** 2 + (immu - 2 * imlam) ** 2) * rho * u
                h[2] += (rer + relam * (pi - 2 * u) / rho + remu * u / rho) ** 2 + (imr + imlam * (pi - 2 * u) / rho + immu * u / rho) ** 2
    return dict(hess=h)


def _exact_update(c, seed):
    grads, model = _update_inputs(c, seed)
    grads = [torch.tensor(g, dtype=torch.float64, device="cuda") for g in grads]
    rho, pi, u = (torch.tensor(a, dtype=torch.float64, device="cuda") for a in model)
    w = [float(x) for x in _weight(c)]
    step = float(np.float32(STEP))
    inner = (slice(1, -1),) * 3

    def move(g, step, rho, pi, u):
        rho, pi, u = rho.clone(), pi.clone(), u.clone()
        r, vp, vs = rho[inner].clone(), torch.sqrt(pi[inner] / rho[inner]), torch.sqrt(u[inner] / rho[inner])
        dv = [step * w[q] * g[q] * V0[q] for q in range(3)]
        rho[inner] = r + dv[2]
        u[inner] = rho[inner] * (vs + dv[1]) ** 2
        pi[inner] = rho[inner] * (vp + dv[0]) ** 2
        return rho, pi, u, torch.stack([dv[q] / V0[q] for q in range(c["numpar"])])
    if c["lbfgs"]:
        k, S, Y = c["numpar"], {}, {}
        for it in range(1, 6):
            g = grads[it - 1].clone()
            q = g[:k].clone()
            if it > 1:
                Y[it - 1] = Y[it - 1] - q
                rh = {v: 1 / (Y[v] * S[v]).sum() for v in S}
                h0 = (Y[it - 1] * S[it - 1]).sum() / (Y[it - 1] ** 2).sum()
                al = {}
                for v in range(it - 1, 0, -1):
                    al[v] = rh[v] * (S[v] * q).sum()
                    q = q - al[v] * Y[v]
                q = q * h0
                for v in range(1, it):
                    q = q + S[v] * (al[v] - rh[v] * (Y[v] * q).sum())
            Y[it] = grads[it - 1][:k].clone()
            g[:k] = q
            rho, pi, u, S[it] = move(g, step, rho, pi, u)
        return dict(g=g[:k], rho=rho, pi=pi, u=u)
    p, g = grads
    beta = [float((g[q] * (g[q] - p[q])).sum() / (p[q] ** 2).sum()) for q in range(3)]
    beta[0] = min(max(beta[0], 0.0), 0.5)
    d = torch.stack([p[q] * beta[q] + g[q] for q in range(3)])
    d = torch.stack([x / x.abs().max() for x in d])
    _, p1, u1, _ = move(d, step, rho, pi, u)
    _, p2, u2, _ = move(d, float(np.float32(2 * STEP)), rho, pi, u)
    return dict(g=d, pi1=p1, u1=u1, pi2=p2, u2=u2)
