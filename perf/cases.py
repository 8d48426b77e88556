"""Cases of the engine's timing: the calls that forward modelling and full-waveform inversion make, through
``dsh.Engine``, ``dsh.Batch`` and ``dsh.nn.UNet``.

A case is a dict of plain values.  ``prepare`` builds what a program holds before the call (engine, models, shots,
data, output tensors), ``run`` makes the call, ``work`` counts the bytes and operations it cannot do without, and
``exact`` computes the same results in 64 bits with plain torch.  Step lengths are cut (NT 200-2000) so that a pass
stays short; the cost of a pass is proportional to NT.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "denise-sh_b200"))

import dsh  # noqa: E402
from dsh import nn as dnn  # noqa: E402

# Holberg operators of maximum relative error 0.1 % (MAXRELERROR 1), orders 2..10
HOLBERG = {2: (1.0010,), 4: (1.1382, -0.046414), 6: (1.1965, -0.078804, 0.0081781),
           8: (1.2257, -0.099537, 0.018063, -0.0026274), 10: (1.2415, -0.11231, 0.026191, -0.0064682, 0.001191)}
FW, FPML_REFLECTION, NPOWER = 20, 0.001, 4.0
WAVE = dict(kind="forward", l=0, dh=0.5, free_surf=1, shots=1, slots=1, ntr=96, ckpt=0, eprecond=1, grad_q=0, lnorm=2,
            new_model=0)


def _wave(**kw):
    return dict(WAVE, **kw)


def listed():
    return [
        # one test shot of a reduced inversion: the smallest model anyone steps, where launches are the whole cost
        _wave(name="forward_160x80_fd4", nx=160, ny=80, nt=300, fdorder=4, ntr=32),
        # plain elastic forward modelling, one shot of a near-surface survey (the small benchmark configuration)
        _wave(name="forward_500x200_fd4", nx=500, ny=200, nt=2000, fdorder=4),
        # a line-search step: a trial model set from the host, its four test shots modelled
        _wave(name="line_search_1200x400_fd8_l3", nx=1200, ny=400, nt=400, fdorder=8, l=3, shots=4, slots=4, ntr=240,
              new_model=1),
        # forward modelling on an odd grid with absorbing top, DH not a power of two, a high order, an uneven last batch
        _wave(name="forward_701x287_fd10", nx=701, ny=287, nt=500, fdorder=10, dh=0.6, free_surf=0, shots=3, slots=2,
              ntr=57),
        # gradient of a reduced inversion: 8 shots of a small elastic model
        _wave(name="gradient_160x80_fd4", kind="gradient", nx=160, ny=80, nt=600, fdorder=4, shots=8, slots=8, ntr=48,
              new_model=1),
        # the headline gradient: one shot of a large viscoelastic model, every forward step stored, data on the device
        _wave(name="gradient_2000x800_fd8_l3", kind="gradient", nx=2000, ny=800, nt=800, fdorder=8, l=3, dh=0.25,
              ntr=200, new_model=1),
        # the batched gradient: 64 shots in one launch, checkpoints and a recomputed forward pass
        _wave(name="gradient_64shots_ckpt_fd8_l2", kind="gradient", nx=1000, ny=300, nt=192, fdorder=8, l=2, shots=64,
              slots=64, ntr=192, ckpt=14, new_model=1),
        # an iteration of learned-preconditioner inversion: raw gradient and the energy sums, data and results on the host
        _wave(name="gradient_energies_1200x400_fd8_l3", kind="gradient", nx=1200, ny=400, nt=400, fdorder=8, l=3,
              shots=8, slots=8, ntr=240, eprecond=10, new_model=1),
        # the Qs gradient with the Cauchy misfit on an odd grid
        _wave(name="gradient_q_333x157_fd6_l1", kind="gradient", nx=333, ny=157, nt=400, fdorder=6, l=1, dh=0.6,
              free_surf=0, shots=3, slots=3, ntr=45, grad_q=1, lnorm=3, new_model=1),
        # pseudo-Hessian diagonals, the training targets of the learned preconditioner
        _wave(name="hessian_1200x400_fd8_l3", kind="hessian", nx=1200, ny=400, nt=300, fdorder=8, l=3, shots=8, slots=8,
              ntr=240),
        # uneven batch: eight models of different sizes, orders and rheologies advanced together
        dict(name="batch_8_models", kind="batch", models=8, nx_min=256, nx_max=1600, ny_min=128, ny_max=400, nt=240,
             shots_min=8, shots_max=20, ntr=48, layout=5),
        # a training step of the learned preconditioner's network
        dict(name="train_2x400x1200", kind="train", batch=2, h=400, w=1200),
    ]


def draw(rng):
    """One more case of the listed ranges."""
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["forward", "forward", "forward", "gradient", "gradient", "gradient", "hessian", "batch", "train"])
    if kind == "train":
        return dict(kind="train", batch=rng.choice([1, 2]), h=8 * logint(10, 50), w=8 * logint(20, 150))
    if kind == "batch":
        return dict(kind="batch", models=rng.randint(3, 8), nx_min=256, nx_max=logint(700, 1600), ny_min=128,
                    ny_max=logint(200, 400), nt=logint(80, 240), shots_min=8, shots_max=rng.randint(9, 20), ntr=48,
                    layout=rng.randrange(1 << 16))
    nx = logint(160, 2000)
    ny = min(800, max(80, int(nx * rng.uniform(0.3, 0.5))))
    nt = logint(200, 800)
    room = 1.2e9 if kind == "forward" else 0.9e9          # grid-point updates of one pass
    shots = max(1, min(64, logint(1, 64), int(room / (nx * ny * nt))))
    nt = max(100, min(nt, int(room / (nx * ny * shots))))
    l = rng.choice([0, 0, 1, 2, 3])
    c = _wave(kind=kind, nx=nx, ny=ny, nt=nt, fdorder=rng.choice([4, 6, 8, 8, 10]), l=l, dh=rng.choice([0.25, 0.5, 0.6]),
              free_surf=rng.choice([0, 1, 1]), shots=shots, slots=rng.choice([shots, shots, (shots + 1) // 2]),
              ntr=rng.randint(16, min(nx // 2, 240)), new_model=rng.choice([0, 1]))
    if kind == "gradient":
        c["eprecond"] = rng.choice([1, 1, 10])
        c["lnorm"] = rng.choice([2, 2, 2, 3])
        c["grad_q"] = int(l > 0 and rng.random() < 0.25)
        c["ckpt"] = int(math.ceil(math.sqrt(nt))) if rng.random() < 0.3 else 0
    return c


# ---------------- inputs ----------------

def _smooth(g, ny, nx, sigma):
    """Smooth noise of unit maximum, [ny, nx] float32, correlated over about sigma points."""
    k = max(1, int(sigma))
    small = torch.randn((1, 1, max(2, ny // k + 2), max(2, nx // k + 2)), generator=g)
    big = torch.nn.functional.interpolate(small, size=(ny, nx), mode="bicubic", align_corners=True)[0, 0]
    return big / big.abs().max()


def _model(g, nx, ny, l):
    """Three layers with smooth +-5 % noise and a blob; Qs 20-60."""
    depth = torch.arange(1, ny + 1, dtype=torch.float32)[:, None] / ny
    vs = torch.where(depth < 0.3, 150.0, torch.where(depth < 0.6, 250.0, 400.0)) * (1.0 + 0.05 * _smooth(g, ny, nx, 6))
    rho = torch.where(depth < 0.3, 1800.0, torch.where(depth < 0.6, 1900.0, 2000.0)).expand(ny, nx)
    qs = 20.0 + 40.0 * torch.rand((ny, nx), generator=g) if l else None
    return (vs.numpy().astype(np.float32), np.ascontiguousarray(rho.numpy(), np.float32),
            qs.numpy().astype(np.float32) if l else None)


def _geometry(g, nx, ny, shots, ntr, fc):
    """Sources along the surface, a common receiver line: [(source table [8, 1], receivers [2, ntr])]."""
    jitter = torch.randint(-2, 3, (shots,), generator=g).tolist()
    rec_i = np.linspace(FW // 2 + 2, nx - FW // 2 - 2, ntr).round().astype(np.int32)
    rec = np.array([rec_i, np.full(ntr, 2)], np.int32)
    out = []
    for s in range(shots):
        ix = int(round(nx * (s + 1) / (shots + 1))) + jitter[s]
        out.append((np.array([[min(max(ix, 3), nx - 3)], [3], [0], [0], [fc], [1], [0], [3]], np.float32), rec))
    return out


def _numerics(fdorder, dh, vmax=420.0):
    dt = 0.6 * dh / (math.sqrt(2.0) * sum(abs(c) for c in HOLBERG[fdorder]) * vmax)
    fc = 135.0 / (8.0 * dh) / 2.0
    return float(np.float32(dt)), float(np.float32(fc))


def _params(c, g):
    dt, fc = _numerics(c["fdorder"], c["dh"])
    fl = (fc / 4, fc, 4 * fc)[:c["l"]]
    kw = dict(nx=c["nx"], ny=c["ny"], nt=c["nt"], dh=c["dh"], dt=dt, fdorder=c["fdorder"], maxrelerror=1, fw=FW,
              free_surf=c["free_surf"], l=c["l"], fl=fl, damping=420.0, fpml=fc)
    return kw, _geometry(g, c["nx"], c["ny"], c["shots"], c["ntr"], fc), fc


def _observed(g, c, geo, dt, fc):
    """Recorded traces [shots, ntr, nt]: a Ricker pulse at the direct arrival with cylindrical spreading, and noise."""
    t = torch.arange(1, c["nt"] + 1, dtype=torch.float32) * dt
    out = torch.empty((c["shots"], c["ntr"], c["nt"]))
    for s, (src, rec) in enumerate(geo):
        r = torch.from_numpy(np.abs(rec[0] - src[0, 0])).float() * c["dh"] + c["dh"]
        tau = math.pi * (t[None, :] - 1.5 / fc - r[:, None] / 160.0) / (1.5 / fc)
        out[s] = (1 - 4 * tau ** 2) * torch.exp(-2 * tau ** 2) / torch.sqrt(r[:, None])
        out[s] += 0.01 * torch.randn((c["ntr"], c["nt"]), generator=g)
    return out


def _batch_members(c):
    """The models of an uneven batch, every member as a forward case (layout fixes the sizes)."""
    r = np.random.default_rng(c["layout"])
    out = []
    for k in range(c["models"]):
        n = int(r.integers(c["shots_min"], c["shots_max"] + 1))
        out.append(_wave(nx=int(r.integers(c["nx_min"], c["nx_max"] + 1)), ny=int(r.integers(c["ny_min"], c["ny_max"] + 1)),
                         nt=int(c["nt"] * r.uniform(0.5, 1.0)), fdorder=int(r.choice([4, 6, 8])), l=2 * (k % 2), shots=n,
                         slots=n, ntr=c["ntr"]))
    return out


def _shots(geo):
    return [dsh.Shot(src, rec) for src, rec in geo]


def prepare(case, seed):
    c = case
    g = torch.Generator().manual_seed(seed)
    if c["kind"] == "train":
        x, target, state = _network_inputs(c, g)
        net = dnn.UNet(torch)
        net.load_state(state)
        return dict(case=c, net=net, x=x.cuda(), target=target.cuda())
    if c["kind"] == "batch":
        members, params, groups, models = _batch_members(c), [], [], []
        for m in members:
            models.append(_model(g, m["nx"], m["ny"], m["l"]))
            kw, geo, _ = _params(m, g)
            params.append(dsh.make_params(**kw, max_shots=m["shots"]))
            groups.append(_shots(geo))
        b = dsh.Batch(params)
        for k, m in enumerate(models):
            b.set_model(k, *m)
        seis = torch.empty(sum(m["shots"] * m["ntr"] * m["nt"] for m in members), device="cuda")
        return dict(case=c, batch=b, groups=groups, seis=seis)
    model = _model(g, c["nx"], c["ny"], c["l"])
    kw, geo, fc = _params(c, g)
    eng = dsh.Engine(dsh.make_params(**kw, max_shots=c["slots"], eprecond=c["eprecond"], grad_q=c["grad_q"],
                                     ckpt_every=c["ckpt"]))
    if not c["new_model"]:
        eng.set_model(*model)
    st = dict(case=c, eng=eng, shots=_shots(geo), model=model)
    if c["kind"] == "forward":
        st["seis"] = torch.empty(c["shots"] * c["ntr"] * c["nt"], device="cuda")
    elif c["kind"] == "gradient":
        eng.set_misfit(c["lnorm"])
        obs = _observed(g, c, geo, kw["dt"], fc)
        if c["eprecond"] == 10:
            st["obs"] = list(obs.numpy())
        else:
            st["obs"] = obs.cuda()
            st["g"] = torch.empty((2, c["ny"], c["nx"]), device="cuda")
    return st


def run(state):
    st, c = state, state["case"]
    if c["kind"] == "train":
        net = st["net"]
        out = net.forward(st["x"], c["batch"], c["h"], c["w"])
        loss, grad = net.loss_grad(st["target"])
        net.zero_grad()
        net.backward(grad)
        net.adam_step(lr=1e-4)
        return {"out": out, "loss": loss, "grad_w": [k.gwt for k in net.layers()], "grad_b": [k.gb for k in net.layers()],
                "grad_head": [net.ghw, net.ghb]}
    if c["kind"] == "batch":
        st["batch"].forward_device(st["groups"], st["seis"].data_ptr())
        return st["seis"]
    eng = st["eng"]
    if c["new_model"]:
        eng.set_model(*st["model"])
    if c["kind"] == "forward":
        eng.forward_device(st["shots"], st["seis"].data_ptr())
        return st["seis"]
    if c["kind"] == "hessian":
        h_vs, h_rho = eng.hessian_diag(st["shots"])
        return {"h_vs": h_vs, "h_rho": h_rho}
    if c["eprecond"] == 10:
        out = eng.gradient(st["shots"], st["obs"])
        ws, wr = eng.energy_sums()
        out = {"g_vs": out["g_vs"], "g_rho": out["g_rho"], "l2": out["l2"], "ws": ws, "wr": wr}
    else:
        l2 = eng.gradient_device(st["shots"], st["obs"].data_ptr(), st["g"][0].data_ptr(), st["g"][1].data_ptr())
        out = {"g_vs": st["g"][0], "g_rho": st["g"][1], "l2": l2}
    if c["grad_q"]:
        out["g_qs"] = eng.gradient_q()
    return out


# ---------------- work ----------------

def _wave_work(c):
    """Per step a grid's wavefield (velocity, two stresses, 2 L memory variables) is read and written once, its model
    factors are read, and a gradient writes the stored forward wavefield (and reads it in the adjoint pass), the energy and
    the correlation sums; all arrays single precision.  The model factors count once per step for all shots together."""
    n, l, half = c["nx"] * c["ny"], c["l"], c["fdorder"] // 2
    state, model = 8 * (3 + 2 * l), 12 if l == 0 else 20
    flops = 2 * 2 * (3 * half - 1) + 10 + (4 if l == 0 else 8 + 16 * l)
    nb = -(-c["shots"] // c["slots"])                     # launches' worth of slots: the model is read once for each
    io = 4 * c["shots"] * c["ntr"] * c["nt"] + 4 * n * (3 if l else 2)
    if c["kind"] == "gradient":
        stored = 12 + 8 * c["grad_q"]
        fwd, adj = state + 8, state + 24
        if c["ckpt"]:
            fwd += state + stored                          # the recomputed pass writes the segment's wavefield
        else:
            fwd += stored
        adj += stored + 32 * c["grad_q"]
        passes = 3 if c["ckpt"] else 2
        return {"bytes": float(c["nt"] * n * (c["shots"] * (fwd + adj) + nb * passes * model) + io + 8 * n),
                "flops": float(c["nt"] * n * c["shots"] * (passes * flops + 12))}
    extra = 16 if c["kind"] == "hessian" else 0
    return {"bytes": float(c["nt"] * n * (c["shots"] * (state + extra) + nb * model) + io),
            "flops": float(c["nt"] * n * c["shots"] * flops)}


def _network_layers():
    """(input channels, output channels, halvings of the grid) of the 3x3 convolutions in order."""
    ch = [32, 64, 128, 256]
    out, cin = [], 8
    for k, co in enumerate(ch):
        out += [(cin, co, k), (co, co, k)]
        cin = co
    for k in (2, 1, 0):
        out += [(ch[k + 1], ch[k], k), (2 * ch[k], ch[k], k), (ch[k], ch[k], k)]
    return out


def work(case):
    c = case
    if c["kind"] == "train":
        p = c["batch"] * c["h"] * c["w"]
        macs = sum((p >> (2 * k)) * 9 * a * b for a, b, k in _network_layers())
        acts = sum((p >> (2 * k)) * (a + b) for a, b, k in _network_layers())
        return {"bytes": float(2 * acts + 4 * 2 * acts), "flops": float(3 * 2 * macs)}
    if c["kind"] == "batch":
        w = [_wave_work(m) for m in _batch_members(c)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    return _wave_work(c)


# ---------------- the same in 64 bits ----------------

def _pml_vectors(n, dh, dt, fc, clamp):
    """CPML recursion coefficients (a, b) on the full and the half grid of one axis, low strip then high strip."""
    thick = FW * dh
    d0 = -(NPOWER + 1) * 420.0 * math.log(FPML_REFLECTION) / (2 * thick)
    amax = 2 * math.pi * fc / 2
    out = []
    for half in (0.0, dh / 2):
        lo = thick - (dh * np.arange(FW) + half)
        hi = dh * np.arange(n - FW, n) + half - ((n - 1) * dh - thick)
        x = np.concatenate([lo, hi])
        ok = x >= -1e-6 * dh
        xn = np.where(ok, x, 0.0).clip(0) / thick
        d = np.where(ok, d0 * xn ** NPOWER, 0.0)
        alpha = np.where(ok, amax * (1 - xn) + 0.1 * amax, 0.0)
        alpha = alpha.clip(0) if clamp else alpha
        b = np.exp(-(d + alpha) * dt)
        a = np.where(np.trunc(d) != 0, d * (b - 1) / np.where(d + alpha > 0, d + alpha, 1.0), 0.0)
        out.append((torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()))
    return out


class _Wave64:
    """The staggered-grid velocity-stress step with CPML strips and memory variables for a batch of shots."""

    def __init__(self, c, model, kw, geo, fc):
        f = torch.float64
        self.c, self.S = c, len(geo)
        self.dt, self.dh, self.nt = float(np.float32(kw["dt"])), float(np.float32(kw["dh"])), c["nt"]
        self.H, self.hc = c["fdorder"] // 2, [float(np.float32(v)) for v in HOLBERG[c["fdorder"]]]
        vs, rho = (torch.from_numpy(m).to(f).cuda() for m in model[:2])
        self.vs, self.rho = vs, rho
        mu = rho * vs * vs
        ip = 2 / (1 / mu + 1 / mu.roll(-1, 1))
        jp = 2 / (1 / mu + 1 / mu.roll(-1, 0))
        L = c["l"]
        if L:
            self.qs = torch.from_numpy(model[2]).to(f).cuda()
            fl = [float(np.float32(v)) for v in kw["fl"]]
            ts = [1 / (2 * math.pi * v) for v in fl]
            w = 2 * math.pi * fl[0]
            self.sumu = sum((w * t) ** 2 / (1 + (w * t) ** 2) for t in ts)
            self.eta = [self.dt / t for t in ts]
            self.tau = 2 / self.qs
            self.tau_ip = 0.25 * (self.tau + self.tau.roll(-1, 1) + self.tau.roll(-1, 0) + self.tau.roll((-1, -1), (0, 1)))
            self.mi, self.mj = ip / (1 + self.sumu * self.tau_ip), jp / (1 + self.sumu * self.tau)
            ip, jp = self.mi * self.dt * (1 + L * self.tau_ip), self.mj * self.dt * (1 + L * self.tau)
        self.ip, self.jp = ip, jp
        self.px, self.py = _pml_vectors(c["nx"], self.dh, self.dt, fc, True), _pml_vectors(c["ny"], self.dh, self.dt, fc, False)
        t = torch.arange(1, self.nt + 1, dtype=f, device="cuda") * self.dt
        tau = math.pi * (t - 1.5 / fc) / (1.5 / fc)
        self.sig = (1 - 4 * tau ** 2) * torch.exp(-2 * tau ** 2)
        self.src = (torch.tensor([int(s[1, 0]) - 1 for s, _ in geo]), torch.tensor([int(s[0, 0]) - 1 for s, _ in geo]))
        rec = geo[0][1]
        self.rec = (torch.from_numpy(rec[1].astype(np.int64) - 1).cuda(), torch.from_numpy(rec[0].astype(np.int64) - 1).cuda())
        self.zero()

    def zero(self):
        c, H, z = self.c, self.H, dict(dtype=torch.float64, device="cuda")
        ny, nx, S = c["ny"], c["nx"], self.S
        self.vy, self.sxy, self.syz = (torch.zeros((S, ny + 2 * H, nx + 2 * H), **z) for _ in range(3))
        self.r, self.q = ([torch.zeros((S, ny, nx), **z) for _ in range(c["l"])] for _ in range(2))
        self.psi = [torch.zeros((S, ny, 2 * FW), **z) for _ in range(2)] + [torch.zeros((S, 2 * FW, nx), **z) for _ in range(2)]

    def _in(self, a):
        return a[:, self.H:self.H + self.c["ny"], self.H:self.H + self.c["nx"]]

    def _dx(self, a, lead):
        H, ny, nx = self.H, self.c["ny"], self.c["nx"]
        row = a[:, H:H + ny]
        return sum(h * (row[..., H + m + lead:H + m + lead + nx] - row[..., H - m - 1 + lead:H - m - 1 + lead + nx])
                   for m, h in enumerate(self.hc))

    def _dy(self, a, lead):
        H, ny, nx = self.H, self.c["ny"], self.c["nx"]
        col = a[..., H:H + nx]
        return sum(h * (col[:, H + m + lead:H + m + lead + ny] - col[:, H - m - 1 + lead:H - m - 1 + lead + ny])
                   for m, h in enumerate(self.hc))

    def _strip(self, d, psi, ab, axis, top=None):
        n = d.shape[axis]
        for k, sl in ((0, slice(0, FW)), (1, slice(n - FW, n))):
            if k == 0 and axis == 1 and self.c["free_surf"]:
                continue
            a, b = (top if (k == 0 and top is not None) else ab)
            part = slice(k * FW, (k + 1) * FW)
            a, b = (v[part] if axis == 2 else v[part, None] for v in (a, b))
            i = (slice(None),) * axis
            p = psi[i + (part,)]
            p.mul_(b).add_(a * d[i + (sl,)])
            d[i + (sl,)] += p

    def velocity(self, signal, points):
        """One velocity update and the injection of signal at points; returns the acceleration."""
        d, e = self._dx(self.sxy, 0), self._dy(self.syz, 0)
        self._strip(d, self.psi[0], self.px[0], 2)
        self._strip(e, self.psi[2], self.py[0], 1)
        acc = (d + e) / self.rho / self.dh
        v = self._in(self.vy)
        v += self.dt * acc
        for s, j, i, amp in points(signal):
            v[s].index_put_((j, i), amp, accumulate=True)
        return acc

    def stress(self):
        """One stress update; returns the strain rates and the stress increments' sensitivities to tau."""
        L, scale = self.c["l"], (1 / self.dh if self.c["l"] else self.dt / self.dh)
        ux, uy = self._dx(self.vy, 1) * scale, self._dy(self.vy, 1) * scale
        self._strip(ux, self.psi[1], self.px[1], 2)
        self._strip(uy, self.psi[3], self.py[1], 1, top=self.py[0] if L else None)
        sens = []
        for s, mem, u, mod, m, tau in ((self.sxy, self.r, ux, self.ip, getattr(self, "mi", None), getattr(self, "tau_ip", None)),
                                       (self.syz, self.q, uy, self.jp, getattr(self, "mj", None), getattr(self, "tau", None))):
            inc = mod * u
            if L:
                both = sum(mem)
                for k, eta in enumerate(self.eta):
                    mem[k].mul_(1 - eta / 2).sub_(m * eta * tau * u).div_(1 + eta / 2)
                both = both + sum(mem)
                inc = inc + self.dt / 2 * both
                if self.c["grad_q"]:
                    den = 1 + self.sumu * tau
                    sens.append(m * self.dt * (L - self.sumu) / den * u + self.dt / 2 / (tau * den) * both)
            self._in(s).add_(inc)
        return ux, uy, sens


def _forward64(w, hook):
    seis = torch.empty((w.S, w.c["ntr"], w.nt), dtype=torch.float64, device="cuda")
    pts = [(s, w.src[0][s:s + 1].cuda(), w.src[1][s:s + 1].cuda()) for s in range(w.S)]
    for t in range(w.nt):
        amp = w.sig[t].reshape(1)
        acc = w.velocity(amp, lambda a: [(s, j, i, a) for s, j, i in pts])
        seis[:, :, t] = w._in(w.vy)[:, w.rec[0], w.rec[1]]
        hook(t, acc, *w.stress())
    return seis


def _residual64(syn, obs, lnorm):
    """Adjoint source in forward time order and the misfit (LNORM 2 or 3), the first sample taken from the synthetics;
    the Cauchy norm reports no misfit."""
    o = obs.clone()
    o[..., 0] = syn[..., 0]
    if lnorm == 3:
        return (o - syn) / (1 + (o - syn).square()), 0.0
    return syn - o, float((syn - o).square().sum())


def _gradient64(c, model, kw, geo, fc, obs):
    f, n = torch.float64, c["nx"] * c["ny"]
    per = max(1, int(50e9 / ((3 + 2 * c["grad_q"]) * 8 * n * c["nt"])))
    su = sr = sws = swr = sqx = sqy = 0.0
    l2 = 0.0
    for s0 in range(0, c["shots"], per):
        g = geo[s0:s0 + per]
        w = _Wave64(c, model, kw, g, fc)
        S, shape = len(g), (len(g), c["ny"], c["nx"])
        store = torch.empty((c["nt"], 3 + 2 * c["grad_q"]) + shape, dtype=f, device="cuda")
        ws, wr, gu, gr = (torch.zeros(shape, dtype=f, device="cuda") for _ in range(4))

        def keep(t, acc, ux, uy, sens):
            for k, a in enumerate([acc, ux, uy] + sens):
                store[t, k] = a
            ws.add_(w._in(w.vy).square())

        syn = _forward64(w, keep)
        res, part = _residual64(syn, obs[s0:s0 + per].to(f).cuda(), c["lnorm"])
        l2 += part
        w.zero()
        ex, ey, gx, gy = (torch.zeros(shape, dtype=f, device="cuda") for _ in range(4)) if c["grad_q"] else (None,) * 4
        for t in range(c["nt"] - 1, -1, -1):
            old = w._in(w.vy).clone()
            w.velocity(t, lambda k: [(s, w.rec[0], w.rec[1], res[s, :, k]) for s in range(S)])
            gr.add_(old * store[t, 0])
            ux, uy, _ = w.stress()
            gu.add_(store[t, 1] * w._in(w.sxy) + store[t, 2] * w._in(w.syz))
            wr.add_(w._in(w.vy).square())
            if c["grad_q"]:
                gx.add_(ex * store[t, 3])
                gy.add_(ey * store[t, 4])
                ex.add_(ux * w.dt)
                ey.add_(uy * w.dt)
        if c["eprecond"] == 1:
            we = (ws * wr).sqrt()
            we = we + 0.005 * we.amax((1, 2), keepdim=True)
            gu, gr = gu / (we * w.vs.mean() ** 2), gr / (we * w.rho.mean() ** 2)
        su, sr, sws, swr = su + gu.sum(0), sr + gr.sum(0), sws + ws.sum(0), swr + wr.sum(0)
        if c["grad_q"]:
            sqx, sqy = sqx + gx.sum(0), sqy + gy.sum(0)
        del store
    mu = -w.dt * su
    out = {"g_vs": 2 * w.rho * w.vs * mu, "g_rho": w.vs ** 2 * mu - w.dt * sr, "l2": l2}
    if c["eprecond"] == 10:
        out["ws"], out["wr"] = sws.cpu().numpy(), swr.cpu().numpy()
        out["g_vs"], out["g_rho"] = out["g_vs"].cpu().numpy(), out["g_rho"].cpu().numpy()
    if c["grad_q"]:
        x = -2 / w.rho * sqx
        x = 0.25 * (x + x.roll(1, 1) + x.roll(1, 0) + x.roll((1, 1), (0, 1)))
        out["g_qs"] = ((-2 / w.rho * sqy + x) * (-2 / w.qs ** 2)).cpu().numpy()
    return out


def _network_inputs(c, g):
    """Network input bf16 [P, 8] (four normalised maps, zero padding), target [P], He-initialised weights."""
    b, h, w = c["batch"], c["h"], c["w"]
    x = torch.zeros((b, h, w, 8))
    t = torch.empty((b, h, w))
    for k in range(b):
        x[k, ..., 0] = _smooth(g, h, w, 12)
        for ch in (1, 2):
            x[k, ..., ch] = -0.5 * (1 + _smooth(g, h, w, 40))
        x[k, ..., 3] = _smooth(g, h, w, 20)
        t[k] = 0.05 * _smooth(g, h, w, 30)
    state = {}
    for k, (a, o, _) in enumerate(_network_layers()):
        state[f"w{k}"] = (torch.randn((o, 9 * a), generator=g) * math.sqrt(2.0 / (9 * a))).numpy()
        state[f"b{k}"] = np.zeros(o, np.float32)
    state["hw"] = (torch.randn(32, generator=g) * math.sqrt(1.0 / 32)).numpy()
    state["hb"] = np.zeros(1, np.float32)
    return x.reshape(-1, 8).to(torch.bfloat16), t.reshape(-1), state


def _train64(c, seed):
    x, target, state = _network_inputs(c, torch.Generator().manual_seed(seed))
    p = {k: torch.from_numpy(v).double().cuda().requires_grad_() for k, v in state.items()}
    a = x.double().cuda().view(c["batch"], c["h"], c["w"], 8).permute(0, 3, 1, 2)
    layers, at = _network_layers(), iter(range(17))
    F = torch.nn.functional

    def conv(a):
        k = next(at)
        cin, cout, _ = layers[k]
        wt = p[f"w{k}"].view(cout, 3, 3, cin).permute(0, 3, 1, 2)
        return torch.relu(F.conv2d(a, wt, p[f"b{k}"], padding=1))

    skips = []
    for lev in range(4):
        a = conv(conv(a if lev == 0 else F.max_pool2d(a, 2)))
        skips.append(a)
    for lev in (2, 1, 0):
        a = conv(a.repeat_interleave(2, 2).repeat_interleave(2, 3))
        a = conv(conv(torch.cat([skips[lev], a], 1)))
    out = torch.einsum("bchw,c->bhw", a, p["hw"]).reshape(-1) + p["hb"]
    loss = (out - target.double().cuda()).square().mean()
    loss.backward()
    return {"out": out.detach(), "loss": loss.detach().reshape(1),
            "grad_w": [p[f"w{k}"].grad.t().contiguous().reshape(-1) for k in range(17)],
            "grad_b": [p[f"b{k}"].grad for k in range(17)], "grad_head": [p["hw"].grad, p["hb"].grad]}


def _forward_member64(c, model, kw, geo, fc):
    per, out = max(1, int(20e9 / (30 * 8 * c["nx"] * c["ny"]))), []
    for s0 in range(0, c["shots"], per):
        w = _Wave64(c, model, kw, geo[s0:s0 + per], fc)
        out.append(_forward64(w, lambda *a: None).reshape(-1))
    return torch.cat(out)


def exact(case, seed):
    c, g = case, torch.Generator().manual_seed(seed)
    if c["kind"] == "train":
        return _train64(c, seed)
    if c["kind"] == "batch":
        out = []
        for m in _batch_members(c):
            model = _model(g, m["nx"], m["ny"], m["l"])
            kw, geo, fc = _params(m, g)
            out.append(_forward_member64(m, model, kw, geo, fc))
        return torch.cat(out)
    model = _model(g, c["nx"], c["ny"], c["l"])
    kw, geo, fc = _params(c, g)
    if c["kind"] == "gradient":
        return _gradient64(c, model, kw, geo, fc, _observed(g, c, geo, kw["dt"], fc))
    if c["kind"] == "forward":
        return _forward_member64(c, model, kw, geo, fc)
    hu = torch.zeros((c["ny"], c["nx"]), dtype=torch.float64, device="cuda")
    hr = torch.zeros_like(hu)
    w = _Wave64(c, model, kw, geo, fc)

    def add(t, acc, ux, uy, sens):
        if t < c["nt"] - 1:
            hu.add_((uy.square() + (0.5 * ux).square()).sum(0))
            hr.add_(acc.square().sum(0))

    _forward64(w, add)
    return {"h_vs": (4 * w.rho ** 2 * w.vs ** 2 * hu).cpu().numpy(), "h_rho": (hr + w.vs ** 4 * hu).cpu().numpy()}
