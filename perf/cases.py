"""Performance cases of the CGFD solver: what its users have it do, through
the Python mirror of the C ABI (cgfd.Solver, cgfd.Batch, cgfd.mlp_gradient).

Three kinds of pass:

  steps   a running simulation is advanced by a few RK4 steps, receivers
          recorded and peak velocities kept on the device where the program
          asked for them, and a snapshot of the nine components is taken: the
          loop of a program that writes snapshots as it goes.  Small grids
          give back every cell, larger ones the strided volume that such a
          program saves (the reference's snapshot start/count/stride).
  shot    a whole forward run from host arrays, as for one of many small
          models: create, upload, step, seismograms and peak velocities.
  train   one gradient evaluation of the learned absorbing layer.

Models are Gaussian hills over a layered medium with a random perturbation
(or a flat half-space), CFS-PML on five faces, a free surface on top, a moment
source, and a random smooth velocity field at the start so that every cell,
absorbing layer and surface layer has work from the first step.

exact() restates a pass in 64 bits with plain torch.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "copara-cgfd3d_b200")
G = 3  # ghost cells per side

H = 100.0
DT = 0.006
VMAX = 7000.0
STORAGE = {"f32": 0, "f16": 1, "bf16": 2}


def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def solver_module():
    path = os.path.join(PKG, "python")
    if path not in sys.path:
        sys.path.insert(0, path)
    import cgfd
    return cgfd


def case_of(name, kind, ni, nj, nk, pml=20, steps=20, stride=4, storage="f32", hill=1500.0,
            fault=0, force=False, peak=False, smooth=False, mlp=False, receivers=25, models=1):
    return dict(name=name, kind=kind, ni=ni, nj=nj, nk=nk, pml=pml, steps=steps, stride=stride,
                storage=storage, hill=hill, fault=fault, force=force, peak=peak, smooth=smooth,
                mlp=mlp, receivers=receivers, models=models)


def listed():
    return [
        # the smallest run: a test-sized flat half-space, every cell read back
        # (launches and latency)
        case_of("flat_28x24x20", "steps", 28, 24, 20, pml=5, steps=10, stride=1, hill=0.0,
                receivers=4),
        # one shot of a study with many small models, host arrays in,
        # seismograms out; sources spread over 7^3 nodes
        case_of("shot_62x54x40", "shot", 62, 54, 40, pml=8, steps=120, force=True, smooth=True,
                peak=True),
        # ragged sizes, a finite fault, a surface force and peak velocities
        case_of("fault_118x95x61", "steps", 118, 95, 61, pml=10, steps=20, stride=2, fault=240,
                force=True, peak=True),
        # the flat half-space benchmark (uniform metric)
        case_of("flat_160x160x80", "steps", 160, 160, 80, pml=12, steps=40, stride=2, hill=0.0),
        # a hill model of ordinary size
        case_of("hill_256x256x128", "steps", 256, 256, 128, steps=20),
        # the 400-wide hill benchmark
        case_of("hill_400x400x200", "steps", 400, 400, 200, steps=16, receivers=400),
        # the default benchmark, the largest
        case_of("hill_600x600x250", "steps", 600, 600, 250, steps=8, stride=5, receivers=400),
        # half-precision storage, ordinary size
        case_of("hill_256x256x128_f16", "steps", 256, 256, 128, steps=20, storage="f16"),
        # bfloat16 storage, ragged sizes
        case_of("hill_237x211x103_bf16", "steps", 237, 211, 103, pml=16, steps=20,
                storage="bf16"),
        # the thin learned layer on half-precision storage
        case_of("learned_400x400x200_f16", "steps", 400, 400, 200, pml=4, steps=16,
                storage="f16", mlp=True, receivers=400),
        # a batch of uneven models in one launch
        case_of("batch_6x_96to192", "steps", 192, 168, 80, pml=12, steps=10, stride=3, models=6),
        # one gradient of the layer's training, its usual minibatch
        case_of("train_20000", "train", 20000, 1, 1, pml=0, steps=1),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    what = rng.choice(["f32"] * 5 + ["f16", "bf16", "f16", "batch", "shot", "learned", "train"])
    if what == "train":
        return _unnamed("train", side(500, 40000), 1, 1, pml=0, steps=1)
    if what == "shot":
        return _unnamed("shot", side(24, 90), side(24, 90), side(18, 50), pml=rng.randint(4, 10),
                        steps=rng.randint(40, 140), force=rng.random() < 0.5,
                        peak=rng.random() < 0.5, smooth=rng.random() < 0.5)
    if what == "batch":
        return _unnamed("steps", side(60, 180), side(60, 180), side(30, 90), pml=rng.randint(6, 12),
                        steps=rng.randint(6, 12), stride=3, models=rng.randint(2, 6))
    ni, nj, nk = side(24, 420), side(24, 420), side(20, 200)
    cells = ni * nj * nk
    steps = max(8, min(40, int(2.5e8 / cells)))
    return _unnamed("steps", ni, nj, nk, pml=rng.randint(0, min(20, min(ni, nj, nk) // 4)),
                    steps=rng.randint(steps // 2, steps),
                    stride=1 if cells < 3e5 else 2 if cells < 3e6 else 4,
                    storage="f16" if what == "learned" else what,
                    hill=rng.choice([0.0, 800.0, 1500.0]),
                    fault=rng.choice([0, 0, 60, 300]) if what == "f32" else 0,
                    force=rng.random() < 0.3, peak=rng.random() < 0.3,
                    mlp=what == "learned" and min(ni, nj, nk) >= 24,
                    receivers=rng.choice([4, 25, 100]))


def _unnamed(*a, **kw):
    c = case_of("", *a, **kw)
    del c["name"]
    return c


def sizes_of(case):
    """The sizes of a case's models: member q of a batch is smaller by a
    step, with sides that are not round."""
    ni, nj, nk, n = case["ni"], case["nj"], case["nk"], case["models"]
    out = []
    for q in range(n):
        f = 1.0 - 0.5 * q / max(1, n - 1) if n > 1 else 1.0
        out.append((max(24, int(ni * f)), max(24, int(nj * f)), max(20, int(nk * f))))
    return out if n > 1 else [(ni, nj, nk)]


# ------------------------------- the models --------------------------------

def smooth_noise(shape, gen, passes=2):
    """Random field, smoothed with a 3-point binomial per axis and pass,
    standard deviation 1."""
    f = torch.randn(shape, generator=gen, device=gen.device, dtype=torch.float32)
    for _ in range(passes):
        for ax in range(3):
            if shape[ax] >= 3:
                n = shape[ax]
                g = f * 0.5
                g.narrow(ax, 1, n - 1).add_(f.narrow(ax, 0, n - 1), alpha=0.25)
                g.narrow(ax, 0, n - 1).add_(f.narrow(ax, 1, n - 1), alpha=0.25)
                f = g
    return f / f.std()


def pad(a):
    """Valid cells to a full array, edge values in the ghost cells."""
    return torch.nn.functional.pad(a[None, None], (G,) * 6, mode="replicate")[0, 0]


def profiles(n, w0, w1):
    """CFS-PML profiles APD, B, DB of one axis (full length): quadratic
    damping and stretch, linear frequency shift, w0 cells at the low end and
    w1 at the high end."""
    apd, b, db = np.zeros(n + 6), np.ones(n + 6), np.zeros(n + 6)
    for w, at in ((w0, lambda q: q), (w1, lambda q: n - 1 - q)):
        for q in range(w):
            r = (w - q) / w
            d = 3.0 * VMAX * math.log(1e4) / (2.0 * w * H) * r * r
            beta, alpha = 1.0 + 1.5 * r * r, 5.0 * (1.0 - r)
            i = at(q) + G
            apd[i], b[i], db[i] = alpha + d / beta, beta, d / beta
    return apd, b, db


def ricker(f0, t0, n, dt):
    t = np.arange(n) * dt
    a = (math.pi * f0 * (t - t0)) ** 2
    return ((1.0 - 2.0 * a) * np.exp(-a)).astype(np.float32)


def steps_room(case, cells):
    """Steps the receiver record and the source have room for: a program
    that runs on for a good while."""
    if case["kind"] == "shot":
        return case["steps"]
    return min(300000, int(20.0 * 12e9 / cells) + 2000)


def build(case, size, seed):
    """One model: host arrays for the uploads, and the same numbers as torch
    tensors for exact()."""
    ni, nj, nk = size
    dev = device()
    gen = torch.Generator(device=dev).manual_seed(seed)
    rng = np.random.RandomState(seed % (2 ** 31))
    flat = case["hill"] == 0.0
    top = nk + G - 1
    sp = torch.full((nk - 1,), H) if flat else torch.linspace(150.0, 50.0, nk - 1)
    zf = torch.zeros(nk, dtype=torch.float64, device=dev)
    zf[:-1] = -torch.flip(torch.cumsum(torch.flip(sp.double(), [0]), 0), [0]).to(dev)
    con = min(max(int((zf < -min(3000.0, -0.4 * float(zf[0]))).sum()) + G, G), top - 3)
    m = dict(size=size, con=con, flat=flat)
    shape = (ni, nj, nk)
    if flat:
        zx = zy = torch.zeros(shape, dtype=torch.float64, device=dev)
        zz = jac = torch.ones(shape, dtype=torch.float64, device=dev)
    else:
        x = (torch.arange(ni, dtype=torch.float64, device=dev) - (ni - 1) / 2.0) * H
        y = (torch.arange(nj, dtype=torch.float64, device=dev) - (nj - 1) / 2.0) * H
        wid = min(3000.0, 0.2 * H * min(ni, nj))
        hh = min(case["hill"], 0.25 * wid, 0.1 * -float(zf[0]))
        hill = hh * torch.exp(-(x[:, None] ** 2 + y[None, :] ** 2) / wid ** 2)
        zc = zf[con - G]
        wt = torch.clamp((zf - zc) / (0.0 - zc), min=0.0)
        z = zf[None, None, :] + hill[:, :, None] * wt[None, None, :]
        gx, gy, gz = torch.gradient(z, spacing=H, edge_order=1)
        zx, zy, zz, jac = -gx / gz, -gy / gz, 1.0 / gz, gz
    m["metric"] = [pad(a) for a in (zx, zy, zz, jac)]
    del zx, zy, zz, jac
    if flat:
        vp = torch.full(shape, 6000.0, device=dev)
        rho = torch.full(shape, 2670.0, device=dev)
    else:
        vp = torch.empty(shape, device=dev)
        rho = torch.empty(shape, device=dev)
        for lo, hi, v, r in ((0.0, 0.15, 3600.0, 2400.0), (0.15, 0.55, 5200.0, 2600.0),
                             (0.55, 2.0, 6300.0, 2800.0)):
            s = (zf / zf[0] >= lo) & (zf / zf[0] < hi)
            vp[:, :, s] = v
            rho[:, :, s] = r
        p = torch.clamp(smooth_noise(shape, gen), -2.0, 2.0) * 0.05
        vp *= 1.0 + p
        rho *= 1.0 + 0.5 * p
        del p
    m["media"] = [pad(a).float() for a in (vp, vp / math.sqrt(3.0), rho)]
    del vp, rho
    w = case["pml"]
    m["nabs"] = (w, w, w, w, w, 0)
    m["pml"] = [profiles(ni, w, w), profiles(nj, w, w), profiles(nk, w, 0)]
    # sources: one moment source at depth, a force at the surface, a fault
    nt = m["nt"] = steps_room(case, ni * nj * nk)
    nstf = 2 * nt + 4
    ci, cj, ck = G + ni // 2, G + nj // 2, G + max(w + 2, nk // 2)
    m["moment"] = (np.array([[ci, cj, ck]], np.int32),
                   (rng.standard_normal(6) * 2e15).astype(np.float32)[None],
                   ricker(2.0, 0.3, nstf, DT / 2)[None])
    m["force"] = None
    if case["force"]:
        m["force"] = (np.array([[ci + 2, cj - 1, top]], np.int32),
                      np.array([[3e14, -2e14, 1e15]], np.float32),
                      ricker(3.0, 0.2, nstf, DT / 2)[None])
    m["fault"] = None
    if case["fault"]:
        # a rupture that spreads over a dipping plane, one point per cell
        n = case["fault"]
        cols = max(1, int(math.sqrt(2.0 * n)))
        q = np.arange(n)
        da, db = q % cols - cols // 2, q // cols - (n // cols) // 2
        loc = np.stack([ci + da, cj + db, ck + (db + 1) // 2], 1)
        loc[:, 0] = np.clip(loc[:, 0], G, ni + G - 1)
        loc[:, 1] = np.clip(loc[:, 1], G, nj + G - 1)
        loc[:, 2] = np.clip(loc[:, 2], G, top)
        loc = np.unique(loc, axis=0).astype(np.int32)
        n = len(loc)
        fdt = 1.7 * DT
        t = np.arange(200) * fdt
        t0 = np.hypot(loc[:, 0] - ci, loc[:, 1] - cj) * H / 2500.0
        tri = np.clip(1.0 - np.abs(t[None] - t0[:, None] - 0.05) / 0.2, 0.0, None)
        wgt = rng.uniform(0.5, 1.5, n)
        mech = rng.standard_normal(6)
        mom = (1e14 * mech[:, None, None] * (wgt[:, None] * tri)[None]).astype(np.float32)
        m["fault"] = (loc, fdt, mom)
    m["weights"] = None
    if case["smooth"]:
        o = np.arange(-3, 4, dtype=np.float64)

        def block(rows):
            g = [np.exp(-(o - s) ** 2 / 2.25) for s in rng.uniform(-0.5, 0.5, 3)]
            b = g[0][:, None, None] * g[1][None, :, None] * g[2][None, None, :]
            return (b / b[:, :, :rows].sum())[None]
        m["weights"] = (block(7), block(4) if case["force"] else None)
    # receivers on the surface
    k = int(math.isqrt(case["receivers"]))
    ii = np.linspace(G, ni + G - 1, k).astype(int)
    jj = np.linspace(G, nj + G - 1, k).astype(int)
    m["receivers"] = np.array([(i, j, top) for i in ii for j in jj], np.int32)
    # the velocity at the start: all components of small models, Vz of large
    # ones (the rest of the state follows from it in the first steps)
    comps = (0, 1, 2) if ni * nj * nk < 1e7 else (2,)
    m["start"] = {}
    if case["kind"] == "steps":
        for c in comps:
            m["start"][c] = torch.nn.functional.pad(smooth_noise(shape, gen, 3)[None, None],
                                                    (G,) * 6)[0, 0]
    m["mlp"] = None
    if case["mlp"]:
        d = np.load(os.path.join(PKG, "data", "layer_mlp_w4.npz"))
        m["mlp"] = (4, d["weights"], d["gains"])
    return m


def describe(cgfd, case, m):
    ni, nj, nk = m["size"]
    return cgfd.make_desc(ni, nj, nk, H, DT, m["nt"], m["con"], m["nabs"],
                          storage=STORAGE[case["storage"]])


def load(s, case, m):
    host = (lambda a: a if isinstance(a, np.ndarray) else a.cpu().numpy())
    s.upload_metric(*[host(a) for a in m["metric"]])
    s.upload_media(*[host(a) for a in m["media"]])
    s.upload_pml(*[[p[t] for p in m["pml"]] for t in range(3)])
    s.upload_moments(*m["moment"])
    if m["force"]:
        s.upload_forces(*m["force"])
    if m["fault"]:
        s.upload_focal(*m["fault"])
    if m["weights"]:
        s.set_source_smoothing(0, m["weights"][0])
        if m["weights"][1] is not None:
            s.set_source_smoothing(1, m["weights"][1])
    s.set_receivers(m["receivers"])
    if case["peak"]:
        s.enable_peak_velocity()
    if m["mlp"]:
        s.set_boundary_mlp(*m["mlp"][:2])
        s.set_boundary_mlp_gains(m["mlp"][2])


def start(s, m):
    for c, f in m["start"].items():
        s.set_field(c, f.cpu().numpy())


def prepare(case, seed):
    if case["kind"] == "train":
        return dict(case=case, inputs=training(case, seed))
    cgfd = solver_module()
    ms = []
    if case["kind"] == "shot":
        m = build(case, sizes_of(case)[0], seed)
        m["metric"] = [a.cpu().numpy() for a in m["metric"]]
        m["media"] = [a.cpu().numpy() for a in m["media"]]
        return dict(case=case, model=m)
    if case["models"] == 1:
        m = build(case, sizes_of(case)[0], seed)
        s = cgfd.Solver(describe(cgfd, case, m))
        load(s, case, m)
        s.prepare()
        start(s, m)
        return dict(case=case, solver=s, sizes=[m["size"]])
    ms = [build(case, z, seed * 16 + q) for q, z in enumerate(sizes_of(case))]
    b = cgfd.Batch([describe(cgfd, case, m) for m in ms])
    for s, m in zip(b.models, ms):
        load(s, case, m)
    b.prepare()
    for s, m in zip(b.models, ms):
        start(s, m)
    return dict(case=case, batch=b, sizes=[m["size"] for m in ms])


def snapshot(s, size, stride):
    first = (G, G, G)
    count = [-(-n // stride) for n in size]
    every = (stride,) * 3
    return {"velocity": s.snapshot(first, count, every, comps=(0, 1, 2)),
            "stress": s.snapshot(first, count, every, comps=range(3, 9))}


def run(state):
    case = state["case"]
    cgfd = solver_module()
    if case["kind"] == "train":
        w, x, t = state["inputs"]
        loss, grad = cgfd.mlp_gradient(w, x, t)
        return {"loss": loss, "gradient": grad}
    if case["kind"] == "shot":
        m = state["model"]
        with cgfd.Solver(describe(cgfd, case, m)) as s:
            load(s, case, m)
            s.step(case["steps"])
            out = seismograms(s.seismograms())
            if case["peak"]:
                out["peak"] = s.peak_velocity()
        return out
    if "batch" in state:
        b = state["batch"]
        b.step(case["steps"])
        return [snapshot(s, z, case["stride"]) for s, z in zip(b.models, state["sizes"])]
    s = state["solver"]
    s.step(case["steps"])
    out = snapshot(s, state["sizes"][0], case["stride"])
    if case["peak"]:
        out["peak"] = s.peak_velocity()
    return out


def seismograms(a):
    """Velocities and stresses apart; at the surface the tractions are zero
    but for rounding, so the in-plane stresses only."""
    return {"velocity": a[:3], "stress": a[[3, 4, 6]]}


def training(case, seed):
    rng = np.random.RandomState(seed % (2 ** 31))
    n = case["ni"]
    x = rng.standard_normal((n, 45)).astype(np.float32)
    x /= np.abs(x).max(axis=1, keepdims=True)
    t = (0.2 * rng.standard_normal((n, 9))).astype(np.float32)
    w = np.concatenate([rng.standard_normal(64 * 45) / math.sqrt(45), 0.1 * rng.standard_normal(64),
                        rng.standard_normal(64 * 64) / 8.0, 0.1 * rng.standard_normal(64),
                        rng.standard_normal(9 * 64) / 8.0, 0.1 * rng.standard_normal(9)])
    return w.astype(np.float16), x, t


def work(case):
    """Least traffic of a pass: each of the four stages reads its input and
    what it combines it with once and writes its result once (117 state
    values per cell and step, 78 auxiliary values per cell and PML
    direction), plus media and metric per stage; about 200 flops per cell and
    stage."""
    if case["kind"] == "train":
        n = case["ni"]
        return {"bytes": 4.0 * n * 54 + 6.0 * 7689, "flops": 6.0 * 7552 * n}
    size = 4 if case["storage"] == "f32" else 2
    total = flops = 0.0
    for ni, nj, nk in sizes_of(case):
        cells = ni * nj * nk
        w = case["pml"]
        pairs = 2 * w * (nj * nk + ni * nk) + w * ni * nj
        media = 16.0 * (3.0 if case["hill"] == 0.0 else 4.6)
        total += case["steps"] * (cells * (117.0 * size + media) + pairs * 78.0 * 4.0)
        flops += case["steps"] * cells * 4 * 200.0
        if case["mlp"]:
            layer = cells - (ni - 8) * (nj - 8) * (nk - 4)
            total += case["steps"] * layer * 18.0 * size
            flops += case["steps"] * layer * 2 * 7552.0
        if case["kind"] == "shot":
            n = (ni + 6) * (nj + 6) * (nk + 6)
            total += n * 44.0 + 9 * 4 * case["receivers"] * case["steps"]
        else:
            s = case["stride"]
            total += 36.0 * (-(-ni // s)) * (-(-nj // s)) * (-(-nk // s))
    return {"bytes": total, "flops": flops}


# --------------------------- the pass in 64 bits ----------------------------

DRP = {-1: -0.30874, 0: -0.6326, 1: 1.2330, 2: -0.3334, 3: 0.04168}
DIRS = [[(1, 1, 1), (-1, -1, -1), (1, 1, 1), (-1, -1, -1)],
        [(1, 1, -1), (-1, -1, 1), (1, 1, -1), (-1, -1, 1)],
        [(-1, -1, -1), (1, 1, 1), (-1, -1, -1), (1, 1, 1)],
        [(-1, -1, 1), (1, 1, -1), (-1, -1, 1), (1, 1, -1)]]
STRESS = [[3, 6, 7], [6, 4, 8], [7, 8, 5]]  # component of sigma_pq


class Exact:
    """The RK4 time stepping of one model in FP64."""

    def __init__(self, m):
        self.m = m
        self.dev = dev = m["metric"][0].device
        self.n = n = m["size"]
        f64 = dict(dtype=torch.float64, device=dev)
        self.zx, self.zy, self.zz, self.jac = m["metric"]
        al, be, rho = [a.double() for a in m["media"]]
        self.irho = self.valid(1.0 / rho).clone()
        mu = rho * be * be
        self.mu = self.valid(mu).clone()
        self.l2m = self.valid(rho * al * al).clone()
        self.lam = self.l2m - 2.0 * self.mu
        self.zp = (self.valid(rho) * self.valid(al)).clone() if m["mlp"] else None
        del al, be, rho, mu
        self.prof = [[torch.as_tensor(p[t][G:-G], **f64) for p in m["pml"]] for t in range(3)]
        self.idx = []
        for ax in range(3):
            lo, hi = m["nabs"][2 * ax], m["nabs"][2 * ax + 1]
            self.idx.append(torch.cat([torch.arange(lo), torch.arange(n[ax] - hi, n[ax])]).to(dev))
        full = [a + 2 * G for a in n]
        self.fw = [torch.zeros(full, **f64) for _ in range(9)]
        for c, f in m["start"].items():
            self.fw[c] += f.double()
        self.aux = {}
        for ax in range(3):
            if len(self.idx[ax]):
                shape = list(n)
                shape[ax] = len(self.idx[ax])
                self.aux[ax] = [torch.zeros(shape, **f64) for _ in range(9)]
        self.surface()
        self.step_no = 0

    def valid(self, a):
        return a[G:-G, G:-G, G:-G]

    def along(self, v, ax):
        s = [1, 1, 1]
        s[ax] = -1
        return v.reshape(s)

    def diff(self, f, ax, sign, taps=DRP):
        out = None
        for d, c in taps.items():
            v = f
            for a in range(3):
                v = v.narrow(a, G + (sign * d if a == ax else 0), self.n[a])
            if out is None:
                out = v * (c * sign / H)
            else:
                out.add_(v, alpha=c * sign / H)
        return out

    def surface(self):
        """Velocity-gradient matrices of the traction-free surface."""
        k = self.n[2] - 1
        l2m, mu = self.l2m[:, :, k], self.mu[:, :, k]
        la = l2m - 2.0 * mu
        one, zero = torch.ones_like(mu), torch.zeros_like(mu)
        e3 = [self.valid(a)[:, :, k] for a in (self.zx, self.zy, self.zz)]
        e = [[one, zero, zero], [zero, one, zero], e3]

        def stiff(p, q):
            r = torch.empty(mu.shape + (3, 3), dtype=torch.float64, device=self.dev)
            for a in range(3):
                for b in range(3):
                    if a == b:
                        v = l2m * p[a] * q[a]
                        for o in range(3):
                            if o != a:
                                v = v + mu * p[o] * q[o]
                    else:
                        v = la * p[a] * q[b] + mu * p[b] * q[a]
                    r[..., a, b] = v
            return r
        inv = torch.linalg.inv(stiff(e[2], e[2]))
        bz = self.prof[1][2][k]
        self.mx = -inv @ stiff(e[2], e[0]) * (bz / self.prof[1][0])[:, None, None, None]
        self.my = -inv @ stiff(e[2], e[1]) * (bz / self.prof[1][1])[None, :, None, None]

    def rhs(self, w, dirs, tindex):
        """Right-hand sides of the nine fields and of the auxiliaries."""
        n, X, Y, Z = self.n, *dirs
        top = n[2] - 1
        kc = self.m["con"] - G
        zz = self.valid(self.zz)
        curved = torch.zeros(n[2], dtype=torch.float64, device=self.dev)
        curved[kc:] = 1.0
        zx, zy = self.valid(self.zx) * curved, self.valid(self.zy) * curved
        b = [self.along(self.prof[1][a], a) for a in range(3)]
        hw, haux = [], {a: [] for a in self.aux}

        def finish(c, parts, extra=None):
            h = 0.0
            for a in range(3):
                if parts[a] is None:
                    parts[a] = torch.zeros(n, dtype=torch.float64, device=self.dev)
                h = h + parts[a] / b[a]
            for a in self.aux:
                ai, ix = self.aux_in[a][c], self.idx[a]
                apd = self.along(self.prof[0][a][ix], a)
                db = self.along(self.prof[2][a][ix], a)
                p = parts[a].index_select(a, ix)
                h.index_add_(a, ix, ai / self.along(self.prof[1][a][ix], a), alpha=-1.0)
                ha = p * db - apd * ai
                if extra is not None and extra[a] is not None:
                    ha[:, :, top] += (db * self.along(self.prof[1][a][ix], a))[:, :, 0] * \
                        extra[a].index_select(a, ix)
                haux[a].append(ha)
            hw.append(h)

        for q in range(3):  # velocities
            t = [w[STRESS[q][p]] for p in range(3)]
            dz = zx * self.diff(t[0], 2, Z) + zy * self.diff(t[1], 2, Z) + zz * self.diff(t[2], 2, Z)
            finish(q, [self.diff(t[0], 0, X) * self.irho, self.diff(t[1], 1, Y) * self.irho,
                       dz * self.irho])
        dv = [[self.diff(w[q], 0, X) for q in range(3)], [self.diff(w[q], 1, Y) for q in range(3)],
              [self.diff(w[q], 2, Z) for q in range(3)]]
        m22 = self.diff_planes(w, Z, {0: -1.0, 1: 1.0}, top - 1)
        m24 = self.diff_planes(w, Z, {0: -7.0 / 6.0, 1: 4.0 / 3.0, 2: -1.0 / 6.0}, top - 2)
        vx = torch.stack([dv[0][q][:, :, top] for q in range(3)], -1)[..., None]
        vy = torch.stack([dv[1][q][:, :, top] for q in range(3)], -1)[..., None]
        fx, fy = (self.mx @ vx)[..., 0], (self.my @ vy)[..., 0]
        for q in range(3):
            dv[2][q][:, :, top] = fx[..., q] + fy[..., q]
            dv[2][q][:, :, top - 1] = m22[q]
            dv[2][q][:, :, top - 2] = m24[q]
        st = (slice(None), slice(None), top)

        def zeta(c, d, at=...):
            l2m, lam, mu = self.l2m[at], self.lam[at], self.mu[at]
            ax, ay, az = zx[at], zy[at], zz[at]
            if c < 6:
                f = [lam, lam, lam]
                f[c - 3] = l2m
                return f[0] * ax * d[0] + f[1] * ay * d[1] + f[2] * az * d[2]
            if c == 6:
                return (ay * d[0] + ax * d[1]) * mu
            return (az * d[0] + ax * d[2]) * mu if c == 7 else (az * d[1] + ay * d[2]) * mu

        def extra(c):
            return [zeta(c, [fx[..., q] for q in range(3)], st),
                    zeta(c, [fy[..., q] for q in range(3)], st), None]
        l2m, lam, mu = self.l2m, self.lam, self.mu
        for c, px, py in ((3, (l2m, 0), (lam, 1)), (4, (lam, 0), (l2m, 1)), (5, (lam, 0), (lam, 1)),
                          (6, (mu, 1), (mu, 0)), (7, (mu, 2), None), (8, None, (mu, 2))):
            finish(c, [px and px[0] * dv[0][px[1]], py and py[0] * dv[1][py[1]],
                       zeta(c, dv[2])], extra(c))
        self.image(w, dirs, hw, haux)
        return hw, haux

    def diff_planes(self, w, Z, taps, k):
        out = []
        for q in range(3):
            f = w[q][G:-G, G:-G]
            out.append(sum(f[:, :, G + k + Z * d] * (c * Z / H) for d, c in taps.items()))
        return out

    def image(self, w, dirs, hw, haux):
        """Velocities of the top three layers by the traction image."""
        n, X, Y, Z = self.n, *dirs
        top = n[2] - 1
        lay = slice(G + top - 2, G + top + 1)  # the three layers, full index
        wx, wy = slice(G, G + n[0]), slice(G, G + n[1])
        bx, by = self.along(self.prof[1][0], 0), self.along(self.prof[1][1], 1)
        for q in range(3):
            t = [w[STRESS[q][p]] for p in range(3)]
            jl = self.jac[:, :, lay]
            ix = self.valid(self.irho_full())[:, :, top - 2:] / self.valid(self.jac)[:, :, top - 2:]
            dx = sum(c * X / H * (jl * t[0][:, :, lay]).narrow(0, G + X * d, n[0])[:, wy]
                     for d, c in DRP.items()) * ix
            dy = sum(c * Y / H * (jl * t[1][:, :, lay]).narrow(1, G + Y * d, n[1])[wx]
                     for d, c in DRP.items()) * ix
            f = self.traction(t, wx, wy, top)
            dz = torch.stack([sum(c * Z / H * f[:, :, 5 + r + Z * d] for d, c in DRP.items())
                              for r in range(-2, 1)], -1) * ix
            h = dx / bx + dy / by + dz
            for a, part in ((0, dx), (1, dy)):
                if a in self.aux:
                    ii = self.idx[a]
                    ai = self.aux_in[a][q][:, :, top - 2:]
                    h.index_add_(a, ii, ai / self.along(self.prof[1][a][ii], a), alpha=-1.0)
                    haux[a][q][:, :, top - 2:] = \
                        part.index_select(a, ii) * self.along(self.prof[2][a][ii], a) \
                        - self.along(self.prof[0][a][ii], a) * ai
            hw[q][:, :, top - 2:] = h

    def irho_full(self):
        return torch.nn.functional.pad(self.irho[None, None], (G,) * 6)[0, 0]

    def traction(self, t, wx, wy, top):
        """J sigma . grad zeta on the layers top-5 .. top, zero on the
        surface, odd above it (planes 0..5 below, 6..8 above)."""
        s = slice(G + top - 5, G + top + 1)
        f = self.jac[wx, wy, s] * (self.zx[wx, wy, s] * t[0][wx, wy, s]
                                   + self.zy[wx, wy, s] * t[1][wx, wy, s]
                                   + self.zz[wx, wy, s] * t[2][wx, wy, s])
        f[:, :, 5] = 0.0
        return torch.cat([f, -torch.flip(f[:, :, 2:5], [2])], -1)

    def sources(self, tindex, time):
        """(component, cell, rate) of every source at a half step."""
        m, out = self.m, []
        top = self.n[2] + G - 1

        def put(kind, loc, vals, weights):
            offs = [((0, 0, 0), 1.0)] if weights is None else \
                [((a - 3, b - 3, c - 3), weights[a, b, c])
                 for a in range(7) for b in range(7) for c in range(7)]
            for o, wt in offs:
                i, j, k = (int(loc[a]) + o[a] for a in range(3))
                if not all(G <= p < self.n[a] + G for a, p in enumerate((i, j, k))):
                    continue
                a = wt / (H ** 3)
                out.append((kind, (i, j, k), a, vals, 2.0 if kind == "force" and k == top else 1.0))
        loc, m6, stf = m["moment"]
        put("moment", loc[0], m6[0].astype(np.float64) * float(stf[0, tindex]),
            m["weights"][0][0] if m["weights"] else None)
        if m["force"]:
            loc, f3, stf = m["force"]
            put("force", loc[0], f3[0].astype(np.float64) * float(stf[0, tindex]),
                m["weights"][1][0] if m["weights"] else None)
        if m["fault"]:
            loc, fdt, mom = m["fault"]
            last = mom.shape[2] - 1
            if 0.0 <= time <= fdt * last:
                p = min(int(time / fdt), last)
                r = min(p + 1, last)
                v = mom[:, :, p] + (mom[:, :, r].astype(np.float64) - mom[:, :, p]) * \
                    (time / fdt - p)
                for q in range(len(loc)):
                    put("moment", loc[q], v[:, q], None)
        return out

    def add_sources(self, hw, tindex, time):
        found = self.sources(tindex, time)
        if not found:
            return
        at = torch.tensor([f[1] for f in found], device=self.dev)
        f64 = dict(dtype=torch.float64, device=self.dev)
        a = torch.tensor([f[2] * f[4] for f in found], **f64) / self.jac[at[:, 0], at[:, 1], at[:, 2]]
        v = at - G
        for kind, comps, sign in (("moment", range(3, 9), -1.0), ("force", range(3), 1.0)):
            sel = [q for q, f in enumerate(found) if f[0] == kind]
            if not sel:
                continue
            s = torch.tensor(sel, device=self.dev)
            vals = torch.tensor(np.array([found[q][3] for q in sel]), **f64)
            i, j, k = v[s, 0], v[s, 1], v[s, 2]
            rate = sign * a[s]
            if kind == "force":
                rate = rate * self.irho[i, j, k]
            for e, c in enumerate(comps):
                hw[c].index_put_((i, j, k), rate * vals[:, e], accumulate=True)

    def step(self):
        a, b = (0.5, 0.5, 1.0), (1 / 6, 1 / 3, 1 / 3, 1 / 6)
        t = self.step_no
        w, self.aux_in = self.fw, self.aux
        tw = [f.clone() for f in self.fw]
        ta = {x: [f.clone() for f in v] for x, v in self.aux.items()}
        for s in range(4):
            tinc = (0, 1, 1, 2)[s]
            hw, haux = self.rhs(w, DIRS[t % 4][s], 2 * t + tinc)
            self.add_sources(hw, 2 * t + tinc, (t + 0.5 * tinc) * DT)
            for c in range(9):
                self.valid(tw[c]).add_(hw[c], alpha=b[s] * DT)
            for x in ta:
                for c in range(9):
                    ta[x][c].add_(haux[x][c], alpha=b[s] * DT)
            if s < 3:
                w = [f.clone() for f in self.fw]
                for c in range(9):
                    self.valid(w[c]).add_(hw[c], alpha=a[s] * DT)
                self.aux_in = {x: [f + a[s] * DT * h for f, h in zip(v, haux[x])]
                               for x, v in self.aux.items()}
            del hw, haux
        self.fw, self.aux = tw, ta
        if self.m["mlp"]:
            self.layer()
        self.step_no += 1

    def layer(self):
        """The learned layer's damping of the new state."""
        width, wts, gains = self.m["mlp"]
        n, nabs = self.n, self.m["nabs"]
        if not hasattr(self, "cells"):
            far = 1 << 30
            r = [torch.arange(x, device=self.dev) for x in n]
            dist = [d if nabs[f] > 0 else torch.full_like(d, far) for f, d in enumerate(
                (r[0], n[0] - 1 - r[0], r[1], n[1] - 1 - r[1], r[2]))]
            best = torch.full(n, width, device=self.dev)
            face = torch.full(n, -1, device=self.dev)
            for f in range(5):
                s = [1, 1, 1]
                s[f // 2] = -1
                d = dist[f].reshape(s).expand(n)
                nearer = d < best
                best = torch.where(nearer, d, best)
                face = torch.where(nearer, torch.full_like(face, f), face)
            self.cells = torch.nonzero(face >= 0)
            f = face[self.cells[:, 0], self.cells[:, 1], self.cells[:, 2]]
            self.depth = best[self.cells[:, 0], self.cells[:, 1], self.cells[:, 2]]
            normal = torch.tensor([(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1)],
                                  device=self.dev)
            self.normal = normal[f]
        wts = torch.as_tensor(wts.astype(np.float64), device=self.dev)
        o = np.cumsum([0, 64 * 45, 64, 64 * 64, 64, 9 * 64, 9])
        W1, b1, W2, b2, W3, b3 = [wts[o[q]:o[q + 1]] for q in range(6)]
        g = torch.as_tensor(gains.astype(np.float64), device=self.dev)
        out = []
        for at in range(0, len(self.cells), 1 << 19):
            c, nm = self.cells[at:at + (1 << 19)], self.normal[at:at + (1 << 19)]
            z = self.zp[c[:, 0], c[:, 1], c[:, 2]]
            x = []
            for s in range(5):
                p = c + G + s * nm
                for q in range(9):
                    v = self.fw[q][p[:, 0], p[:, 1], p[:, 2]]
                    x.append(v / z if q >= 3 else v)
            x = torch.stack(x, 1)
            m = x.abs().amax(1, keepdim=True)
            on = m > 1e-30
            x = torch.where(on, x / torch.where(on, m, torch.ones_like(m)), torch.zeros_like(x))
            h = torch.nn.functional.silu(x @ W1.reshape(64, 45).T + b1)
            h = torch.nn.functional.silu(h @ W2.reshape(64, 64).T + b2)
            y = h @ W3.reshape(9, 64).T + b3
            d = g[self.depth[at:at + (1 << 19)]] * 0.25 * torch.tanh(y / 0.25)
            u = x[:, :9]
            d = torch.minimum(torch.maximum(d, torch.clamp(-u, max=0.0)), torch.clamp(-u, min=0.0))
            d = torch.where(on, d * m, torch.zeros_like(d))
            d[:, 3:] *= z[:, None]
            out.append(d)
        d = torch.cat(out)
        c = self.cells + G
        for q in range(9):
            self.fw[q].index_put_((c[:, 0], c[:, 1], c[:, 2]), d[:, q], accumulate=True)


def exact(case, seed):
    if case["kind"] == "train":
        w, x, t = training(case, seed)
        p = torch.tensor(w.astype(np.float64), requires_grad=True)
        o = np.cumsum([0, 64 * 45, 64, 64 * 64, 64, 9 * 64, 9])
        W1, b1, W2, b2, W3, b3 = [p[o[q]:o[q + 1]] for q in range(6)]
        silu = torch.nn.functional.silu
        h = silu(torch.tensor(x).double() @ W1.reshape(64, 45).T + b1)
        h = silu(h @ W2.reshape(64, 64).T + b2)
        e = h @ W3.reshape(9, 64).T + b3 - torch.tensor(t).double()
        loss = (e * e).sum() / len(x)
        loss.backward()
        return {"loss": float(loss.detach()), "gradient": p.grad.numpy()}
    out = []
    with torch.no_grad():
        for q, size in enumerate(sizes_of(case)):
            m = build(case, size, seed if case["models"] == 1 else seed * 16 + q)
            e = Exact(m)
            top = m["size"][2] + G - 1
            peak = torch.zeros((3,) + tuple(size[:2]), dtype=torch.float64, device=e.dev)
            trace = []
            rc = torch.as_tensor(m["receivers"].astype(np.int64), device=e.dev)
            for _ in range(case["steps"]):
                e.step()
                if case["peak"]:
                    for c in range(3):
                        v = e.fw[c][G:-G, G:-G, top].abs()
                        peak[c] = torch.maximum(peak[c], v)
                if case["kind"] == "shot":
                    trace.append(torch.stack([f[rc[:, 0], rc[:, 1], rc[:, 2]] for f in e.fw]))
            if case["kind"] == "shot":
                r = seismograms(torch.stack(trace, -1).cpu().numpy())
            else:
                s = case["stride"]
                f = [e.valid(a)[::s, ::s, ::s].cpu().numpy() for a in e.fw]
                r = {"velocity": np.stack(f[:3]), "stress": np.stack(f[3:])}
            if case["peak"]:
                r["peak"] = peak.cpu().numpy()
            del e, m
            out.append(r)
    return out if case["models"] > 1 else out[0]
