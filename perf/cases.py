"""The work that a user of this framework has it do, as measurable cases.

A simulation run is: the constants set, the host particle SoA and its cohesion
uploaded, the cell sort, some substeps, the particles (and, where the program
draws, the animation-frame records) read back. A calibration run is: the force
history forward, the reverse sweep, the gradients read back. Both go through
the package's public entry points (MPMHandle, indenter_force_history).

Inputs are states as they are in the middle of a run: a jittered lattice (or a
lattice with loose grains above it, or an ice block in a water tank) with a
smooth velocity field, small elastic strain and, around the indenter, points
that have crushed already.

exact() restates the substep in plain torch, in 64 bits, from the published
MLS-MPM equations and the material model; it shares no code with the package.
"""
import dataclasses
import math

import numpy as np
import torch

CRUSHED, LIQUID = 0x10000, 0x40000
STRENGTH = dict(compressive=100e6, tensile=10e6, shear=6e6, tensile2=5e6)
COHESION = 3.0e5
GRAVITY, WATER_DENSITY, POISSON, PHI_DEG, RADIUS, PAD = 9.81, 1000.0, 0.3, 62.0, 0.05, 3


# ------------------------------------------------------------------ the cases

def _case(name, kind="run", n=250_000, precision="mixed", scene="block", steps=100, **more):
    """One case; the fields that `more` does not name take these values."""
    c = dict(name=name, kind=kind, n=n, precision=precision, scene=scene, steps=steps,
             h=0.01, dt=5e-6,
             ppc=2.0,             # particles per cell
             aspect=2.0,          # block length over its height and width
             halo=0,              # GridHaloSize
             velocity=1.0,        # indenter, m/s
             depth=0,             # cells that the indenter is inside the block at the start
             cohesion=True,       # per-particle cohesion (lognormal), else the uniform threshold
             grain_var=0.0,       # GrainVariability
             accum="float",       # the mixed form's grid sums
             api="step",          # "step" (mpm_step) or "phases" (reset, P2G, update, G2P by the caller)
             shuffled=False,      # points in the order of a mesh file, not of space
             pinned=True,         # page-locked host buffers
             frame=False,         # a full animation frame at the end
             ckpt=10)             # substeps between checkpoints (gradients)
    c.update(more)
    return c


def listed():
    return [
        # the smallest calls (a unit of a parameter study, a test): latency and launches
        _case("small_4k_fp64", n=4_000, precision="fp64", steps=20, dt=1e-5, velocity=0.2, cohesion=False, pinned=False),
        # an odd size with halo slabs and grain-dependent strengths, as the shipped configurations have them
        _case("odd_3001_mixed", n=3_001, steps=40, halo=3, grain_var=0.5, cohesion=False, pinned=False),
        # a host program that drives the phases itself, as the reference's step loop does
        _case("phases_50k_fp64", n=50_000, precision="fp64", steps=20, dt=1e-5, ppc=1.0, cohesion=False, api="phases"),
        # the indentation block at about one particle per cell, with a frame for the viewer
        _case("block250k_mixed", n=250_000, steps=100, dt=1e-5, ppc=1.0, velocity=0.2, cohesion=False, frame=True),
        # the default precision at scale, per-particle cohesion
        _case("block2m_fp64", n=2_000_000, precision="fp64", steps=60, h=0.0125, velocity=0.5),
        # the largest: the 8 M block over a stretch of substeps
        _case("block8m_mixed", n=8_000_000, steps=200, aspect=4.0),
        # non-uniform density: a block with loose grains above it, odd size
        _case("grains3m_mixed", n=3_000_017, scene="grains", steps=100, h=0.008, dt=2e-6, velocity=2.0, aspect=4.0),
        # the indenter deep in the ice: a crushed zone that takes the return map at every substep
        _case("crush500k_mixed", n=500_000, steps=100, dt=1e-5, velocity=2.0, depth=3),
        # an ice block in a water tank, points in mesh order: liquid points, no indenter
        _case("tank1m_mixed", n=1_000_003, scene="tank", steps=60, cohesion=False, shuffled=True),
        # runs that have to repeat bit for bit: order-independent grid sums
        _case("fixed1m_mixed", n=1_000_000, steps=40, accum="fixed"),
        # a gradient for calibrating the ice strength: FP64, a handle that the program keeps
        _case("gradient100k_fp64", kind="gradient", n=100_000, precision="svd64", steps=40, dt=1e-5, velocity=2.0, depth=3),
        # the same through torch.autograd with the mixed forward, one evaluation of an optimiser
        _case("gradient20k_mixed", kind="autograd", n=20_000, precision="mixed", steps=40, dt=1e-5, velocity=2.0, depth=3,
              ckpt=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | rng.randint(0, 1)


def draw(rng):
    kind = rng.choice(["run"] * 7 + ["gradient", "gradient", "autograd"])
    c = _case("", kind=kind)
    del c["name"]
    c["aspect"] = rng.choice([1.0, 2.0, 3.3, 4.0])
    c["halo"] = rng.choice([0, 0, 3, 15])
    c["cohesion"] = rng.random() < 0.6
    if kind != "run":
        c["n"] = _log_int(rng, 2_000, 150_000)
        c["precision"] = rng.choice(["svd64", "mixed"])
        c["ckpt"] = rng.randint(5, 20)
        c["steps"] = rng.randint(10, 45)
        c["dt"], c["depth"], c["velocity"] = 1e-5, rng.choice([2, 3]), rng.choice([1.0, 2.0])
        c["halo"] = rng.choice([0, 3])
        return c
    c["precision"] = rng.choice(["mixed"] * 4 + ["fp64"] * 3 + ["svd64"])
    c["accum"] = "fixed" if c["precision"] == "mixed" and rng.random() < 0.2 else "float"
    c["scene"] = rng.choice(["block"] * 4 + ["grains", "tank"])
    c["n"] = _log_int(rng, 2_000, 4_000_000 if c["precision"] == "mixed" and c["accum"] == "float" else 1_500_000)
    c["steps"] = rng.randint(10, 100)
    c["ppc"] = rng.choice([1.0, 2.0, 2.0, 4.0, 8.0])
    c["grain_var"] = rng.choice([0.0, 0.0, 0.5])
    c["velocity"] = rng.choice([0.2, 0.5, 1.0, 2.0])
    c["depth"] = rng.choice([0, 0, 3])
    c["api"] = rng.choice(["step"] * 4 + ["phases"])
    c["shuffled"] = rng.random() < 0.3
    c["frame"] = rng.random() < 0.2
    c["pinned"] = c["n"] > 100_000
    return c


# ------------------------------------------------- geometry and constants

def _geometry(c):
    """Block size, grid and indenter of a case, as the package's loader places them."""
    h, n, ppc = c["h"], c["n"], c["ppc"]
    a = c["aspect"]
    if c["scene"] == "grains":
        n_lat = n - int(round(0.3 * n))
        s = (n_lat / ppc * h ** 3 / (a * 0.4)) ** (1.0 / 3.0)     # domain a*s x s x s, lattice in its lower 40 %
        dom = (a * s, s, s)
        lat = (a * s, 0.4 * s, s)
    else:
        n_lat = n
        s = (n / ppc * h ** 3 / a) ** (1.0 / 3.0)
        dom = lat = (a * s, s, s)
    nb = [int(math.ceil(d / h - 1e-9)) for d in dom]
    clear = int(math.ceil(RADIUS / h)) + 2
    g = (nb[0] + 2 * (PAD + clear), nb[1] + 2 + PAD + 3, nb[2] + 2 * PAD + 2)
    off = ((g[0] * h - dom[0]) / 2, 2 * h, (g[2] * h - dom[2]) / 2)
    ind_x = math.floor((off[0] - RADIUS) / h) * h + c["depth"] * h
    return dict(n_lat=n_lat, dom=dom, lat=lat, grid=g, off=off, ind=(ind_x, off[1] + lat[1]))


def _points(c, seed):
    """The particles on the GPU, in 64 bits: x (3, n), v, F (n, 3, 3), C, Jp_inv, status, cohesion."""
    geo = _geometry(c)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 7919 + 13)
    f8 = dict(dtype=torch.float64, device=dev)
    n, h, n_lat, lat = c["n"], c["h"], geo["n_lat"], geo["lat"]

    def rand(*s):
        return torch.rand(*s, generator=gen, **f8)

    def randn(*s):
        return torch.randn(*s, generator=gen, **f8)

    sp = (lat[0] * lat[1] * lat[2] / n_lat) ** (1.0 / 3.0)
    cnt = [max(1, int(math.ceil(d / sp - 1e-9))) for d in lat]
    total = cnt[0] * cnt[1] * cnt[2]
    site = torch.arange(total, device=dev)
    if total > n_lat:
        site = torch.randperm(total, generator=gen, device=dev)[:n_lat].sort().values
    x = torch.empty((3, n), **f8)
    ijk = (site // (cnt[1] * cnt[2]), (site // cnt[2]) % cnt[1], site % cnt[2])
    for d in range(3):
        x[d, :n_lat] = (ijk[d] + 0.5 + 0.3 * (2 * rand(n_lat) - 1)) * (lat[d] / cnt[d]) + geo["off"][d]
    if n > n_lat:
        grains = max(1, n // 1500)
        lo = torch.tensor([geo["off"][0], geo["off"][1] + lat[1], geo["off"][2]], **f8)
        hi = torch.tensor([geo["off"][d] + geo["dom"][d] for d in range(3)], **f8)
        rad = (2.5 + 5.0 * rand(grains)) * h
        rad = torch.minimum(rad, 0.45 * (hi - lo).min())
        centre = lo[:, None] + rad + (hi - lo)[:, None] * rand(3, grains) * (1 - 2 * rad / (hi - lo)[:, None])
        own = torch.multinomial(rad ** 3, n - n_lat, replacement=True, generator=gen)
        own = own.sort().values
        dirs = randn(3, n - n_lat)
        dirs /= dirs.norm(dim=0).clamp_min(1e-300)
        x[:, n_lat:] = centre[:, own] + dirs * rad[own] * rand(n - n_lat) ** (1.0 / 3.0)
    L = geo["dom"][0]
    ph = 2 * math.pi * rand(6)
    k = 2 * math.pi / L
    v = torch.stack([0.1 * torch.sin(k * x[0] + ph[0]), 0.05 * torch.sin(k * x[1] + ph[1]) - 0.02,
                     0.05 * torch.cos(k * x[2] + ph[2])])
    F = 2e-5 * randn(n, 9)
    wave = 2e-4 * torch.sin(k * (x[0] + x[1]) + ph[3])
    for d in range(3):
        F[:, 4 * d] += 1.0 + wave * (1.0 if d else -1.5)
    C = 0.5 * randn(n, 9)
    status = torch.randint(0, 4000, (n,), generator=gen, device=dev) if c["grain_var"] else torch.zeros(n, dtype=torch.int64, device=dev)
    Jp = torch.ones(n, **f8)
    if c["scene"] == "tank":
        cut = [0.4 * d for d in geo["dom"]]
        ctr = [geo["off"][0] + geo["dom"][0] / 2, geo["off"][1] + geo["dom"][1] - cut[1] / 2, geo["off"][2] + geo["dom"][2] / 2]
        out = torch.zeros(n, dtype=torch.bool, device=dev)
        for d in range(3):
            out |= (x[d] - ctr[d]).abs() > cut[d] / 2
        status = torch.where(out, status | LIQUID, status)
        Jp = torch.where(out, 1.0 + 1e-5 * randn(n), Jp)
    else:
        r2 = (x[0] - geo["ind"][0]) ** 2 + (x[1] - geo["ind"][1]) ** 2
        near = (r2 < (RADIUS + 4 * h) ** 2) & (rand(n) < 0.8)
        status = torch.where(near, status | CRUSHED, status)
        Jp = torch.where(near, 1.0 + (2e-3 * randn(n)).abs(), Jp)
        F = torch.where(near[:, None], F + 1e-3 * randn(n, 9), F)
    coh = COHESION * torch.exp(0.3 * randn(n)) if c["cohesion"] else None
    if c["shuffled"]:
        p = torch.randperm(n, generator=gen, device=dev)
        x, v, F, C, Jp, status = x[:, p], v[:, p], F[p], C[p], Jp[p], status[p]
        coh = coh[p] if coh is not None else None
    return geo, dict(x=x, v=v, F=F.reshape(n, 3, 3), C=C.reshape(n, 3, 3), Jp=Jp, status=status, cohesion=coh)


def _volume(c):
    return c["h"] ** 3 / c["ppc"]


# ------------------------------------------------------------ prepare and run

def _params(c, geo):
    from icempm_3dm_b200 import generator as g
    from icempm_3dm_b200._lib import LIB
    cfg = g.BlockConfig("case", c["n"], geo["dom"], c["h"], 0, c["dt"], c["steps"], c["velocity"],
                        cohesion_median=COHESION, phi_deg=PHI_DEG, poisson=POISSON, ind_radius=RADIUS, pad=PAD, halo=c["halo"])
    if c["scene"] == "tank":
        cfg = dataclasses.replace(cfg, youngs=1e8, density=200.0)
    p = g.make_params(cfg)
    assert (p.GridXTotal, p.GridY, p.GridZ) == geo["grid"]
    p.GrainVariability = c["grain_var"]
    if c["scene"] == "tank":
        p.SetupType, p.DragGlobal = 2, 2e-3
    p.Volume = _volume(c) * c["n"]
    p.ParticleVolume = _volume(c)
    p.indenter_x = p.indenter_x_initial = geo["ind"][0]
    p.indenter_y = p.indenter_y_initial = geo["ind"][1]
    LIB.mpm_params_compute_helper_variables(p)
    return p


def _to_soa(pts, rows):
    """Fills the (28, n) rows of the host SoA."""
    t = torch.from_numpy(rows)
    t[0].copy_(pts["status"].view(torch.float64))
    t[1:3].zero_()
    t[3].copy_(pts["Jp"])
    t[4:7].copy_(pts["x"])
    t[7:10].copy_(pts["v"])
    n = rows.shape[1]
    t[10:19].copy_(pts["F"].reshape(n, 9).t())
    t[19:28].copy_(pts["C"].reshape(n, 9).t())


def prepare(case, seed):
    from icempm_3dm_b200 import MPMHandle
    from icempm_3dm_b200.layout import ACCUM_FIXED, PRECISION_FP64, PRECISION_FP64_SVD64, PRECISION_MIXED
    from icempm_3dm_b200.simulation import pinned_empty
    c = case
    geo, pts = _points(c, seed)
    prms = _params(c, geo)
    n = c["n"]
    prec = {"fp64": PRECISION_FP64, "svd64": PRECISION_FP64_SVD64, "mixed": PRECISION_MIXED}[c["precision"]]
    new = (lambda s: pinned_empty(s)) if c["pinned"] else (lambda s: np.zeros(s))
    soa = new((28, n))
    _to_soa(pts, soa)
    s = dict(case=c, prms=prms, soa=soa, prec=prec, cohesion=None)
    if c["cohesion"]:
        s["cohesion"] = new((n,))
        torch.from_numpy(s["cohesion"]).copy_(pts["cohesion"])
    if c["kind"] != "run":
        # the loss: a weighted sum of the force history, weights of either sign
        s["weights"] = _weights(c, seed)
        if s["cohesion"] is None:
            s["cohesion"] = np.full(n, COHESION)
    if c["kind"] != "autograd":
        s["handle"] = MPMHandle(prms, n, prec)
        if c["accum"] == "fixed":
            s["handle"].set_grid_accumulation(ACCUM_FIXED)
        s["out"] = new((28, n))
    else:
        s["state"] = torch.from_numpy(soa)
        s["coh_t"] = torch.from_numpy(s["cohesion"])
    return s


def _weights(c, seed):
    return np.random.default_rng(int(seed) + 5).standard_normal((c["steps"], 3)) * 1e-3


def _views(out):
    return dict(status=out[0].view(np.int64), P=out[1], Q=out[2], Jp=out[3], x=out[4:7], v=out[7:10], F=out[10:19], C=out[19:28])


def run(state):
    s, c = state, state["case"]
    if c["kind"] == "autograd":
        from icempm_3dm_b200.autograd import indenter_force_history
        st = s["state"].requires_grad_(True)
        co = s["coh_t"].requires_grad_(True)
        E = torch.tensor(float(s["prms"].YoungsModulus), dtype=torch.float64, requires_grad=True)
        hist = indenter_force_history(st, co, E, s["prms"], c["steps"], c["ckpt"], precision=s["prec"])
        g = torch.autograd.grad((hist * torch.from_numpy(s["weights"])).sum(), (st, co, E))
        return dict(hist=hist.detach(), x=g[0][4:7], v=g[0][7:10], C=g[0][19:28], F=g[0][10:19], Jp=g[0][3], cohesion=g[1], E=g[2])
    h = s["handle"]
    h.update_constants(s["prms"])
    if c["kind"] == "gradient":
        h.upload(s["soa"], cohesion=s["cohesion"])
        hist = h.adjoint_forward(c["steps"], c["ckpt"])
        dc, dE = h.adjoint_backward(s["weights"])
        a = h.adjoint_state()
        return dict(hist=hist, x=a[0:3], v=a[3:6], C=a[6:15], F=a[15:24], Jp=a[24], cohesion=dc, E=dE)
    h.reset_indenter_force_accumulator()
    h.upload(s["soa"], cohesion=s["cohesion"])
    h.sort()
    got = {}
    if c["api"] == "phases":
        p = s["prms"]
        for k in range(c["steps"]):
            h.reset_grid()
            h.p2g()
            h.update_nodes(p.indenter_x_initial + (k + 1) * p.InitialTimeStep * p.IndVelocity, p.indenter_y)
            h.g2p(k == 0)
        got["sensor"], got["total"] = h.sensors()
    else:
        got["hist"] = h.step(c["steps"])
    got.update(_views(h.download(out=s["out"])))
    if c["frame"]:
        f = h.frame_records(1, True)
        got["frame"] = {name: f[name] for name in f.dtype.names}
    return got


# ------------------------------------------------------------------ the scale

def work(case):
    """Host SoA in and out once, the sort's read and write once; each substep the state
    that it must carry (position, F, Jp_inv, status; velocity and C follow from the grid)
    read and written once and the touched nodes' mass and momentum and velocity written
    and read once."""
    c = case
    n, word = c["n"], 4 if c["precision"] == "mixed" else 8
    nodes = n / c["ppc"]
    per_step = n * 14 * 2 * word + nodes * 4 * 2 * 2 * word
    flops = n * 1500.0
    if c["kind"] != "run":
        # forward and recompute; the reverse step reads the state and its adjoint and writes the adjoint
        return {"bytes": n * 8.0 * (28 + 25) + c["steps"] * (2 * per_step + n * 8.0 * (28 + 25 * 2) + nodes * 8 * 14),
                "flops": c["steps"] * n * 5000.0}
    return {"bytes": n * 8.0 * 28 * 4 + c["steps"] * per_step, "flops": c["steps"] * flops}


def tolerance(case):
    """Measured on one B200, largest over the outputs (C, a velocity difference over h):
    the same inputs twice, float against fixed-point grid sums, and against exact().
    mixed: 1e-5 against exact(), 8e-6 between two orders of the sums; where a contact or
    floor switch meets two values that differ by rounding, 3.2e-3 at the indenter and 3.3e-4
    in the tank. fp64 (whose return map uses a 32-bit SVD, as the reference does): 4e-12
    between two runs, and 2.4e-3 where that SVD takes another branch for a crushed point.
    svd64: 8e-12. Gradients: 2e-11, dL/dE (a sum that cancels) 5e-8; mixed forward 7e-6."""
    c = case
    if c["kind"] != "run":
        return {"rel": 2e-4 if c["precision"] == "mixed" else 2e-7}
    if c["precision"] == "svd64":
        return {"rel": 1e-9, "differ": 1e-5}
    return {"rel": 2e-3 if c["scene"] == "tank" else 1e-2, "differ": 1e-4}


# -------------------------------------------------------- the step in 64 bits

def _constants(c, geo):
    tank = c["scene"] == "tank"
    E = 1e8 if tank else 5e8
    rho = 200.0 if tank else 917.0
    vol, h, dt = _volume(c), geo["grid"][0] * c["h"] / geo["grid"][0], c["dt"]
    phi = math.tan(PHI_DEG * math.pi / 180.0)
    return dict(E=E, mass=vol * rho, liquid_mass=vol * WATER_DENSITY, kdt=dt * vol * 4.0 / (h * h), h=h, hi=1.0 / h, dt=dt,
                vmax=0.5 * h / dt, tan_phi=phi, p0=COHESION / phi, drag=2e-3 if tank else 0.0, tank=tank)


def _moduli(E):
    mu = E / (2 * (1 + POISSON))
    return mu, mu * 2.0 / 3.0 + E * POISSON / ((1 + POISSON) * (1 - 2 * POISSON))


def _det(A):
    return (A[:, 0, 0] * (A[:, 1, 1] * A[:, 2, 2] - A[:, 1, 2] * A[:, 2, 1])
            - A[:, 0, 1] * (A[:, 1, 0] * A[:, 2, 2] - A[:, 1, 2] * A[:, 2, 0])
            + A[:, 0, 2] * (A[:, 1, 0] * A[:, 2, 1] - A[:, 1, 1] * A[:, 2, 0]))


def _inv(A):
    r = [A[:, i] for i in range(3)]
    adj = torch.stack([torch.linalg.cross(r[1], r[2]), torch.linalg.cross(r[2], r[0]), torch.linalg.cross(r[0], r[1])], dim=2)
    return adj / _det(A)[:, None, None]


def _roots(b):
    """b^(1/2) and b^(-1/2) of symmetric positive 3x3 matrices near I (Denman-Beavers)."""
    Y, Z = b, torch.eye(3, dtype=b.dtype, device=b.device).expand_as(b)
    for _ in range(8):
        Y, Z = 0.5 * (Y + _inv(Z)), 0.5 * (Z + _inv(Y))
    return Y, Z


def _deviator(F):
    b = F @ F.transpose(1, 2)
    mean = (b[:, 0, 0] + b[:, 1, 1] + b[:, 2, 2]) / 3
    eye = torch.eye(3, dtype=F.dtype, device=F.device)
    return b, mean, b - mean[:, None, None] * eye, eye


def _stencil(x, g, k):
    base = (x * k["hi"] - 0.5).detach().to(torch.int64)
    fx = x * k["hi"] - base.double()
    w = torch.stack([0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1) ** 2, 0.5 * (fx - 0.5) ** 2])   # (3 offsets, 3 axes, n)
    node = ((base[0] + g["halo"]) * g["gy"] + base[1]) * g["gz"] + base[2]
    for a in range(3):
        for b in range(3):
            for e in range(3):
                off = torch.tensor([a, b, e], dtype=x.dtype, device=x.device)
                yield node + (a * g["gy"] + b) * g["gz"] + e, w[a, 0] * w[b, 1] * w[e, 2], (off[:, None] - fx) * k["h"]


def _return_map(F, Jp, p0, mu, kappa, k):
    """Crushed points: projection of the trial state on the yield surface."""
    S = STRENGTH
    J = _det(F)
    b, mean, dev, eye = _deviator(F)
    p = -0.5 * kappa * (J * J - 1)
    nrm2 = (dev * dev).sum((1, 2))
    nrm = torch.where(nrm2 > 0, nrm2, torch.ones_like(nrm2)).sqrt() * (nrm2 > 0)
    q = math.sqrt(1.5) * mu * J ** (-2.0 / 3.0) * nrm
    _, isq = _roots(b)
    R = isq @ F
    apex = (p < -p0) | (Jp < 1)
    Je = (2 * p0 / kappa + 1).sqrt()
    inside = (S["compressive"] - p) * (p + S["tensile"])
    q_fs = 2 * torch.where(inside > 0, inside, torch.ones_like(inside)).sqrt() * S["shear"] / (S["compressive"] + S["tensile"])
    q_dp = (p + p0) * k["tan_phi"]
    q1 = torch.where(p > S["compressive"], torch.zeros_like(q_dp), torch.where(q_fs <= q_dp, q_fs, q_dp))
    coef = q1 * math.sqrt(2.0 / 3.0) * J ** (2.0 / 3.0) / mu
    dirn = dev / torch.where(nrm > 0, nrm, torch.ones_like(nrm))[:, None, None]
    sq, _ = _roots(torch.where(apex[:, None, None], b, coef[:, None, None] * dirn + mean[:, None, None] * eye))
    yields = ~apex & (q >= q1)
    Fn = torch.where(apex[:, None, None], Je[:, None, None] ** (1.0 / 3.0) * R, torch.where(yields[:, None, None], sq @ R, F))
    return Fn, torch.where(apex, Jp * Je / J, Jp)


def _outside(p, q, status, c):
    S, gv = STRENGTH, c["grain_var"]
    grain = status & 0xffff
    v2 = 1.0 + gv * 0.033 * (-15 + (grain + 3) % 30).double()
    v3 = 1.0 + gv * 0.1 * (-10 + (grain + 4) % 11).double()
    pmax, pmin, beta = S["compressive"], -S["tensile"], S["tensile"] / S["compressive"]
    qmax, pmin2 = S["shear"] * v3, -S["tensile2"] * v2
    q0 = 2 * math.sqrt(-pmax * pmin) * qmax / (pmax - pmin)
    neg = (p < pmin2) | (q > -q0 / pmin2 * (p - pmin2))
    msq = 4 * qmax * qmax * (1 + 2 * beta) / (pmax - pmin) ** 2
    return torch.where(p < 0, neg, (1 + 2 * beta) * q * q + msq * (p + beta * pmax) * (p - pmax) > 0)


def _substep(s, g, k, c, mu, kappa, ind_x, ind_y):
    """One substep; the state s in and out, the force on the indenter, trial p and q."""
    x, v, F, C, Jp, status = s["x"], s["v"], s["F"], s["C"], s["Jp"], s["status"]
    p0 = s["p0"]
    f8 = dict(dtype=x.dtype, device=x.device)
    liquid = (status & LIQUID) != 0
    mass = torch.where(liquid, torch.full_like(Jp, k["liquid_mass"]), torch.full_like(Jp, k["mass"]))
    J = _det(F)
    b, mean, dev, eye = _deviator(F)
    tau = (mu * J ** (-2.0 / 3.0))[:, None, None] * dev + (0.5 * kappa * (J * J - 1))[:, None, None] * eye
    if bool(liquid.any()):
        tau = torch.where(liquid[:, None, None], (kappa * (1 - Jp ** -3.0))[:, None, None] * eye, tau)
    S = mass[:, None, None] * C - k["kdt"] * tau
    grid = torch.zeros((g["nodes"], 4), **f8)
    for node, w, d in _stencil(x, g, k):
        mom = w * (mass * v + (S @ d.t()[:, :, None])[:, :, 0].t())
        grid = grid.index_add(0, node, torch.cat([(w * mass)[None], mom]).t())
    act = (grid[:, 0] != 0).nonzero()[:, 0]
    ga = grid[act]
    m = ga[:, 0]
    u = ga[:, 1:] / m[:, None]
    u = u - torch.tensor([0.0, k["dt"] * GRAVITY, 0.0], **f8)
    sp = (u * u).sum(1)
    fast = sp > k["vmax"] ** 2
    if bool(fast.any()):
        u = torch.where(fast[:, None], u / sp.sqrt()[:, None] * k["vmax"], u)
    gz = act % g["gz"]
    gy = (act // g["gz"]) % g["gy"]
    gx = act // (g["gz"] * g["gy"]) - g["halo"]
    force = torch.zeros(3, **f8)
    if not k["tank"]:
        n0, n1 = gx.double() * k["h"] - ind_x, gy.double() * k["h"] - ind_y
        r2 = n0 * n0 + n1 * n1
        r = torch.where(r2 > 0, r2, torch.ones_like(r2)).sqrt()
        nx, ny = n0 / r, n1 / r
        vn = (u[:, 0] - c["velocity"]) * nx + u[:, 1] * ny
        hit = ((r2 < RADIUS ** 2) & (vn < 0)).nonzero()[:, 0]
        dv = torch.stack([nx[hit] * vn[hit], ny[hit] * vn[hit], torch.zeros_like(vn[hit])], 1)
        force = (dv * m[hit, None] / k["dt"]).sum(0)
        u = u.index_add(0, hit, -dv)
        keep = (gy > 2)[:, None].expand(-1, 3).clone()
    else:
        keep = torch.ones((act.numel(), 3), dtype=torch.bool, device=x.device)
        keep[:, 1] &= ~((gy <= 2) & (u[:, 1] < 0))
    keep[:, 1] &= ~((gy >= g["gy"] - 3) & (u[:, 1] > 0))
    keep[:, 0] &= ~((gx <= 2) & (u[:, 0] < 0)) & ~((gx > 2) & (gx >= g["gx"] - 3) & (u[:, 0] > 0))
    keep[:, 2] &= ~((gz <= 2) & (u[:, 2] < 0)) & ~((gz > 2) & (gz >= g["gz"] - 3) & (u[:, 2] > 0))
    u = torch.where(keep, u, torch.zeros_like(u)) * (1 - k["drag"])
    vel = torch.zeros((g["nodes"], 3), **f8).index_copy(0, act, u)
    nv = torch.zeros_like(v)
    nC = torch.zeros_like(C)
    for node, w, d in _stencil(x, g, k):
        gv = (w[:, None] * vel[node])
        nv = nv + gv.t()
        nC = nC + gv[:, :, None] * d.t()[:, None, :]
    nC = nC * (4.0 * k["hi"] * k["hi"])
    A = eye + k["dt"] * nC
    Ft = A @ F
    Jt = _det(Ft)
    _, _, dev, _ = _deviator(Ft)
    zero = torch.zeros_like(Jt)
    with torch.no_grad():
        p = torch.where(liquid, zero, -0.5 * kappa * (Jt * Jt - 1))
        q = torch.where(liquid, zero, math.sqrt(1.5) * mu * Jt ** (-2.0 / 3.0) * (dev * dev).sum((1, 2)).sqrt())
        status = torch.where(~liquid & _outside(p, q, status, c), status | CRUSHED, status)
        idx = (((status & CRUSHED) != 0) & ~liquid).nonzero()[:, 0]
    nJp = torch.where(liquid, Jp * _det(A), Jp)
    if idx.numel():
        Fr, Jr = _return_map(Ft[idx], nJp[idx], p0[idx], mu, kappa, k)
        Ft = Ft.index_copy(0, idx, Fr)
        nJp = nJp.index_copy(0, idx, Jr)
    return dict(x=x + k["dt"] * nv, v=nv, F=Ft, C=nC, Jp=nJp, status=status, p0=p0), force, p, q


def exact(case, seed):
    c = case
    cost = c["n"] * c["steps"]
    if cost > (4_500_000 if c["kind"] != "run" else 400_000_000):
        return None
    geo, pts = _points(c, seed)
    k = _constants(c, geo)
    gx, gy, gz = geo["grid"]
    g = dict(gx=gx, gy=gy, gz=gz, halo=c["halo"], nodes=(gx + 2 * c["halo"]) * gy * gz)
    n = c["n"]
    dev = pts["x"].device
    if c["kind"] == "run":
        # the stable cell sort (the mixed form holds positions in 2^-20 cells)
        t = pts["x"] * k["hi"]
        if c["precision"] == "mixed":
            t = torch.round(t * 2.0 ** 20) * 2.0 ** -20 * k["h"] * k["hi"]
        i = (t + 0.5).to(torch.int64)
        order = torch.sort((i[0] * gy + i[1]) * gz + i[2], stable=True).indices
        for f in ("x", "v"):
            pts[f] = pts[f][:, order]
        for f in ("F", "C", "Jp", "status"):
            pts[f] = pts[f][order]
        if pts["cohesion"] is not None:
            pts["cohesion"] = pts["cohesion"][order]
    coh = pts["cohesion"]
    if coh is None:
        coh = torch.full((n,), COHESION, dtype=torch.float64, device=dev)
    grad = c["kind"] != "run"
    E = torch.tensor(k["E"], dtype=torch.float64, device=dev, requires_grad=grad)
    leaf = [pts[f].clone().requires_grad_(grad) for f in ("x", "v", "C", "F", "Jp")]
    coh = coh.clone().requires_grad_(grad)
    s = dict(zip(("x", "v", "C", "F", "Jp"), leaf), status=pts["status"], p0=coh / k["tan_phi"])
    ind_y = geo["ind"][1]
    hist, P, Q = [], None, None
    with torch.set_grad_enabled(grad):
        mu, kappa = _moduli(E)
        for j in range(c["steps"]):
            args = (g, k, c, mu, kappa, geo["ind"][0] + (j + 1) * k["dt"] * c["velocity"], ind_y)
            s, f, p, q = _substep(s, *args)
            hist.append(f)
            if j == 0:
                P, Q = p, q
        hist = torch.stack(hist)
        if grad:
            w = torch.from_numpy(_weights(c, seed)).to(dev)
            d = torch.autograd.grad((hist * w).sum(), leaf + [coh, E], allow_unused=True)
            d = [torch.zeros_like(t) if u is None else u for t, u in zip(leaf + [coh, E], d)]
            rows = lambda t: t.reshape(n, 9).t()  # noqa: E731
            return dict(hist=hist.detach(), x=d[0], v=d[1], C=rows(d[2]), F=rows(d[3]), Jp=d[4], cohesion=d[5], E=d[6])
    rows = lambda t: t.reshape(n, 9).t()  # noqa: E731
    got = dict(status=s["status"], P=P, Q=Q, Jp=s["Jp"], x=s["x"], v=s["v"], F=rows(s["F"]), C=rows(s["C"]))
    if c["api"] == "phases":
        every = int(1.0 / (200 * c["dt"]))
        got["sensor"], got["total"] = None, hist.sum(0) / every
    else:
        got["hist"] = hist
    if c["frame"]:
        got["frame"] = dict(zip(("px", "py", "pz", "vx", "vy", "vz"), torch.cat([s["x"], s["v"]])), Jp_inv=s["Jp"],
                            status=((s["status"] & CRUSHED) != 0).to(torch.uint8) * 0x80)
    return got
