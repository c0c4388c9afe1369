"""What users of the framework have it do, as cases that can be timed and checked.

A case is a dict of plain values; `kind` says which public entry point it goes
through:

  run       engine.Simulation: set_m, run(seconds) with the adaptive RK45DP, get_m
  steps     engine.Simulation: set_m, steps(n) with a fixed dt and any stepper, get_m
  demag     opencl.NewNewellDemag(...).Exec: one demag field
  stage     the device-op layer as the reference's engine drives it: the terms of
            the effective field one call each, torque, Madd2, Normalize, reductions
  adjoint   adjoint.AdjointRK4: forward and backward
  ensemble  engine.Ensemble: set_m of every instance, run(seconds), get_m

`exact` restates each of them in 64 bits with torch alone: the demag tensor
(Newell, Williams and Dunlop 1993 near the source cell, Gauss quadrature of the
dipole kernel over both cells away from it), the local terms, the torque, the
steppers and the step controller.
"""
import math

import numpy as np
import torch

from umagnus_b200 import adjoint, config, engine, opencl

MU0 = 4e-7 * math.pi
GAMMA = 1.7595e11  # rad / (T s)
SOLVERS = {"heun": 2, "rk23": 3, "rk4": 4, "rk45": 5}
STAGES = {"heun": 2, "rk23": 3, "rk4": 4, "rk45": 6}


def listed():
    return [
        # the small permalloy film of the plain method: every launch counts
        dict(name="film_64x64x1", kind="run", nx=64, ny=64, nz=1, cell="4,4,3", ms=8e5, aex=1.3e-11, alpha=0.1,
             bz=0.01, steps=120),
        # standard problem 4 (500 x 125 x 3 nm) with 2.5 nm cells: sizes that are no powers of two
        dict(name="strip_200x50x1", kind="run", nx=200, ny=50, nz=1, cell="2.5,2.5,3", ms=8e5, aex=1.3e-11,
             alpha=0.02, bx=-0.0246, by=0.0043, steps=60),
        # a vortex disc: geometry in a square mesh
        dict(name="disc_250x250x1", kind="steps", nx=250, ny=250, nz=1, cell="4,4,10", ms=8e5, aex=1.3e-11,
             alpha=0.05, geom=True, bx=0.005, solver="rk45", steps=24),
        # a skyrmion track, periodic along x, with interfacial DMI; Heun as for runs at finite temperature
        dict(name="track_512x64x1_periodic", kind="steps", nx=512, ny=64, nz=1, cell="2,2,1", ms=5.8e5, aex=1.5e-11,
             alpha=0.3, dind=3e-3, ku=8e5, bz=0.02, pbcx=2, solver="heun", steps=64),
        # a thick element with per-cell anisotropy: three dimensions, sizes that are no powers of two
        dict(name="box_100x60x20", kind="steps", nx=100, ny=60, nz=20, cell="3,3,3", ms=1.4e6, aex=2.1e-11,
             alpha=0.05, ku=4e4, kumap=True, solver="rk4", steps=16),
        # the multilayer with interfacial DMI and anisotropy: the headline workload
        dict(name="multilayer_256x256x16", kind="run", nx=256, ny=256, nz=16, cell="2,2,1", ms=1.1e6, aex=1.6e-11,
             alpha=0.3, dind=3e-3, ku=5e5, bz=0.05, steps=24),
        # polycrystal of 64 Voronoi grains: region maps, per-cell maps; the largest
        dict(name="grains_512x512x32", kind="steps", nx=512, ny=512, nz=32, cell="2,2,2", ms=6e5, aex=1.0e-11,
             alpha=0.05, ku=2e5, kumap=True, grains=64, solver="rk45", steps=3),
        # one demag field of a ragged body through the device-op layer: the smallest call
        dict(name="demag_75x45x9", kind="demag", nx=75, ny=45, nz=9, cell="5,5,4", ms=8e5),
        # one demag field of a large film
        dict(name="demag_1024x1024x1", kind="demag", nx=1024, ny=1024, nz=1, cell="4,4,4", ms=8e5),
        # a stepper stage driven call by call, with regions
        dict(name="stage_256x256x4", kind="stage", nx=256, ny=256, nz=4, cell="2,2,2", ms=1.1e6, aex=1.6e-11,
             alpha=0.1, dind=2e-3, ku=5e5, bz=0.05, grains=16),
        # gradients through fixed-step RK4
        dict(name="adjoint_128x128x1", kind="adjoint", nx=128, ny=128, nz=1, cell="4,4,4", ms=6e5, aex=1.3e-11,
             alpha=0.02, ku=2e5, bx=0.005, by=0.005, steps=60, every=20),
        # a parameter sweep of small films, batched
        dict(name="ensemble_48_films", kind="ensemble", count=48, sizes="32,48,64,96,128", cell="4,4,3", steps=64),
    ]


# ------------------------------------------------------------------ more cases of the same ranges
def _smooth(n):
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def _size(rng, lo, hi, even=False):
    """A mesh size spread over the logarithm of the range; prime factors up to 13, which every path takes."""
    while True:
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if _smooth(n) and not (even and n % 2):
            return n


def draw(rng):
    kind = rng.choice(["run", "steps", "steps", "steps", "demag", "demag", "stage", "adjoint", "ensemble"])
    mat = dict(ms=round(rng.uniform(4e5, 1.5e6), -3), aex=round(rng.uniform(0.8, 2.2), 2) * 1e-11,
               alpha=round(rng.uniform(0.02, 0.4), 3), bz=round(rng.uniform(-0.1, 0.1), 3))
    if kind == "ensemble":
        ks = rng.sample([32, 48, 64, 96, 128], rng.randint(2, 4))
        return dict(kind=kind, count=rng.randint(6, 40), sizes=",".join(map(str, sorted(ks))), cell="4,4,3",
                    steps=rng.randint(32, 64))
    flat = rng.random() < 0.5
    cell = ",".join("%g" % rng.choice([2, 2.5, 3, 4]) for _ in range(2)) + ",%g" % rng.choice([1, 2, 3, 4])
    case = dict(kind=kind, nx=_size(rng, 24, 640), ny=_size(rng, 16, 512), nz=1 if flat else _size(rng, 2, 24),
                cell=cell, **mat)
    while case["nx"] * case["ny"] * case["nz"] > 1 << 20 or (case["nx"] + 1) * case["nz"] > 20000:
        case["nx"], case["ny"] = _size(rng, 24, 640), _size(rng, 16, 512)
    big = case["nx"] * case["ny"] * case["nz"]
    if kind in ("run", "steps"):
        case["steps"] = max(3, min(60, (1 << 21) // big))
    if kind == "steps":
        case["solver"] = rng.choice(list(SOLVERS))
        opt = rng.choice(["none", "geom", "pbc", "grains", "dmi"])
        if opt == "geom":
            case["geom"] = True
        elif opt == "pbc":
            case["nx"], case["pbcx"] = _size(rng, 24, 320, even=True), 1
        elif opt == "grains":
            case["grains"] = rng.randint(2, 100)
        if opt in ("dmi", "pbc"):
            case["dind"] = round(rng.uniform(0.5, 3), 1) * 1e-3
        if rng.random() < 0.5:
            case["ku"], case["kumap"] = round(rng.uniform(0.1, 8), 2) * 1e5, rng.random() < 0.5
    elif kind == "stage":
        case.update(dind=round(rng.uniform(0.5, 3), 1) * 1e-3, ku=round(rng.uniform(0.1, 8), 2) * 1e5,
                    grains=rng.randint(1, 60))
    elif kind == "adjoint":
        n = rng.choice([48, 64, 96, 128])
        case.update(nx=n, ny=rng.choice([32, 64, n]), nz=1, ku=2e5, steps=rng.randint(20, 50), every=rng.randint(5, 25))
    return case


# ------------------------------------------------------------------ inputs
def _cell(case):
    return tuple(float(v) * 1e-9 for v in case["cell"].split(","))


def _mesh(case):
    return case["nx"], case["ny"], case["nz"]


def _unit(m):
    n = m.norm(dim=0, keepdim=True)
    return torch.where(n > 0, m / n.clamp_min(1e-30), m)


def _random_m(shape, seed):
    """Random unit vectors, the usual seeded start."""
    g = torch.Generator("cuda").manual_seed(seed)
    return _unit(torch.randn((3,) + tuple(shape), generator=g, device="cuda", dtype=torch.float32))


def _inputs(case, seed):
    """The arrays of one simulation: m0 on the device, maps as numpy arrays (what Simulation takes)."""
    nx, ny, nz = _mesh(case)
    rng = np.random.default_rng(seed)
    d = dict(m0=_random_m((nz, ny, nx), seed), geom=None, regions=None, ms=case["ms"], aex=case.get("aex"),
             ku=case.get("ku", 0.0), axis=(0.0, 0.0, 1.0))
    if case.get("geom"):
        c = _cell(case)
        d["geom"] = config.ellipse((nx, ny, nz), c, nx * c[0], ny * c[1])
    grains = case.get("grains", 0)
    if grains:  # columnar Voronoi grains, each of one of two materials
        px, py = rng.uniform(0, nx, grains), rng.uniform(0, ny, grains)
        y, x = torch.meshgrid(torch.arange(ny, device="cuda"), torch.arange(nx, device="cuda"), indexing="ij")
        best = torch.full((ny, nx), float("inf"), device="cuda")
        reg = torch.zeros((ny, nx), dtype=torch.uint8, device="cuda")
        for g in range(grains):
            r2 = (x - px[g]) ** 2 + (y - py[g]) ** 2
            reg = torch.where(r2 < best, torch.full_like(reg, g), reg)
            best = torch.minimum(best, r2)
        reg = reg.cpu().numpy()
        cls = rng.integers(0, 2, grains)
        d["regions"] = np.ascontiguousarray(np.broadcast_to(reg, (nz, ny, nx)))
        d["ms"] = np.where(cls[d["regions"]] == 1, np.float32(1.5 * case["ms"]), np.float32(case["ms"]))
        d["aex"] = np.zeros(256, np.float32)
        d["aex"][:grains] = np.where(cls == 1, 1.5 * case["aex"], case["aex"])
        d["aex"][grains:] = case["aex"]
        if case.get("kumap"):  # a random easy axis per grain
            u = rng.standard_normal((3, grains))
            u = (u / np.sqrt((u * u).sum(0))).astype(np.float32)
            d["axis"] = np.ascontiguousarray(u[:, d["regions"]])
    elif case.get("kumap"):
        d["ku"] = (case["ku"] * rng.uniform(0.8, 1.2, (nz, ny, nx))).astype(np.float32)
    return d


def _b_ext(case):
    return case.get("bx", 0.0), case.get("by", 0.0), case.get("bz", 0.0)


def _fix_dt(case):
    """A time step that resolves the exchange field of a random state (0.1 rad of its largest precession)."""
    c = _cell(case)
    b = 8 * case["aex"] / case["ms"] * sum(1 / v ** 2 for v, n in zip(c, _mesh(case)) if n > 1)
    return 0.1 / (GAMMA * (b + MU0 * case["ms"] + 2 * case.get("ku", 0.0) / case["ms"] + 0.05))


def _seconds(case):
    """What the adaptive stepper covers in about case["steps"] steps."""
    return case["steps"] * 6 * _fix_dt(case)


def _ens_instances(case, seed):
    """Films of the listed sizes with parameters drawn per instance (the sizes belong to the case, not the seed)."""
    rng = np.random.default_rng(seed)
    sizes = [int(v) for v in case["sizes"].split(",")]
    out = []
    for i in range(case["count"]):
        n = sizes[i % len(sizes)]
        d = rng.standard_normal(3)
        b = d / np.linalg.norm(d) * rng.uniform(0, 0.1)
        out.append(dict(N=(n, n, 1), cell=_cell(case), Msat=float(rng.uniform(4e5, 1.2e6)),
                        Aex=float(rng.uniform(5e-12, 2e-11)), alpha=float(rng.uniform(0.05, 0.5)),
                        B_ext=tuple(float(v) for v in b)))
    return out


def _ens_seconds(case):
    return case["steps"] * 1.7e-13


def _adj_probe(case):
    return case["nx"] // 2 - 8, case["ny"] // 2 - 8, 16, 16


def _adj_inputs(case, seed):
    nx, ny, nz = _mesh(case)
    g = torch.Generator("cuda").manual_seed(seed)
    m0 = 0.3 * torch.randn((3, nz, ny, nx), generator=g, device="cuda")
    m0[0] += 1.0
    ms = case["ms"] * (1 + 0.5 * torch.rand((nz, ny, nx), generator=g, device="cuda"))
    t = np.random.default_rng(seed).standard_normal(3)
    return _unit(m0), ms, tuple(float(v) for v in t / np.linalg.norm(t))


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    k = case["kind"]
    s = dict(case=case)
    if k in ("run", "steps"):
        d = _inputs(case, seed)
        fix = _fix_dt(case) if k == "steps" else 0.0
        s["m0"] = d["m0"]
        s["sim"] = engine.Simulation(_mesh(case), _cell(case), d["ms"], d["aex"], case["alpha"],
                                     Dind=case.get("dind", 0.0), Ku1=d["ku"], anisU=d["axis"], B_ext=_b_ext(case),
                                     regions=d["regions"], geom=d["geom"], pbc=(case.get("pbcx", 0), 0, 0),
                                     solver=SOLVERS[case.get("solver", "rk45")], FixDt=fix)
        s["out"] = torch.empty_like(d["m0"])
    elif k == "demag":
        s["m0"] = _random_m(_mesh(case)[::-1], seed)
        s["plan"] = opencl.NewNewellDemag(_mesh(case), (0, 0, 0), _cell(case))
        s["B"] = torch.empty_like(s["m0"])
    elif k == "stage":
        d = _inputs(case, seed)
        s["m0"] = d["m0"]
        s["mesh"] = opencl.Mesh(_mesh(case), _cell(case))
        s["plan"] = opencl.NewNewellDemag(_mesh(case), (0, 0, 0), _cell(case))
        s["regions"] = torch.from_numpy(d["regions"]).cuda()
        s["ms"] = opencl.MSlice(torch.from_numpy(d["ms"]).cuda())
        s["alut"] = torch.from_numpy(engine.exchange_lut(d["aex"])).cuda()
        s["dlut"] = torch.from_numpy(engine.exchange_lut(case["dind"])).cuda()
        s["blut"] = torch.tensor(_b_ext(case), device="cuda").reshape(3, 1).repeat(1, 256).contiguous()
        s["B"], s["tau"], s["m1"] = (torch.empty_like(s["m0"]) for _ in range(3))
    elif k == "adjoint":
        m0, ms, target = _adj_inputs(case, seed)
        s.update(m0=m0, ms=ms)
        s["sim"] = adjoint.AdjointRK4(_mesh(case), _cell(case), case["alpha"], (1.0, 0.0, 0.0), 1e-13, case["steps"],
                                      case["every"], _adj_probe(case), max(1, case["steps"] // 2), target=target)
    else:
        inst = _ens_instances(case, seed)
        s["sim"] = engine.Ensemble(inst)
        s["m0"] = [_random_m((1, d["N"][1], d["N"][0]), seed * 1000 + i).cpu().numpy() for i, d in enumerate(inst)]
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k in ("run", "steps"):
        sim = s["sim"]
        sim.set_m(s["m0"])
        if k == "run":
            sim.set_time(0.0, 1e-15)
            sim.run(_seconds(case))
        else:
            sim.steps(case["steps"])
        return {"m": sim.get_m(s["out"])}
    if k == "demag":
        s["plan"].Exec(s["B"], s["m0"], None, case["ms"])
        return {"B": s["B"]}
    if k == "stage":
        m, B, tau, m1 = s["m0"], s["B"], s["tau"], s["m1"]
        s["plan"].Exec(B, m, None, s["ms"])
        opencl.AddDMI(B, m, s["alut"], s["dlut"], s["ms"], s["regions"], s["mesh"])
        opencl.AddUniaxialAnisotropy2(B, m, s["ms"], case["ku"], 0.0, (0.0, 0.0, 1.0))
        opencl.RegionAddV(B, s["blut"], s["regions"])
        opencl.LLTorque(tau, m, B, case["alpha"])
        opencl.Madd2(m1, m, tau, 1.0, _fix_dt(case) * GAMMA)
        opencl.Normalize(m1)
        return {"B": B, "tau": tau, "m": m1, "max_torque": opencl.MaxVecNorm(tau), "mean_mz": opencl.Sum(m1[2]),
                "max_change": opencl.MaxVecDiff(m1, m)}
    if k == "adjoint":
        sim = s["sim"]
        loss = sim.forward(s["m0"], s["ms"], case["aex"], case["ku"], _b_ext(case))
        return {"loss": loss, "m": sim.final_m(), "grad": sim.backward()}
    sim = s["sim"]
    for i, m in enumerate(s["m0"]):
        sim.set_m(i, m)
    sim.run(_ens_seconds(case))
    return [sim.get_m(i) for i in range(len(sim))]


# ------------------------------------------------------------------ work and tolerance
def _pad(n):
    return 2 * n if n > 5 else 2 * n - 1


def _eval_work(case):
    """One effective field and torque: m read and the torque written, the demag kernel's spectrum read, the
    half spectrum of three components written and read once (the rows and planes of zero padding left out)."""
    nx, ny, nz = _mesh(case)
    n = nx * ny * nz
    px = nx if case.get("pbcx") else 2 * nx
    py, pz = 2 * ny, _pad(nz) if nz > 1 else 1
    hx = px // 2 + 1
    kern = hx * (py // 2 + 1) * (pz // 2 + 1) * (6 if nz > 1 else 4)
    spec = hx * ny * pz * 3
    lines = 2 * 2.5 * (nz * ny * px * math.log2(max(2, px)) + 2 * hx * ny * pz * math.log2(max(2, pz)) +
                       2 * hx * py * pz * math.log2(max(2, py))) * 3
    maps = 4 * n * (2 + (3 if case.get("kumap") else 0)) + n if case.get("grains") else 0
    return dict(bytes=24 * n + 4 * kern + 16 * spec + maps, flops=lines + 30 * hx * py * pz + 150 * n)


def work(case):
    k = case["kind"]
    if k == "ensemble":
        sizes = [int(v) for v in case["sizes"].split(",")]
        tot = dict(bytes=0.0, flops=0.0)
        for i in range(case["count"]):
            n = sizes[i % len(sizes)]
            w = _eval_work(dict(nx=n, ny=n, nz=1))
            for key in tot:
                tot[key] += 6 * case["steps"] * (w[key] + (80 * n * n if key == "bytes" else 60 * n * n))
        return tot
    nx, ny, nz = _mesh(case)
    n = nx * ny * nz
    w = _eval_work(case)
    if k == "demag":
        return dict(bytes=w["bytes"], flops=w["flops"])
    if k == "stage":  # every term reads and writes the field
        return dict(bytes=w["bytes"] + n * (37 + 36 + 25 + 36 + 36 + 24 + 12 + 4 + 24), flops=w["flops"])
    evals = case["steps"] * STAGES.get(case.get("solver", "rk45"), 6)
    if k == "adjoint":  # forward, recomputation and reverse
        evals = 3 * 4 * case["steps"]
    return dict(bytes=evals * (w["bytes"] + 80.0 * n), flops=evals * (w["flops"] + 60.0 * n))


def tolerance(case):
    """About four times the largest error against `exact` seen over the ranges: one field evaluation in 32 bits is
    2e-7 off, fixed steps up to 8e-7, an adaptive run (whose dt follows the rounding of its error estimate, and whose
    random start spreads rounding differences) up to 5e-6."""
    return {"rel": {"demag": 1e-6, "stage": 2e-6, "steps": 4e-6, "run": 2e-5, "ensemble": 2e-5,
                    "adjoint": 1e-5}[case["kind"]]}


# ------------------------------------------------------------------ 64 bits: the demag tensor
def _newell_f(x, y, z):
    x, y, z = x.abs(), y.abs(), z.abs()
    x2, y2, z2 = x * x, y * y, z * z
    r = (x2 + y2 + z2).sqrt()
    t = (2 * x2 - y2 - z2) * r / 6
    a = torch.asinh(y / (x2 + z2).sqrt().clamp_min(1e-300))
    b = torch.asinh(z / (x2 + y2).sqrt().clamp_min(1e-300))
    t = t + torch.where(x2 + z2 > 0, 0.5 * y * (z2 - x2) * a, 0.0)
    t = t + torch.where(x2 + y2 > 0, 0.5 * z * (y2 - x2) * b, 0.0)
    return t - torch.where(x * r > 0, x * y * z * torch.atan(y * z / (x * r).clamp_min(1e-300)), 0.0)


def _newell_g(x, y, z):
    x2, y2, z2 = x * x, y * y, z * z
    r = (x2 + y2 + z2).sqrt()

    def ash(p, q2):
        return torch.where(q2 > 0, torch.asinh(p / q2.sqrt().clamp_min(1e-300)), 0.0)

    def atn(p, q):
        return torch.where(q != 0, torch.atan(p / torch.where(q == 0, 1.0, q)), 0.0)

    t = x * y * z * ash(z, x2 + y2) + y / 6 * (3 * z2 - y2) * ash(x, y2 + z2) + x / 6 * (3 * z2 - x2) * ash(y, x2 + z2)
    t = t - z * z2 / 6 * atn(x * y, z * r) - z * y2 / 2 * atn(x * z, y * r) - z * x2 / 2 * atn(y * z, x * r)
    return t - x * y * r / 3


def _near(i, j, k, d):
    """Minus the demag tensor (xx yy zz yz xz xy) between cells i, j, k apart: Newell's second differences."""
    dx, dy, dz = d
    acc = [torch.zeros_like(i) for _ in range(6)]
    for a in (-1, 0, 1):
        for b in (-1, 0, 1):
            for c in (-1, 0, 1):
                w = (2 if a == 0 else -1) * (2 if b == 0 else -1) * (2 if c == 0 else -1)
                x, y, z = (i + a) * dx, (j + b) * dy, (k + c) * dz
                for n, v in enumerate((_newell_f(x, y, z), _newell_f(y, x, z), _newell_f(z, y, x),
                                       _newell_g(y, z, x), _newell_g(x, z, y), _newell_g(x, y, z))):
                    acc[n] += w * v
    return [-v / (4 * math.pi * dx * dy * dz) for v in acc]


def _far(i, j, k, d):
    """The same by Gauss quadrature of the dipole kernel over the offsets between points of the two cells (eight
    points an axis over the triangular weight), for cells at least eight cell sizes apart."""
    u, w = np.polynomial.legendre.leggauss(4)
    u, w = 0.5 * (u + 1), 0.5 * w
    pts = [(s * a, b * (1 - a)) for s in (-1.0, 1.0) for a, b in zip(u, w)]
    acc = [torch.zeros_like(i) for _ in range(6)]
    vol = d[0] * d[1] * d[2] / (4 * math.pi)
    for a, wa in pts:
        x = (i + a) * d[0]
        for b, wb in pts:
            y = (j + b) * d[1]
            for c, wc in pts:
                z = (k + c) * d[2]
                r2 = x * x + y * y + z * z
                q = (wa * wb * wc * vol) / (r2 * r2 * r2.sqrt())
                for n, v in enumerate((3 * x * x - r2, 3 * y * y - r2, 3 * z * z - r2, 3 * y * z, 3 * x * z, 3 * x * y)):
                    acc[n].addcmul_(v, q)
    return acc


def _kernel_spectrum(mesh, cell, pbc):
    pad = [n if p else (_pad(n) if ax == 2 else 2 * n) for ax, (n, p) in enumerate(zip(mesh, pbc))]
    s = max(cell)
    d = [c / s for c in cell]
    K = [torch.zeros(pad[::-1], dtype=torch.float64, device="cuda") for _ in range(6)]
    idx, off = [], []
    for ax in range(3):
        o = torch.arange(-(pad[ax] * pbc[ax] - 1) if pbc[ax] else 1 - mesh[ax], pad[ax] * pbc[ax] if pbc[ax] else mesh[ax],
                         device="cuda")
        off.append(o.double())
        idx.append(o % pad[ax])
    for z0 in range(0, len(off[2]), 8):  # in slabs, for the memory's sake
        k, j, i = torch.meshgrid(off[2][z0:z0 + 8], off[1], off[0], indexing="ij")
        T = _far(i, j, k, d)
        close = (i * d[0]) ** 2 + (j * d[1]) ** 2 + (k * d[2]) ** 2 <= 8.5 ** 2
        N = _near(i[close], j[close], k[close], d)
        at = (idx[2][z0:z0 + 8][:, None, None], idx[1][None, :, None], idx[0][None, None, :])
        for c in range(6):
            T[c][close] = N[c]
            K[c].index_put_(at, T[c], accumulate=True)
    return pad, [torch.fft.rfftn(v) for v in K]


class _Demag:
    def __init__(self, mesh, cell, pbc=(0, 0, 0)):
        self.mesh = mesh
        self.pad, self.K = _kernel_spectrum(mesh, cell, pbc)

    def __call__(self, M):
        """The field (T) of the magnetisation M (3, nz, ny, nx) in A/m times mu0."""
        P = self.pad[::-1]
        xx, yy, zz, yz, xz, xy = self.K
        F = [torch.fft.rfftn(M[c], s=P) for c in range(3)]
        H = (xx * F[0] + xy * F[1] + xz * F[2], xy * F[0] + yy * F[1] + yz * F[2], xz * F[0] + yz * F[1] + zz * F[2])
        nx, ny, nz = self.mesh
        return torch.stack([torch.fft.irfftn(h, s=P)[:nz, :ny, :nx] for h in H])


# ------------------------------------------------------------------ 64 bits: field, torque, steppers
def _f64(v):
    return float(np.float32(v))


class _Model:
    """The effective field and torque of one simulation. Maps broadcast against (nz, ny, nx)."""

    def __init__(self, mesh, cell, ms, alpha, a_pair, dind=0.0, ku=0.0, axis=(0, 0, 1), b=(0, 0, 0), vol=None,
                 pbcx=0, demag=None):
        self.cell, self.ms, self.alpha, self.a_pair = cell, ms, alpha, a_pair
        self.dind, self.ku, self.b, self.vol, self.pbcx, self.mesh = dind, ku, b, vol, pbcx, mesh
        self.u = [torch.as_tensor(v, dtype=torch.float64, device="cuda") for v in axis]
        self.demag = demag or _Demag(mesh, cell, (pbcx, 0, 0))

    def _shift(self, t, ax, side, wrap):
        """The neighbour of every cell along axis ax (0 x, 1 y, 2 z) of a (..., nz, ny, nx) array, and which exist."""
        dim = t.dim() - 1 - ax
        n = t.shape[dim]
        r = torch.roll(t, -side, dim)
        there = torch.ones(n, dtype=torch.bool, device=t.device)
        if not wrap:
            there[n - 1 if side > 0 else 0] = False
        shape = [1] * t.dim()
        shape[dim] = n
        return r, there.reshape(shape)

    def exchange(self, m):
        h = torch.zeros_like(m)
        full = (m * m).sum(0, keepdim=True) > 0
        for ax in range(3 if self.mesh[2] > 1 else 2):
            c = self.cell[ax]
            for side in (-1, 1):
                wrap = ax == 0 and self.pbcx
                mn, there = self._shift(m, ax, side, wrap)
                there = there & ((mn * mn).sum(0, keepdim=True) > 0)
                A, D = self.a_pair(ax, side), self.dind
                if torch.is_tensor(A) and A.dim():  # a missing neighbour counts with the cell's own material
                    A = torch.where(there[0], A, self.a_pair(ax, 0))
                if D and ax < 2:  # interfacial DMI: a missing neighbour takes the value the boundary condition gives
                    q = side * c * 0.5 * D / A
                    o = torch.zeros_like(m[0])
                    ext = torch.stack([m[0] - q * m[2] if ax == 0 else m[0], m[1] if ax == 0 else m[1] - q * m[2],
                                       m[2] + q * m[ax]])
                    mn = torch.where(there, mn, ext)
                    dm = [o, o, -side * mn[ax]]
                    dm[ax] = side * mn[2]
                    h = h + D / c * torch.stack(dm)
                else:
                    mn = torch.where(there, mn, m)
                h = h + 2 * A / c ** 2 * (mn - m)
        return torch.where(full, h, 0.0) / self.ms

    def field(self, m):
        B = self.demag(MU0 * self.ms * (m if self.vol is None else m * self.vol)) + self.exchange(m)
        if torch.is_tensor(self.ku) or self.ku:
            mu = sum(m[c] * self.u[c] for c in range(3))
            B = B + torch.stack([2 * self.ku / self.ms * mu * self.u[c] for c in range(3)])
        b = self.b if torch.is_tensor(self.b) else torch.tensor(self.b, dtype=torch.float64, device="cuda")
        return B + b.reshape(3, 1, 1, 1)

    def torque_of(self, m, B):
        mb = torch.linalg.cross(m, B, dim=0)
        return -(mb + self.alpha * torch.linalg.cross(m, mb, dim=0)) / (1 + self.alpha ** 2)

    def torque(self, m):
        return self.torque_of(m, self.field(m))

    def norm(self, m):
        return _unit(m) if self.vol is None else torch.where(self.vol > 0, _unit(m), 0.0)

    # one step of each stepper: (new m, error vector or None, last torque)
    def step(self, solver, m, h, k1=None):
        f, n = self.torque, self.norm
        if solver == "heun":
            k1 = f(m)
            y = m + h * k1
            return n(y + 0.5 * h * (f(y) - k1)), None, None
        if solver == "rk4":
            k1 = f(m)
            k2 = f(n(m + 0.5 * h * k1))
            k3 = f(n(m + 0.5 * h * k2))
            k4 = f(n(m + h * k3))
            return n(m + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)), None, None
        k1 = f(m) if k1 is None else k1
        if solver == "rk23":
            k2 = f(n(m + 0.5 * h * k1))
            k3 = f(n(m + 0.75 * h * k2))
            y = n(m + h * (2 / 9 * k1 + 1 / 3 * k2 + 4 / 9 * k3))
            return y, None, f(y)
        k2 = f(n(m + h / 5 * k1))
        k3 = f(n(m + h * (3 / 40 * k1 + 9 / 40 * k2)))
        k4 = f(n(m + h * (44 / 45 * k1 - 56 / 15 * k2 + 32 / 9 * k3)))
        k5 = f(n(m + h * (19372 / 6561 * k1 - 25360 / 2187 * k2 + 64448 / 6561 * k3 - 212 / 729 * k4)))
        k6 = f(n(m + h * (9017 / 3168 * k1 - 355 / 33 * k2 + 46732 / 5247 * k3 + 49 / 176 * k4 - 5103 / 18656 * k5)))
        y = n(m + h * (35 / 384 * k1 + 500 / 1113 * k3 + 125 / 192 * k4 - 2187 / 6784 * k5 + 11 / 84 * k6))
        k7 = f(y)
        err = (71 / 57600 * k1 - 71 / 16695 * k3 + 71 / 1920 * k4 - 17253 / 339200 * k5 + 22 / 525 * k6 - 1 / 40 * k7)
        return y, err, k7

    def fixed(self, solver, m, dt, steps):
        k = None
        for _ in range(steps):
            m, _, k = self.step(solver, m, dt * GAMMA, k)
        return m

    def adaptive(self, m, dt, seconds, max_err=1e-5):
        """RK45DP with the step controller's defaults: headroom 0.8, dt changed by 1/2 to 2, the last step cut to end
        at `seconds` (the relative criterion only counts above a torque that no sample reaches)."""
        t, k1 = 0.0, self.torque(m)
        while t < seconds:
            h = dt * GAMMA
            y, e, k7 = self.step("rk45", m, h, k1)
            err = float(e.norm(dim=0).max()) * h
            if err < max_err:
                t, m, k1, corr = t + dt, y, k7, (max_err / err) ** (1 / 5)
            else:
                corr = (max_err / err) ** (1 / 6)
            dt *= min(2.0, max(0.5, 0.8 * corr))
            if t < seconds and t + dt > seconds:
                dt = seconds - t
        return m


def _model(case, d):
    """The 64-bit model of a case's inputs."""
    mesh, cell = _mesh(case), _cell(case)
    t64 = lambda v: torch.as_tensor(np.asarray(v, np.float32), device="cuda").double()  # noqa: E731
    ms = t64(d["ms"]) if np.ndim(d["ms"]) else _f64(d["ms"])
    if d["regions"] is None:
        a = _f64(d["aex"])
        pair = lambda ax, side: a  # noqa: E731
    else:
        A = t64(d["aex"])[torch.from_numpy(d["regions"]).cuda().long()]

        def pair(ax, side):
            return 2 / (1 / A + 1 / torch.roll(A, -side, 2 - ax))
    ku = t64(d["ku"]) if np.ndim(d["ku"]) else _f64(d["ku"])
    axis = [t64(v) for v in d["axis"]]
    vol = None if d["geom"] is None else t64(d["geom"])
    return _Model(mesh, cell, ms, _f64(case["alpha"]), pair, _f64(case.get("dind", 0.0)), ku, axis,
                  [_f64(v) for v in _b_ext(case)], vol, case.get("pbcx", 0))


@torch.no_grad()
def _exact_plain(case, seed):
    k = case["kind"]
    if k == "ensemble":
        out, demag = [], {}
        for i, d in enumerate(_ens_instances(case, seed)):
            if i >= 10:  # two of every listed size; the rest would take minutes
                out.append(None)
                continue
            if d["N"] not in demag:
                demag[d["N"]] = _Demag(d["N"], d["cell"])
            a = _f64(d["Aex"])
            M = _Model(d["N"], d["cell"], _f64(d["Msat"]), _f64(d["alpha"]), lambda ax, side: a,
                       b=[_f64(v) for v in d["B_ext"]], demag=demag[d["N"]])
            m = M.norm(_random_m((1, d["N"][1], d["N"][0]), seed * 1000 + i).double())
            out.append(M.adaptive(m, 1e-15, _ens_seconds(case)))
        return out
    d = _inputs(case, seed) if k != "demag" else None
    if k == "demag":
        m = _random_m(_mesh(case)[::-1], seed).double()
        return {"B": _Demag(_mesh(case), _cell(case))(MU0 * _f64(case["ms"]) * m)}
    M = _model(case, d)
    if k == "stage":
        m = d["m0"].double()
        B = M.field(m)
        tau = M.torque_of(m, B)
        m1 = M.norm(m + _f64(_fix_dt(case) * GAMMA) * tau)
        return {"B": B, "tau": tau, "m": m1, "max_torque": float(tau.norm(dim=0).max()), "mean_mz": float(m1[2].sum()),
                "max_change": float((m1 - m).norm(dim=0).max())}
    m = M.norm(d["m0"].double())
    if k == "steps":
        return {"m": M.fixed(case["solver"], m, _fix_dt(case), case["steps"])}
    return {"m": M.adaptive(m, 1e-15, _seconds(case))}


def exact(case, seed):
    if case["kind"] != "adjoint":
        return _exact_plain(case, seed)
    m0, ms, target = _adj_inputs(case, seed)
    leaf = lambda v: torch.as_tensor(v, dtype=torch.float64, device="cuda").clone().requires_grad_(True)  # noqa: E731
    m0, ms, a, ku = leaf(m0), leaf(ms), leaf(_f64(case["aex"])), leaf(_f64(case["ku"]))
    b = leaf([_f64(v) for v in _b_ext(case)])
    M = _Model(_mesh(case), _cell(case), ms, _f64(case["alpha"]), lambda ax, side: a, 0.0, ku, (1.0, 0.0, 0.0), b)
    x, y, w, h = _adj_probe(case)
    first = max(1, case["steps"] // 2)
    m, probe = M.norm(m0), 0.0
    for n in range(1, case["steps"] + 1):
        m = M.step("rk4", m, 1e-13 * GAMMA)[0]
        if n >= first:
            probe = probe + m[2, 0, y:y + h, x:x + w].mean()
    avg = m.mean(dim=(1, 2, 3))
    t = torch.tensor(target, dtype=torch.float64, device="cuda")
    loss = probe / (case["steps"] - first + 1) + ((avg - t) ** 2).sum()
    loss.backward()
    return {"loss": float(loss), "m": m.detach(),
            "grad": {"Ms": ms.grad, "Aex": float(a.grad), "Ku1": float(ku.grad), "B_ext": [float(v) for v in b.grad],
                     "m0": m0.grad}}
