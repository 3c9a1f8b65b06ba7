"""The solves that programs run with this framework, as cases that can be timed
and compared: lid-driven and heated cavities in their storage forms, spheres
carried through a channel, the D2Q9 cavity and circles, and the solve server.

A pass of a one-solve case is what a driver does between two looks at its
flow: step(n) and the macroscopic fields (with the residual, the Nusselt
numbers or the particle states where a driver reads them).  A pass of the
server submits a batch of requests and takes their fields.

Fields come back in the precision that the form computes in: FP64 for the
FP64 and FX64 forms, FP32 for the forms whose arithmetic is FP32.
"""
import math

import numpy as np
import torch

import mglc_gb300 as mg
from mglc_gb300 import capi

DEV = "cuda"
FP64_FORMS = ("fp64", "fx64")
FORM_BYTES = {"fp64": 8, "fx64": 8, "fp32": 4, "fp16": 2, "fp16s": 2, "bf16": 2, "bf16s": 2}


def listed():
    return [
        # the smallest grid of the served range: launches and latency count, fields
        # and residual come to the host as the reference's main loop takes them
        {"name": "lid_small", "kind": "lid", "nx": 32, "ny": 32, "nz": 32, "form": "fp64",
         "in_place": False, "steps": 20, "start": "flow", "host": True},
        # a non-cubic cavity with odd edges, rows that do not fill warps
        {"name": "lid_odd_fp32", "kind": "lid", "nx": 97, "ny": 63, "nz": 129, "form": "fp32",
         "in_place": False, "steps": 50, "start": "flow", "host": False},
        # the benchmark's own workload: 384^3 from rest, the drop-in precision
        {"name": "lid_384_fp64", "kind": "lid", "nx": 384, "ny": 384, "nz": 384, "form": "fp64",
         "in_place": False, "steps": 6, "start": "rest", "host": False},
        # the mixed form: 16-bit storage with stochastic rounding, one buffer
        {"name": "lid_256_fp16s", "kind": "lid", "nx": 256, "ny": 256, "nz": 256, "form": "fp16s",
         "in_place": True, "steps": 20, "start": "flow", "host": False},
        # FP64 parity through the fixed-point collision
        {"name": "lid_160_fx64", "kind": "lid", "nx": 160, "ny": 160, "nz": 160, "form": "fx64",
         "in_place": False, "steps": 10, "start": "flow", "host": False},
        # the differentially heated cavity of the configurations, with its Nusselt numbers
        {"name": "heated_128_fp64", "kind": "thermal", "nx": 128, "ny": 128, "nz": 128,
         "form": "fp64", "in_place": False, "ekman": 0.0, "steps": 10, "host": False},
        # rotating convection (the reference ships with Coriolis), odd sizes, one buffer
        {"name": "heated_rot_fp32", "kind": "thermal", "nx": 81, "ny": 97, "nz": 72,
         "form": "fp32", "in_place": True, "ekman": 1e-3, "steps": 50, "host": False},
        # the particle-laden channel of the configurations
        {"name": "channel_fp32", "kind": "spheres", "nx": 256, "ny": 128, "nz": 128, "np": 200,
         "radius": 5.0, "form": "fp32", "steps": 20, "warm": 100},
        # a smaller channel in the parity precision
        {"name": "channel_fp64", "kind": "spheres", "nx": 128, "ny": 64, "nz": 64, "np": 24,
         "radius": 5.0, "form": "fp64", "steps": 10, "warm": 100},
        # the 2-D cavity, bitwise the reference's statements
        {"name": "lid2d_1024", "kind": "lid2d", "nx": 1024, "ny": 1024, "steps": 40},
        # three circles settling in a box (the reference's case4)
        {"name": "circles2d", "kind": "circles", "nx": 400, "ny": 800, "np": 3, "radius": 10.0,
         "bisection": True, "steps": 20, "warm": 40},
        # a batch of requests of uneven sizes through the solve server
        {"name": "serve_batch", "kind": "serve", "count": 8, "n_lo": 32, "n_hi": 96,
         "form": "fp32", "in_place": False, "steps": 200},
    ]


def _loguniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi, cells):
    """Three edges in [lo, hi], log-uniform, with at most `cells` cells."""
    while True:
        n = [_loguniform(rng, lo, hi) for _ in range(3)]
        if n[0] * n[1] * n[2] <= cells:
            return dict(zip(("nx", "ny", "nz"), n))


def draw(rng):
    kind = rng.choice(("lid", "lid", "lid", "thermal", "thermal", "spheres", "spheres", "lid2d",
                       "circles", "shear", "serve"))
    if kind == "lid":
        return {"kind": kind, **_box(rng, 24, 320, 12_000_000),
                "form": rng.choice(("fp64", "fp64", "fx64", "fp32", "fp16", "fp16s", "bf16")),
                "in_place": rng.random() < 0.4, "steps": rng.randint(5, 40), "start": "flow",
                "host": rng.random() < 0.2}
    if kind == "thermal":
        return {"kind": kind, **_box(rng, 24, 200, 3_000_000),
                "form": rng.choice(("fp64", "fp64", "fx64", "fp32", "fp16s")),
                "in_place": rng.random() < 0.4, "ekman": rng.choice((0.0, 0.0, 1e-3)),
                "steps": rng.randint(5, 40), "host": False}
    if kind == "spheres":
        radius = rng.choice((3.5, 5.0, 6.3))
        box = {"nx": _loguniform(rng, 48, 300), "ny": _loguniform(rng, 40, 140),
               "nz": _loguniform(rng, 40, 140)}
        room = box["nx"] * (box["ny"] - 2 * radius - 8) * (box["nz"] - 2 * radius - 8)
        most = max(1, int(0.12 * room / (2 * radius + 4) ** 3))
        return {"kind": kind, **box, "np": _loguniform(rng, 1, max(2, min(200, most))),
                "radius": radius, "form": rng.choice(("fp32", "fp32", "fp64")),
                "steps": rng.randint(5, 30), "warm": 60}
    if kind == "lid2d":
        return {"kind": kind, "nx": _loguniform(rng, 65, 1500), "ny": _loguniform(rng, 65, 1500),
                "steps": rng.randint(10, 60)}
    if kind == "circles":
        return {"kind": kind, "nx": _loguniform(rng, 150, 700), "ny": _loguniform(rng, 150, 900),
                "np": rng.randint(1, 6), "radius": rng.choice((6.5, 8.0, 10.0)),
                "bisection": rng.random() < 0.5, "steps": rng.randint(5, 30), "warm": 40}
    if kind == "shear":
        return {"kind": kind, "nx": _loguniform(rng, 120, 900), "ny": _loguniform(rng, 100, 500),
                "np": rng.randint(1, 2), "radius": rng.choice((8.0, 10.4, 12.6)),
                "moving_frame": rng.random() < 0.5, "linear": rng.random() < 0.5,
                "steps": rng.randint(5, 30), "warm": 40}
    n_lo = rng.randint(16, 40)
    return {"kind": kind, "count": rng.randint(2, 8), "n_lo": n_lo,
            "n_hi": rng.randint(n_lo + 8, 96), "form": rng.choice(("fp32", "fp32", "fp16s")),
            "in_place": rng.random() < 0.5, "steps": 100}


# ---------------------------------------------------------------- lattice --
EX = [0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0]
EY = [0, 0, 0, 1, -1, 0, 0, 1, 1, -1, -1, 0, 0, 0, 0, 1, -1, 1, -1]
EZ = [0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1, 1, 1, -1, -1]
OPP = [0, 2, 1, 4, 3, 6, 5, 10, 9, 8, 7, 14, 13, 12, 11, 18, 17, 16, 15]
W19 = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
EX9, EY9 = [0, 1, 0, -1, 0, 1, -1, -1, 1], [0, 0, 1, 0, -1, 1, 1, -1, -1]
OPP9 = [0, 3, 4, 1, 2, 7, 8, 5, 6]
W9 = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4


def _numbers(case, seed):
    """The flow's numbers, from the seed: Re or Ra over the configurations' range."""
    r = np.random.default_rng(seed)
    return {"re": float(r.uniform(100.0, 1000.0)), "u0": float(r.uniform(0.08, 0.1)),
            "ra": _rayleigh(r, case.get("nz", 1), 1e4, 1e6)}


def _rayleigh(r, n, lo, hi):
    """Ra for a cavity n nodes high: above n^2 the D3Q7 diffusivity stays in its stable range."""
    return float(10 ** r.uniform(math.log10(max(lo, n * n)), math.log10(hi)))


def _waves(case, seed, count, amplitude):
    """`count` smooth seeded fields (nz, ny, nx) that vanish at the walls."""
    r = np.random.default_rng(seed + 1)
    axes = [(torch.arange(n, dtype=torch.float64, device=DEV) + 0.5) / n
            for n in (case["nz"], case["ny"], case["nx"])]
    out = []
    for _ in range(count):
        s = 0.0
        for _ in range(3):
            k, a = r.integers(1, 5, 3), float(r.uniform(-1, 1))
            z, y, x = (torch.sin(math.pi * int(kk) * ax) for kk, ax in zip(k, axes))
            s = s + a * z[:, None, None] * y[None, :, None] * x[None, None, :]
        out.append(amplitude * s / 2.0)
    return out


def _equilibrium(rho, u, v, w):
    usq = u * u + v * v + w * w
    f = []
    for a in range(19):
        un = EX[a] * u + EY[a] * v + EZ[a] * w
        f.append(rho * W19[a] * (1.0 + 3.0 * un + 4.5 * un * un - 1.5 * usq))
    return torch.stack(f)


def _cavity_state(case, seed):
    """A flow under way: f (19, nz, ny, nx) near the equilibrium of seeded waves."""
    u, v, w = _waves(case, seed, 3, 0.05)
    rho = 1.0 + _waves(case, seed + 7, 1, 2e-3)[0]
    f = _equilibrium(rho, u, v, w)
    g = torch.Generator(device=DEV).manual_seed(seed)
    noise = torch.rand(f.shape, generator=g, dtype=torch.float64, device=DEV) - 0.5
    return f + 2e-4 * noise * torch.tensor(W19, dtype=torch.float64, device=DEV)[:, None, None, None]


def _para_a(case, ra, pr=0.71, mach=0.1):
    nu = mach * case["nz"] * math.sqrt(3.0 * pr / ra) / 3.0
    return 42.0 * math.sqrt(3.0) * nu / pr - 6.0


def _heat_state(case, seed, para_a):
    """Temperature populations (7, nz, ny, nx): conduction between the y walls and waves."""
    y = (torch.arange(case["ny"], dtype=torch.float64, device=DEV) + 0.5) / case["ny"]
    T = (0.5 - y)[None, :, None] + _waves(case, seed + 13, 1, 0.2)[0]
    w = torch.tensor([(1.0 - para_a) / 7.0] + [(para_a + 6.0) / 42.0] * 6, dtype=torch.float64,
                     device=DEV)
    return w[:, None, None, None] * T


def _host(pops):
    """(Q, ...) on the device to the reference's layout: (..., Q) on the host."""
    return torch.movedim(pops, 0, -1).contiguous().cpu().numpy()


def _place(case, seed, dims, gap_wall, gap):
    """Seeded centres, rejected until the gaps between them and to the walls are kept."""
    r = np.random.default_rng(seed + 3)
    R = case["radius"]
    n = [case["nx"], case["ny"], case.get("nz", 1)][:dims]
    out = np.zeros((0, dims))
    for _ in range(400_000):
        if len(out) == case["np"]:
            break
        c = np.array([r.uniform(gap_wall + R + 1, m - R - gap_wall) for m in n])
        if dims == 3:  # the channel is periodic in x
            c[0] = r.uniform(0.5, n[0] + 0.5)
        d = out - c
        if dims == 3:
            d[:, 0] -= n[0] * np.round(d[:, 0] / n[0])
        if not len(out) or (d * d).sum(1).min() >= (2 * R + gap) ** 2:
            out = np.vstack([out, c])
    return out


# ---------------------------------------------------------------- prepare --
def prepare(case, seed):
    kind, num = case["kind"], _numbers(case, seed)
    if kind == "serve":
        srv = mg.SolveServer(hbm_budget_gb=4.0, max_active=32, precision=case["form"],
                             steps_per_iteration=100, tol=1e-12, max_steps=case["steps"],
                             keep_results=True, in_place=case["in_place"])
        srv.submit("lid", 16)  # a server that is up: tile shape chosen, graph built
        srv.run()
        return {"case": case, "srv": srv, "requests": _requests(case, seed)}
    stream = torch.cuda.Stream()
    s = {"case": case, "stream": stream}
    cells = case["nx"] * case["ny"] * case.get("nz", 1)
    if kind == "lid":
        c = mg.LidDrivenCavity(case["nx"], case["ny"], case["nz"], reynolds=num["re"], u0=num["u0"],
                               top_layer_u0=False, precision=case["form"],
                               in_place=case["in_place"])
        if case["start"] == "rest":
            c.initial()
        else:
            c.load_state(_host(_cavity_state(case, seed)))
        fields = 4
    elif kind == "thermal":
        c = mg.BuoyancyCavity(case["nx"], case["ny"], case["nz"], rayleigh=num["ra"], prandtl=0.71,
                              mach=0.1, t_hot=0.5, t_cold=-0.5, ekman=case["ekman"],
                              precision=case["form"], in_place=case["in_place"])
        c.load_state(_host(_cavity_state(case, seed)),
                     _host(_heat_state(case, seed, _para_a(case, num["ra"]))))
        fields = 5
    elif kind == "spheres":
        c = mg.ParticleFlow(case["nx"], case["ny"], case["nz"],
                            _place(case, seed, 3, 2.0, 2.0), case["radius"], tauf=0.65,
                            rho_solid=1.2, periodic_x=True, body_force=(1e-6, 0.0, 0.0),
                            precision=case["form"])
        fields = 4
    elif kind == "lid2d":
        c = mg.LidDrivenCavity2D(case["nx"], case["ny"], reynolds=num["re"] * 4.0, u0=num["u0"])
        c.load_state(_lid2d_state(case, seed))
        fields = 3
    elif kind == "circles":
        c = mg.ParticleFlow2D(case["nx"], case["ny"], _place(case, seed, 2, 8.0, 8.0),
                              case["radius"], tauf=0.7, gravity=0.01,
                              q_bisection=case["bisection"])
        fields = 0
    else:
        c = mg.ShearFlow2D(case["nx"], case["ny"], _place(case, seed, 2, 8.0, 8.0),
                           case["radius"], moving_frame=case["moving_frame"],
                           linear=case["linear"])
        fields = 0
    c.set_stream(stream.cuda_stream)
    if "warm" in case:  # particles on their way: a settled pattern of links, nodes changing phase
        c.initial()
        c.step(case["warm"])
    shape = (case["nz"], case["ny"], case["nx"]) if "nz" in case else (case["ny"], case["nx"])
    s["solve"], s["fields"] = c, [torch.empty(shape, dtype=torch.float64, device=DEV)
                                  for _ in range(fields)]
    s["cells"] = cells
    return s


def _requests(case, seed):
    r = np.random.default_rng(seed + 5)
    out = []
    for q in range(case["count"]):
        t = q / max(1, case["count"] - 1)
        n = int(round(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** t))
        out.append(("thermal" if q % 2 else "lid", n, float(r.uniform(100.0, 1000.0)),
                    _rayleigh(r, n, 1e3, 1e5)))
    return out


def _lid2d_state(case, seed):
    """f (ny, nx, 9): the equilibrium of a seeded wave."""
    r = np.random.default_rng(seed + 2)
    y, x = (np.arange(case["ny"]) + 0.5) / case["ny"], (np.arange(case["nx"]) + 0.5) / case["nx"]
    u, v = (0.05 * float(r.uniform(0.3, 1.0)) * np.outer(np.sin(math.pi * int(r.integers(1, 4)) * y),
                                                         np.sin(math.pi * int(r.integers(1, 4)) * x))
            for _ in range(2))
    rho = 1.0 + 1e-3 * np.outer(np.cos(math.pi * y), np.cos(math.pi * x))
    un = np.stack([EX9[a] * u + EY9[a] * v for a in range(9)], -1)
    return rho[..., None] * np.array(W9) * (1 + 3 * un + 4.5 * un * un - 1.5 * (u * u + v * v)[..., None])


# -------------------------------------------------------------------- run --
def _fields(s):
    """The macroscopic fields on the device, in the form's precision."""
    p = [f.data_ptr() for f in s["fields"]] + [None] * 5
    rc = capi.lib().mglc_get_macros_device(s["solve"].handle, *p[:5])
    if rc:
        capi.check(s["solve"].handle, rc)
    if s["case"].get("form", "fp64") in FP64_FORMS:
        return s["fields"]
    with torch.cuda.stream(s["stream"]):
        return [f.float() for f in s["fields"]]


def run(state):
    case = state["case"]
    if case["kind"] == "serve":
        srv = state["srv"]
        ids = [srv.submit(kind, n, reynolds=re, rayleigh=ra)
               for kind, n, re, ra in state["requests"]]
        srv.run()
        got = {r["id"]: r for r in srv.results()}
        return {"fields": [srv.field(i) for i in ids], "steps": [got[i]["steps"] for i in ids]}
    c = state["solve"]
    c.step(case["steps"])
    if case["kind"] in ("circles", "shear"):
        return {"fields": list(c.macro()), "particles": c.state(), "mask": c.mask()}
    if case.get("host"):
        fields = c.macro()
        out = {"fields": [f if case["form"] in FP64_FORMS else f.astype(np.float32)
                          for f in fields]}
        c.check()
        return out
    out = {"fields": _fields(state)}
    if case["kind"] == "thermal":
        c.nusselt()
    if case["kind"] == "spheres":
        real = np.float64 if case["form"] == "fp64" else np.float32
        out["particles"] = {k: v.astype(real) for k, v in c.state().items()}
        out["mask"] = c.mask()
    return out


# ------------------------------------------------------------------- work --
def work(case):
    """Every stored population read and written once a step, the fields written once."""
    kind = case["kind"]
    if kind == "serve":
        cell = FORM_BYTES[case["form"]]
        b = f = 0.0
        for k, n, _, _ in _requests(case, 0):
            heat = 2 * 7 * 4 + 2 * 4 if k == "thermal" else 0
            b += n ** 3 * (case["steps"] * (2 * 19 * cell + heat) + (5 if heat else 4) * 4)
            f += n ** 3 * case["steps"] * (360 if heat else 260)
        return {"bytes": b, "flops": f}
    cells = case["nx"] * case["ny"] * case.get("nz", 1)
    steps = case["steps"]
    if kind in ("lid2d", "circles", "shear"):
        return {"bytes": cells * (steps * 2 * 9 * 8 + 3 * 8), "flops": cells * steps * 190}
    cell, ops, fields = 2 * 19 * FORM_BYTES[case["form"]], 260, 4
    if kind == "thermal":
        wide = 8 if case["form"] in FP64_FORMS else 4
        cell += 2 * 7 * wide + 2 * wide * (3 if case["ekman"] else 1)
        ops, fields = 360, 5
    if kind == "spheres":
        cell += 4
    real = 8 if case["form"] in FP64_FORMS else 4
    return {"bytes": cells * (steps * cell + fields * real), "flops": cells * steps * ops}


# ------------------------------------------------------------------ exact --
def _basis19():
    """The D3Q19 moments of d'Humieres et al. (2002), as the reference orders them."""
    x, y, z = (np.array(a, float) for a in (EX, EY, EZ))
    e = x * x + y * y + z * z
    rows = [np.ones(19), 19 * e - 30, (21 * e * e - 53 * e + 24) / 2, x, (5 * e - 9) * x, y,
            (5 * e - 9) * y, z, (5 * e - 9) * z, 3 * x * x - e, (3 * e - 5) * (3 * x * x - e),
            y * y - z * z, (3 * e - 5) * (y * y - z * z), x * y, y * z, x * z,
            (y * y - z * z) * x, (z * z - x * x) * y, (x * x - y * y) * z]
    return np.array(rows)


def _rates(tau):
    return 1.0 / tau, 8.0 * (2.0 * tau - 1.0) / (8.0 * tau - 1.0)


def _stream(post, ex, opp):
    """Each population moves along its direction; one that would leave comes back reflected."""
    out = torch.empty_like(post)
    dims = post.dim() - 1
    for a in range(len(opp)):
        out[a] = post[opp[a]]
        to, fro = [], []
        for d in range(dims):  # the array's axes run z, y, x (or y, x)
            e = ex[dims - 1 - d][a]
            to.append(slice(max(e, 0), post.shape[1 + d] + min(e, 0)))
            fro.append(slice(max(-e, 0), post.shape[1 + d] + min(-e, 0)))
        out[a][tuple(to)] = post[a][tuple(fro)]
    return out


def _moments_eq(rho, u, v, w, lid):
    usq = u * u + v * v + w * w
    p9, p11 = 2 * u * u - v * v - w * w, v * v - w * w
    o = torch.zeros_like(rho)
    return torch.stack([rho, rho * (-11 + 19 * usq), rho * (3 - 5.5 * usq), rho * u,
                        -2 / 3 * rho * u, rho * v, -2 / 3 * rho * v, rho * w, -2 / 3 * rho * w,
                        rho * p9, -0.5 * rho * p9, rho * p11,
                        -0.5 * (p11 if lid else rho * p11),  # the lid's twelfth has no rho
                        rho * u * v, rho * v * w, rho * u * w, o, o, o])


def _times(matrix, pops):
    m = torch.tensor(matrix, dtype=torch.float64, device=pops.device)
    return (m @ pops.reshape(pops.shape[0], -1)).reshape(m.shape[0], *pops.shape[1:])


def _macro(f, force=None):
    e = torch.tensor([EX, EY, EZ], dtype=torch.float64, device=f.device)
    rho, j = f.sum(0), _times(e.cpu().numpy(), f)
    if force is not None:
        j = j + 0.5 * force
    return rho, j[0] / rho, j[1] / rho, j[2] / rho


def _lid_exact(f, re, u0, steps, rho=None):
    snu, sq = _rates(u0 * f.shape[3] / re * 3.0 + 0.5)
    M = _basis19()
    Minv = M.T / (M * M).sum(1)
    S = np.array([0, snu, snu, 0, sq, 0, sq, 0, sq] + [snu] * 7 + [sq] * 3)
    for _ in range(steps):
        rho, u, v, w = _macro(f)
        post = f - _times(Minv * S, _times(M, f) - _moments_eq(rho, u, v, w, True))
        f = _stream(post, (EX, EY, EZ), OPP)
        lid = rho[-1] / 6.0 * u0
        f[14][-1] -= lid
        f[13][-1] += lid
    return list(_macro(f))


def _heat_exact(f, g, ra, ekman, steps, pr=0.71, mach=0.1):
    nz = f.shape[1]
    tau = 0.5 + mach * nz * math.sqrt(3.0 * pr / ra)
    nu = (tau - 0.5) / 3.0
    kappa = nu / pr
    spin = nu / 2.0 / ekman / nz ** 2 if ekman > 0 else 0.0
    para_a = 42.0 * math.sqrt(3.0) * kappa - 6.0
    gbeta = ra * nu * kappa / nz ** 3
    qd, qnu = 3.0 - math.sqrt(3.0), 4.0 * math.sqrt(3.0) - 6.0
    snu, sq = _rates(tau)
    M = _basis19()
    Minv = M.T / (M * M).sum(1)
    S = np.array([0, snu, snu, 0, sq, 0, sq, 0, sq] + [snu] * 7 + [sq] * 3)
    x, y, z = (np.array(a[:7], float) for a in (EX, EY, EZ))
    N = np.array([np.ones(7), x, y, z, 7 * (x * x + y * y + z * z) - 6, 3 * x * x - (x + y + z) ** 2,
                  y * y - z * z])
    Ninv = N.T / (N * N).sum(1)
    force = torch.zeros(3, *f.shape[1:], dtype=torch.float64, device=f.device)
    wall = (6.0 + para_a) / 21.0 * 0.5
    for _ in range(steps):
        rho, u, v, w = _macro(f, force)
        T = g.sum(0)
        force = torch.stack([-2.0 * rho * v * spin, 2.0 * rho * u * spin, rho * gbeta * T])
        fx, fy, fz = force
        uf = u * fx + v * fy + w * fz
        o = torch.zeros_like(rho)
        src = torch.stack([o, 38 * uf, -11 * uf, fx, -2 / 3 * fx, fy, -2 / 3 * fy, fz, -2 / 3 * fz,
                           4 * u * fx - 2 * v * fy - 2 * w * fz, -2 * u * fx + v * fy + w * fz,
                           2 * v * fy - 2 * w * fz, w * fz - v * fy, u * fy + v * fx,
                           v * fz + w * fy, u * fz + w * fx, o, o, o])
        post = (f - _times(Minv * S, _times(M, f) - _moments_eq(rho, u, v, w, False)) +
                _times(Minv * (1.0 - 0.5 * S), src))
        f = _stream(post, (EX, EY, EZ), OPP)
        neq = torch.stack([T, T * u, T * v, T * w, T * para_a, o, o])
        q = np.array([0, qd, qd, qd, qnu, qnu, qnu])
        gp = g - _times(Ninv * q, _times(N, g) - neq)
        g = _stream(gp, (EX[:7], EY[:7], EZ[:7]), OPP[:7])
        g[3][:, 0] = -gp[4][:, 0] + wall
        g[4][:, -1] = -gp[3][:, -1] - wall
    return [*_macro(f, force), g.sum(0)]


def _lid2d_exact(f, re, u0, steps):
    snu, sq = _rates(u0 * f.shape[2] / re * 3.0 + 0.5)
    x, y = np.array(EX9, float), np.array(EY9, float)
    e = x * x + y * y
    M = np.array([np.ones(9), 3 * e - 4, (9 * e * e - 21 * e + 8) / 2, x, (3 * e - 5) * x, y,
                  (3 * e - 5) * y, x * x - y * y, x * y])
    Minv = M.T / (M * M).sum(1)
    S = np.array([0, snu, snu, 0, sq, 0, sq, snu, snu])
    for _ in range(steps):
        rho = f.sum(0)
        u, v = (_times(np.array([k], float), f)[0] / rho for k in (EX9, EY9))
        usq = u * u + v * v
        meq = torch.stack([rho, rho * (-2 + 3 * usq), rho * (1 - 3 * usq), rho * u, -rho * u,
                           rho * v, -rho * v, rho * (u * u - v * v), rho * u * v])
        post = f - _times(Minv * S, _times(M, f) - meq)
        f = _stream(post, (EX9, EY9), OPP9)
        lid = rho[-1] * u0 / 6.0
        f[7][-1] = post[5][-1] - lid
        f[8][-1] = post[6][-1] + lid
        f[4][-1] = post[2][-1]
    rho = f.sum(0)
    return [rho] + [_times(np.array([k], float), f)[0] / rho for k in (EX9, EY9)]


def exact(case, seed):
    """The same pass in plain torch, 64 bits, from the collision's moment form; None for
    the particle flows, whose solver would have to be written out again."""
    kind, num = case["kind"], _numbers(case, seed)
    if kind == "lid":
        if case["start"] == "rest":
            o = torch.zeros(case["nz"], case["ny"], case["nx"], dtype=torch.float64, device=DEV)
            f = _equilibrium(o + 1.0, o, o, o)
        else:
            f = _cavity_state(case, seed)
        return {"fields": _lid_exact(f, num["re"], num["u0"], case["steps"])}
    if kind == "thermal":
        return {"fields": _heat_exact(_cavity_state(case, seed),
                                      _heat_state(case, seed, _para_a(case, num["ra"])),
                                      num["ra"], case["ekman"], case["steps"])}
    if kind == "lid2d":
        f = torch.movedim(torch.from_numpy(_lid2d_state(case, seed)).to(DEV), -1, 0).contiguous()
        return {"fields": _lid2d_exact(f, num["re"] * 4.0, num["u0"], case["steps"])}
    if kind == "serve":
        fields = []
        for k, n, re, ra in _requests(case, seed):
            o = torch.zeros(n, n, n, dtype=torch.float64, device=DEV)
            f = _equilibrium(o + 1.0, o, o, o)
            if k == "lid":
                fields.append(torch.stack(_lid_exact(f, re, 0.1, case["steps"])))
                continue
            T = o.clone()
            T[:, 0], T[:, -1] = 0.5, -0.5
            a = _para_a({"nz": n}, ra)
            w = torch.tensor([(1.0 - a) / 7.0] + [(a + 6.0) / 42.0] * 6, dtype=torch.float64,
                             device=DEV)
            fields.append(torch.stack(_heat_exact(f, w[:, None, None, None] * T, ra, 0.0,
                                                  case["steps"])))
        return {"fields": fields, "steps": None}
    return None
