"""Performance cases of the solver and of the design-loop steps around it.

Each case is one call (or one design iteration) that a program using this
library makes: the density filter, the compliance sensitivity, the projected
design update, the drop-in ``mgcg1`` / ``mgcg9`` on host arrays, the
preconditioner of a new design, the operator apply, a whole design iteration,
a periodic homogenization, a batch of designs, and the learned correction's
network forward and training step.  ``listed()`` gives one case of each kind at
a size this repository's configurations use, ``draw()`` more of the same ranges.

Solves run to a tighter tolerance than a design loop needs (1e-10 where the
preconditioner is FP32), so that U, chi and the new design are converged
outputs that two versions of the solver have to agree on, whatever the rounding
inside their preconditioners.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-to_b200"))

NU, PENAL, EMIN, MOVE = 0.3, 3.0, 1e-9, 0.2
# local corner order of an element: (x, y, z) of the eight nodes
CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]


def listed():
    return [
        # the smallest call of a design loop: the filter on the 64x32x32 cantilever, bound by latency
        {"name": "filter_64", "kind": "filter", "nx": 64, "ny": 32, "nz": 32, "rmin": 3 ** 0.5, "div": False,
         "norm": True},
        # the sensitivity filter (divided by dHs, not normalised) with a wider radius at the bench grid
        {"name": "filter_256_wide", "kind": "filter", "nx": 256, "ny": 128, "nz": 128, "rmin": 2.5, "div": True,
         "norm": False},
        # element energies of a displacement field on a grid without any round number
        {"name": "sens_odd", "kind": "sens", "nx": 193, "ny": 97, "nz": 95},
        # Heaviside projection, chain rule and OC update of a bench-size design
        {"name": "update_256", "kind": "update", "n": 256 * 128 * 128, "volfrac": 0.12, "beta": 2.0},
        # the MATLAB drop-in on host arrays, the 64x32x32 cantilever with the reference's own schedule
        {"name": "mgcg1_64", "kind": "mgcg", "variant": 1, "nx": 64, "ny": 32, "nz": 32, "nl": 4, "tol": 1e-8},
        # a new design's FP64 hierarchy and one V-cycle on it
        {"name": "precond_128", "kind": "precond", "nx": 128, "ny": 64, "nz": 64, "nl": 5},
        # the plain FP64 operator on the largest configured grid (101.6M dofs)
        {"name": "apply_512", "kind": "apply", "nx": 512, "ny": 256, "nz": 256, "nl": 7},
        # one design iteration of the bench cantilever, mixed precision, the autotuner's schedule
        {"name": "design_256", "kind": "design", "nx": 256, "ny": 128, "nz": 128, "nl": 6, "ft": 1, "volfrac": 0.12,
         "nswp": 1, "nswp_coarse": 6, "coarse_from": 3, "tol": 1e-10},
        # periodic homogenization of a 128^3 random-field cell, six load cases
        {"name": "homog_128", "kind": "homog", "nx": 128, "ny": 128, "nz": 128, "nl": 6, "tol": 1e-10},
        # uneven designs solved together
        {"name": "batch_4", "kind": "batch", "shapes": "96x48x48,128x64x64,160x80x80,192x96x96", "nl": 5,
         "tol": 1e-10},
        # the learned correction's inference on the level-2 grid of the 512x256x256 bridge
        {"name": "net_forward_512", "kind": "net_forward", "X": 129, "Z": 65, "Y": 65},
        # one training step, eight samples on the level-2 grid of a 128^3 design
        {"name": "net_train_128", "kind": "net_train", "X": 33, "Z": 33, "Y": 33, "samples": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["filter", "sens", "update", "mgcg", "precond", "apply", "design", "homog", "batch",
                       "net_forward", "net_train"])

    def grid(lo, hi):   # a cantilever-like grid, halved down to three to five coarsest elements across
        ny = _log_int(rng, lo, hi)
        nl = int(np.log2(ny / 3)) + 1
        m = 2 ** (nl - 1)
        sizes = {"ny": ny, "nz": int(ny * rng.uniform(0.6, 1.4)), "nx": min(int(ny * rng.uniform(1.0, 2.5)), 2 * hi)}
        return {"nl": nl, **{k: max(2, v // m) * m for k, v in sizes.items()}}

    if kind in ("filter", "sens"):
        c = {"kind": kind, "nx": _log_int(rng, 24, 300), "ny": _log_int(rng, 16, 140), "nz": _log_int(rng, 16, 140)}
        if kind == "filter":
            c.update(rmin=rng.choice([3 ** 0.5, 1.5, 2.0, 2.5, 3.0, 3.5, 4.2]), div=rng.random() < 0.5,
                     norm=rng.random() < 0.5)
        return c
    if kind == "update":
        return {"kind": kind, "n": _log_int(rng, 30000, 4400000), "volfrac": rng.uniform(0.1, 0.4),
                "beta": rng.choice([1.0, 2.0, 4.0, 8.0])}
    if kind == "mgcg":
        return {"kind": kind, "variant": rng.choice([1, 1, 9]), "tol": rng.choice([1e-8, 1e-9, 1e-10]),
                **grid(16, 48)}
    if kind == "precond":
        return {"kind": kind, **grid(32, 96)}
    if kind == "apply":
        return {"kind": kind, **grid(16, 200)}
    if kind == "design":
        nsw = rng.choice([1, 2, 3])
        return {"kind": kind, "ft": rng.choice([1, 1, 3]), "volfrac": rng.uniform(0.1, 0.3), "nswp": nsw,
                "nswp_coarse": rng.choice([0, 4, 6]), "coarse_from": rng.choice([2, 3]), "tol": 1e-10,
                **grid(32, 112)}
    if kind == "homog":
        return {"kind": kind, "tol": 1e-10, "nl": 5, **{k: 16 * rng.randint(2, 8) for k in ("nx", "ny", "nz")}}
    if kind == "batch":
        shapes = []
        for _ in range(rng.randint(2, 6)):
            n = rng.randint(2, 5)
            shapes.append("%dx%dx%d" % (32 * n, 16 * n, 16 * rng.randint(2, 5)))
        return {"kind": kind, "shapes": ",".join(shapes), "nl": 4, "tol": 1e-10}
    c = {"kind": kind, "X": _log_int(rng, 9, 120), "Z": _log_int(rng, 9, 64), "Y": _log_int(rng, 9, 64)}
    if kind == "net_train":
        c.update(X=min(c["X"], 65), Z=min(c["Z"], 33), Y=min(c["Y"], 33), samples=rng.randint(1, 8))
    return c


# --- inputs --------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _smooth_field(g, shape, corr):
    """Gaussian random field with correlation length corr (grid units), zero mean, unit variance."""
    f = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
    k2 = sum((torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) * 2 * np.pi)
             .reshape([-1 if a == b else 1 for b in range(3)]) ** 2 for a, n in enumerate(shape))
    f = torch.fft.ifftn(torch.fft.fftn(f) * torch.exp(-0.5 * k2 * corr ** 2)).real
    return (f - f.mean()) / f.std()


def _design(seed, nx, ny, nz, volfrac):
    """A mid-optimisation cantilever density: a bottom chord that carries the load at the free end, a
    sloping top chord and diagonals between them, of uneven thickness with grey rims, in a soft
    background (density 0.03, a stiffness contrast of 4e4); the volume fraction is about volfrac."""
    g = _gen(seed)
    p = torch.rand(3, generator=g, device="cuda", dtype=torch.float64).tolist()
    x, z = (((torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n).reshape(sh)
            for n, sh in ((nx, (-1, 1, 1)), (nz, (1, -1, 1))))
    top = 1.0 - (0.6 + 0.2 * p[0]) * x
    turns = 2 + p[1]
    web = [((turns * (x + s * 0.5 * z) + p[2] + 0.5 * s) % 1.0 - 0.5).abs() / turns + 2.0 * (z - top).clamp(min=0.0)
           for s in (1, -1)]
    d = torch.minimum(torch.minimum(z + 0 * x, (z - top).abs()), torch.minimum(web[0], web[1]))
    d = (d * torch.exp(0.25 * _smooth_field(g, (nx, nz, ny), max(2.0, ny / 16)))).reshape(-1)
    cut = torch.sort(d).values[int(volfrac * (d.numel() - 1))]
    rim = torch.clamp(cut / 3.0, min=1.2 / nz)   # about an element at least, as the filter leaves it
    return (0.03 + 0.97 * torch.sigmoid((cut - d) / rim)).contiguous()


def _cell(seed, nx, ny, nz):
    """Random-field cell: sigmoid of a field with correlation length 8, in [1e-3, 1]."""
    f = _smooth_field(_gen(seed), (nx, nz, ny), 8.0).reshape(-1)
    return (1e-3 + (1 - 1e-3) * torch.sigmoid(3.0 * f)).contiguous()


def _simp(x):
    return EMIN + x ** PENAL * (1 - EMIN)


def _clamped(ny, nz):
    return np.arange(1, 3 * (ny + 1) * (nz + 1) + 1, dtype=np.float64)


def _load(nx, ny, nz, seed):
    """Unit -z load over the bottom edge of the free end, a little uneven from design to design."""
    F = np.zeros((nx + 1, nz + 1, ny + 1, 3))
    w = 1.0 + 0.1 * np.random.default_rng(seed).random(ny + 1)
    F[nx, 0, :, 2] = -w / w.sum()
    return F.reshape(-1)


def _displacement(seed, nx, ny, nz):
    """A bending field with local variation, the clamped x = 0 face at rest."""
    g = _gen(seed)
    x = torch.linspace(0, 1, nx + 1, device="cuda", dtype=torch.float64).reshape(-1, 1, 1)
    y = torch.linspace(-0.5, 0.5, ny + 1, device="cuda", dtype=torch.float64).reshape(1, 1, -1)
    z = torch.linspace(-0.5, 0.5, nz + 1, device="cuda", dtype=torch.float64).reshape(1, -1, 1)
    a, b = (1.0 + 0.2 * torch.rand(2, generator=g, device="cuda", dtype=torch.float64)).tolist()
    u = torch.zeros((nx + 1, nz + 1, ny + 1, 3), device="cuda", dtype=torch.float64)
    u[..., 2] = -100.0 * a * x * x + 0 * y + 0 * z
    u[..., 0] = 80.0 * b * x * z + 0 * y
    u[..., 1] = 10.0 * x * y * z
    u += 0.05 * torch.rand(u.shape, generator=g, device="cuda", dtype=torch.float64) * x.unsqueeze(-1)
    u[0] = 0
    return u.reshape(-1)


def _ke():
    """24x24 stiffness of the unit trilinear cube element, E = 1 (2x2x2 Gauss points)."""
    nu = NU
    lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 1 / (2 * (1 + nu))
    D = np.diag([2 * mu] * 3 + [mu] * 3)
    D[:3, :3] += lam
    K = np.zeros((24, 24))
    pts = (0.5 - 0.5 / 3 ** 0.5, 0.5 + 0.5 / 3 ** 0.5)
    for p in ((a, b, c) for a in pts for b in pts for c in pts):
        B = np.zeros((6, 24))
        for n, cr in enumerate(CORNERS):
            s = [p[d] if cr[d] else 1 - p[d] for d in range(3)]
            t = [1.0 if cr[d] else -1.0 for d in range(3)]
            gx, gy, gz = t[0] * s[1] * s[2], s[0] * t[1] * s[2], s[0] * s[1] * t[2]
            B[:, 3 * n:3 * n + 3] = [[gx, 0, 0], [0, gy, 0], [0, 0, gz], [gy, gx, 0], [0, gz, gy], [gz, 0, gx]]
        K += B.T @ D @ B / 8
    return 0.5 * (K + K.T)


NET = [(4, 16, 27), (16, 32, 27), (32, 64, 27), (64, 3, 1)]   # (inputs, outputs, taps) of the layers


def _net_params(seed):
    r = np.random.default_rng(seed)
    out = []
    for l, (ci, co, t) in enumerate(NET):
        out.append(r.standard_normal(co * ci * t) * (2.0 / (ci * t)) ** 0.5 * (0.1 if l == 3 else 1.0))
        out.append(0.02 * r.standard_normal(co))
    return np.concatenate(out).astype(np.float32)


def _net_input(seed, X, Z, Y, samples=1):
    """Density feature and the residual's three components in Jacobi-scaled units, RMS one."""
    g = _gen(seed)
    out = []
    for _ in range(samples):
        d = torch.sigmoid(3 * _smooth_field(g, (X, Z, Y), 2.0))
        out += [d.reshape(-1)] + [0.7 * (_smooth_field(g, (X, Z, Y), 1.5).reshape(-1)
                                         + torch.randn(X * Z * Y, generator=g, device="cuda", dtype=torch.float64))
                                  for _ in range(3)]
    return torch.cat(out).float().contiguous()


def _net_target(seed, X, Z, Y, samples):
    t = 0.3 * torch.randn((samples, 3, X, Z * Y), generator=_gen(seed + 7919), device="cuda")
    m = torch.ones_like(t)
    m[:, :, 0] = 0   # the clamped face has no error to learn
    return t.reshape(-1).contiguous(), m.reshape(-1).contiguous()


def _filter_inputs(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    x = _design(seed, nx, ny, nz, 0.2)
    div = None
    if case["div"]:   # the sensitivity form: dc ./ Hs, negative values over orders of magnitude
        x = -(x ** 2) * torch.rand(x.numel(), generator=_gen(seed + 1), device="cuda", dtype=torch.float64)
        div = 5.0 + torch.rand(x.numel(), generator=_gen(seed + 2), device="cuda", dtype=torch.float64)
    return x.contiguous(), div


def _update_inputs(case, seed):
    g = _gen(seed)
    n = case["n"]
    xt = torch.sigmoid(2.5 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64) - 2.0)
    x = (xt + 0.05 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)).clamp(1e-3, 1.0)
    dc = -torch.exp(2.0 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64)) * (0.05 + x)
    dv = torch.full((n,), 1.0 / n / case["volfrac"], device="cuda", dtype=torch.float64)
    return xt.contiguous(), x.contiguous(), dc.contiguous(), dv


# --- one case ------------------------------------------------------------------------------------

def prepare(case, seed):
    import gputo
    c = case
    s = {"case": c, "gputo": gputo, "stream": torch.cuda.Stream()}
    k = c["kind"]
    if k == "filter":
        s["x"], s["div"] = _filter_inputs(c, seed)
        s["out"] = torch.empty_like(s["x"])
    elif k == "sens":
        x = _design(seed, c["nx"], c["ny"], c["nz"], 0.2)
        s.update(Ke=_ke(), U=_displacement(seed, c["nx"], c["ny"], c["nz"]), CX=_simp(x), dsK=-PENAL * x ** 2,
                 ce=torch.empty_like(x), dc=torch.empty_like(x))
    elif k == "update":
        s["xt"], s["x"], s["dc"], s["dv"] = _update_inputs(c, seed)
        s.update({q: torch.empty_like(s["x"]) for q in ("xPhys", "dprj", "dcp", "dvp", "xnew")})
    elif k == "mgcg":
        s.update(Ke=_ke(), F=_load(c["nx"], c["ny"], c["nz"], seed), fixed=_clamped(c["ny"], c["nz"]),
                 CX=_simp(_design(seed, c["nx"], c["ny"], c["nz"], 0.3)).cpu().numpy())
        s["U"] = np.zeros_like(s["F"])
    elif k in ("precond", "apply"):
        s["solver"] = gputo.Solver(c["nx"], c["ny"], c["nz"], c["nl"])
        s["solver"].set_problem(_ke(), _clamped(c["ny"], c["nz"]))
        s["CX"] = _simp(_design(seed, c["nx"], c["ny"], c["nz"], 0.2))
        if k == "precond":
            r = torch.randn(3 * (c["nx"] + 1) * (c["ny"] + 1) * (c["nz"] + 1), generator=_gen(seed + 3),
                            device="cuda", dtype=torch.float64)
            r[:3 * (c["ny"] + 1) * (c["nz"] + 1)] = 0
            s["in"] = r
        else:
            s["in"] = _displacement(seed, c["nx"], c["ny"], c["nz"])
            torch.cuda.synchronize()
            s["solver"].setup(s["CX"])
        s["out"] = torch.empty_like(s["in"])
    elif k == "design":
        o = gputo.default_options(precision=gputo.PREC_MIXED, nswp=c["nswp"], nswp_coarse=c["nswp_coarse"],
                                  coarse_from=c["coarse_from"], check_every=8)
        s["x0"] = _design(seed, c["nx"], c["ny"], c["nz"], c["volfrac"])
        s["loop"] = gputo.DesignLoop(c["nx"], c["ny"], c["nz"], c["nl"], _load(c["nx"], c["ny"], c["nz"], seed),
                                     _clamped(c["ny"], c["nz"]), _ke(), volfrac=c["volfrac"], penal=PENAL,
                                     move=MOVE, tol=c["tol"], maxit=1500, options=o, stream=s["stream"], ft=c["ft"])
    elif k == "homog":
        s.update(Ke=_ke(), CX=_simp(_cell(seed, c["nx"], c["ny"], c["nz"])),
                 homog=gputo.Homog(c["nx"], c["ny"], c["nz"], c["nl"]),
                 chi=torch.empty(18 * c["nx"] * c["ny"] * c["nz"], device="cuda", dtype=torch.float64))
    elif k == "batch":
        s.update(solvers=[], F=[], U=[], CX=[])
        for q, t in enumerate(c["shapes"].split(",")):
            nx, ny, nz = (int(v) for v in t.split("x"))
            sv = gputo.Solver(nx, ny, nz, c["nl"], gputo.default_options(precision=gputo.PREC_MIXED, nswp=2))
            sv.set_problem(_ke(), _clamped(ny, nz))
            s["solvers"].append(sv)
            s["F"].append(torch.as_tensor(_load(nx, ny, nz, seed + q), device="cuda"))
            s["U"].append(torch.zeros_like(s["F"][-1]))
            s["CX"].append(_simp(_design(seed + 31 * q, nx, ny, nz, 0.2)))
        s["batch"] = gputo.Batch(s["solvers"])
    else:
        n = c["X"] * c["Z"] * c["Y"]
        s["net"] = gputo.Net(0)
        s["net"].set_params(_net_params(seed))
        if k == "net_forward":
            s["x"] = _net_input(seed, c["X"], c["Z"], c["Y"])
            s["y"] = torch.empty(3 * n, device="cuda", dtype=torch.float32)
        else:
            s["x"] = _net_input(seed, c["X"], c["Z"], c["Y"], c["samples"])
            s["t"], s["m"] = _net_target(seed, c["X"], c["Z"], c["Y"], c["samples"])
            s["grads"] = np.zeros(gputo.Net.num_params(), dtype=np.float32)
    return s


def run(s):
    c, gputo, st = s["case"], s["gputo"], s["stream"]
    k = c["kind"]
    if k == "filter":
        gputo.density_filter_dev(s["x"], s["out"], c["nx"], c["ny"], c["nz"], c["rmin"], divisor=s["div"],
                                 normalize=c["norm"], stream=st)
        return s["out"]
    if k == "sens":
        comp = gputo.compliance_sens_dev(s["Ke"], s["U"], s["CX"], s["dsK"], c["nx"], c["ny"], c["nz"], s["ce"],
                                         s["dc"], stream=st)
        return {"ce": s["ce"], "dc": s["dc"], "compliance": comp}
    if k == "update":
        eta = gputo.heaviside_dev(s["xt"], s["xPhys"], c["volfrac"], c["beta"], 0.4, s["dprj"], stream=st)
        gputo.mul_dev(s["dc"], s["dprj"], s["dcp"], stream=st)
        lmid = gputo.oc_update_dev(s["x"], s["dcp"], s["dv"], s["xnew"], c["volfrac"], MOVE, stream=st)
        return {"xPhys": s["xPhys"], "dprj": s["dprj"], "dc": s["dcp"], "xnew": s["xnew"], "eta": eta, "lmid": lmid}
    if k == "mgcg":
        a = (s["Ke"], s["F"], s["U"], s["CX"], s["fixed"], s["fixed"].size, c["nx"], c["ny"], c["nz"], c["nl"],
             c["tol"], 1000)
        if c["variant"] == 9:
            gputo.mgcg9(*a, 3, printLev=0)
        else:
            gputo.mgcg1(*a, printLev=0)
        return s["U"]
    if k == "precond":
        s["solver"].setup(s["CX"], stream=st)
        s["solver"].vcycle(s["in"], s["out"], stream=st)
        return s["out"]
    if k == "apply":
        s["solver"].apply(s["in"], s["out"], stream=st)
        return s["out"]
    if k == "design":
        lp = s["loop"]
        with torch.cuda.stream(st):
            lp.x.copy_(s["x0"])
            lp.eta = 0.4
            info = lp.step()
        return {"x": lp.x, "xPhys": lp.xPhys, "U": lp.U, "ce": lp.ce, "dc": lp.dcf, "compliance": info["c"]}
    if k == "homog":
        C, _, _ = s["homog"].solve(s["Ke"], s["CX"], tol=c["tol"], maxit=1000, chi=s["chi"], stream=st)
        return {"C": C, "chi": s["chi"]}
    if k == "batch":
        for sv, cx in zip(s["solvers"], s["CX"]):
            sv.setup(cx)
        s["batch"].solve(s["F"], s["U"], c["tol"], 1500, check_every=8)
        return s["U"]
    if k == "net_forward":
        s["net"].forward(s["x"], (c["X"], c["Z"], c["Y"]), s["y"], stream=st)
        return s["y"]
    s["net"].train_step(s["x"], s["t"], s["m"], c["samples"], (c["X"], c["Z"], c["Y"]), 1e-3, grads_out=s["grads"],
                        stream=st)
    return s["grads"]


def work(case):
    """Inputs read once and outputs written once; for the solves that is a floor of any
    method, their iterations come on top."""
    c = case
    k = c["kind"]
    if k in ("net_forward", "net_train"):
        n = c["X"] * c["Z"] * c["Y"]
        par = sum((ci * t + 1) * co for ci, co, t in NET)
        mac = sum(ci * co * t for ci, co, t in NET) * n
        if k == "net_forward":
            return {"bytes": 4.0 * (7 * n + par), "flops": 2.0 * mac}
        # forward, weight gradients, and data gradients of all but the first layer
        back = mac - 4 * 16 * 27 * n
        return {"bytes": 4.0 * (10 * n * c["samples"] + 5 * par), "flops": 2.0 * c["samples"] * (2 * mac + back)}
    if k == "update":   # xt, x, dc, dv read; xPhys, dprj, dc dprj, xnew written
        return {"bytes": 64.0 * c["n"], "flops": 40.0 * c["n"]}
    if k == "batch":
        shapes = [tuple(int(v) for v in t.split("x")) for t in c["shapes"].split(",")]
        return {"bytes": float(sum(8 * x * y * z + 48 * (x + 1) * (y + 1) * (z + 1) for x, y, z in shapes)),
                "flops": 0.0}
    nel = c["nx"] * c["ny"] * c["nz"]
    dof = 3 * (c["nx"] + 1) * (c["ny"] + 1) * (c["nz"] + 1)
    if k == "filter":
        return {"bytes": 8.0 * nel * (3 if c["div"] else 2), "flops": 0.0}
    if k == "sens":
        return {"bytes": 8.0 * (dof + 4 * nel), "flops": 149.0 * nel}
    if k == "apply":
        return {"bytes": 8.0 * (2 * dof + nel), "flops": 149.0 * nel}
    if k == "homog":
        return {"bytes": 8.0 * (18 * nel + nel), "flops": 0.0}
    if k == "design":   # x and F read; x, xPhys, U, ce and dc written
        return {"bytes": 8.0 * (2 * dof + 5 * nel), "flops": 0.0}
    return {"bytes": 8.0 * (2 * dof + nel), "flops": 0.0}   # F (or r) and CX read, U (or z) written


# --- the values in 64 bits -----------------------------------------------------------------------

def _corner_values(u, nx, ny, nz):
    """[24, elements] corner values of a nodal field, local order."""
    u = u.reshape(nx + 1, nz + 1, ny + 1, 3)
    return torch.cat([u[a:a + nx, b:b + nz, j:j + ny].reshape(-1, 3).T for a, j, b in CORNERS])


def _apply_exact(CX, u, nx, ny, nz):
    K = torch.as_tensor(_ke(), device="cuda")
    r = torch.zeros((nx + 1, nz + 1, ny + 1, 3), device="cuda", dtype=torch.float64)
    u = u.reshape(nx + 1, nz + 1, ny + 1, 3)
    CX = CX.reshape(nx, nz, ny)
    for x0 in range(0, nx, 64):   # slabs of element planes
        m = min(64, nx - x0)
        f = (K @ _corner_values(u[x0:x0 + m + 1], m, ny, nz)) * CX[x0:x0 + m].reshape(1, -1)
        for n, (a, j, b) in enumerate(CORNERS):
            r[x0 + a:x0 + a + m, b:b + nz, j:j + ny] += f[3 * n:3 * n + 3].T.reshape(m, nz, ny, 3)
    r[0] = 0
    return r.reshape(-1)


def _filter_exact(case, seed):
    nx, ny, nz, rmin = case["nx"], case["ny"], case["nz"], case["rmin"]
    x, div = _filter_inputs(case, seed)
    x = (x / div if div is not None else x).reshape(nx, nz, ny)
    R = int(np.ceil(rmin)) - 1

    def mirrored(n):   # edge sample included
        i = torch.arange(-R, n + R, device="cuda")
        i = torch.where(i < 0, -1 - i, i)
        return torch.where(i >= n, 2 * n - 1 - i, i)

    p = x[mirrored(nx)][:, mirrored(nz)][:, :, mirrored(ny)]
    out, hs = torch.zeros_like(x), 0.0
    for a in range(-R, R + 1):
        for b in range(-R, R + 1):
            for j in range(-R, R + 1):
                w = max(0.0, rmin - (a * a + b * b + j * j) ** 0.5)
                hs += w
                if w > 0:
                    out += w * p[a + R:a + R + nx, b + R:b + R + nz, j + R:j + R + ny]
    return (out / hs if case["norm"] else out).reshape(-1)


def _update_exact(case, seed):
    xt, x, dc, dv = _update_inputs(case, seed)
    beta, vf, eta, th = case["beta"], case["volfrac"], 0.4, np.tanh

    def prj(e):
        return (th(beta * e) + torch.tanh(beta * (xt - e))) / (th(beta * e) + th(beta * (1 - e)))

    for _ in range(60):
        f = float(prj(eta).mean()) - vf
        if abs(f) <= 1e-6:
            break
        d = -beta / np.sinh(beta) / torch.cosh(beta * (xt - eta)) ** 2 * torch.sinh(beta * xt) \
            * torch.sinh(beta * (1 - xt))
        eta -= f / float(d.mean())
    dprj = beta * (1 - torch.tanh(beta * (xt - eta)) ** 2) / (th(beta * eta) + th(beta * (1 - eta)))
    dcp = dc * dprj
    ocp = x * torch.sqrt(-dcp / dv)
    l1, l2, mid = 0.0, float(ocp.mean()) / vf, 0.0
    xn = x.clone()
    while (l2 - l1) / (l2 + l1) > 1e-4:
        mid = 0.5 * (l1 + l2)
        xn = torch.maximum(torch.minimum(torch.minimum(ocp / mid, x + MOVE), torch.ones_like(x)), x - MOVE)
        xn = xn.clamp(min=0.0)
        if float(xn.mean()) > vf:
            l1 = mid
        else:
            l2 = mid
    return {"xPhys": prj(eta), "dprj": dprj, "dc": dcp, "xnew": xn, "eta": eta, "lmid": mid}


def _net_layers(p):
    """The layers' weights [outputs, inputs, taps] and biases as 64-bit leaves; the network uses weights rounded to
    BF16."""
    out, o = [], 0
    for ci, co, t in NET:
        w = torch.as_tensor(p[o:o + co * ci * t], device="cuda").to(torch.bfloat16).double().reshape(co, ci, t)
        b = torch.as_tensor(p[o + co * ci * t:o + co * (ci * t + 1)], device="cuda").double()
        out.append((w.requires_grad_(), b.requires_grad_()))
        o += co * (ci * t + 1)
    return out


def _net_exact(layers, x, X, Z, Y):
    h = x.double().reshape(4, X, Z, Y)
    for l, (w, b) in enumerate(layers):
        if w.shape[2] == 1:
            y = torch.einsum("oi,ixzy->oxzy", w[:, :, 0], h)
        else:
            p = torch.nn.functional.pad(h, (1, 1, 1, 1, 1, 1))
            y = 0
            for t in range(27):
                dx, dz, dy = t // 9, t // 3 % 3, t % 3
                y = y + torch.einsum("oi,ixzy->oxzy", w[:, :, t], p[:, dx:dx + X, dz:dz + Z, dy:dy + Y])
        y = y + b.reshape(-1, 1, 1, 1)
        h = torch.relu(y) if l < 3 else y
    return h.reshape(-1)


def exact(case, seed):
    """The single steps in 64 bits; the solves have none (a direct one of their size is out of reach)."""
    c = case
    k = c["kind"]
    if k == "filter":
        return _filter_exact(c, seed)
    if k == "sens":
        x = _design(seed, c["nx"], c["ny"], c["nz"], 0.2)
        u = _corner_values(_displacement(seed, c["nx"], c["ny"], c["nz"]), c["nx"], c["ny"], c["nz"])
        ce = (u * (torch.as_tensor(_ke(), device="cuda") @ u)).sum(0)
        return {"ce": ce, "dc": -PENAL * x ** 2 * ce, "compliance": float((_simp(x) * ce).sum())}
    if k == "update":
        return _update_exact(c, seed)
    if k == "apply":
        return _apply_exact(_simp(_design(seed, c["nx"], c["ny"], c["nz"], 0.2)),
                            _displacement(seed, c["nx"], c["ny"], c["nz"]), c["nx"], c["ny"], c["nz"])
    if k == "net_forward":
        with torch.no_grad():
            return _net_exact(_net_layers(_net_params(seed)), _net_input(seed, c["X"], c["Z"], c["Y"]), c["X"],
                              c["Z"], c["Y"])
    if k == "net_train":
        layers = _net_layers(_net_params(seed))
        S, n = c["samples"], c["X"] * c["Z"] * c["Y"]
        x = _net_input(seed, c["X"], c["Z"], c["Y"], S).reshape(S, 4 * n)
        t, m = (v.reshape(S, 3 * n).double() for v in _net_target(seed, c["X"], c["Z"], c["Y"], S))
        for q in range(S):
            d = _net_exact(layers, x[q], c["X"], c["Z"], c["Y"]) - t[q]
            ((m[q] * d * d).sum() / m[q].sum().clamp(min=1.0)).backward()
        return torch.cat([v.grad.reshape(-1) for wb in layers for v in wb])
    return None
