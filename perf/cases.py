"""Performance cases: what programs built on pdds_gb300 call, from one knot to a whole batch.

A case's "kind" says which public call it times:

  knot        one knot with a caller-built stencil (EMFKACSolver.Solve_GPU_Analytic, FP64): the
              reference's per-knot worker call
  solve       PDDSparseGM.Solve on a rectangular layout (MIXED estimate of G and B, interface
              solve), with or without G's variances and the subdomain interiors
  estimate    PDDSparseGM.estimate alone in the plain FP64 form or the bit-exact replay form
  lut         a table-served variable-coefficient estimate (MIXED)
  circle      a variance-adaptive estimate on the disk layout, and its interface solve
  batch       many Helmholtz instances through Batch.run
  semilinear  the Newton outer loop: tables, estimate, interface solve, subdomain solves per step
  interface   PDDSparseGM.solve_interface alone, by GMRES with refinement or by BiCGSTAB

The layouts, problems and step sizes are the ones of this repository's benchmark configurations
and tests.  The Philox seed is the input that changes with `seed`: every path of a pass draws other
normals, and the systems that the interface cases solve differ with it.
"""
import math

import numpy as np
import torch

import pdds_gb300 as P
from pdds_gb300.config import batch_instances, fac_rule, varcoef_tables

RICH = dict(adaptive_h=True, richardson=True, dup_sum=True)

# problem -> side length and lower corner of its square domain
DOMAIN = {"poisson": (2.0, -1.0), "monegros": (10.0, -5.0), "helmholtz": (1.0, 0.0), "varcoef": (1.0, 0.0)}


# --------------------------------------------------------------------------- the cases
def listed():
    return [
        # the reference's worker step, once per knot: the smallest call, where launches and waits count
        dict(name="knot_fp64", kind="knot", problem="poisson", gap_nodes=11, npaths=5000, h=2e-3, richardson=False),
        # the CPU-runnable benchmark configuration by the reference's plain method: a small interactive solve
        dict(name="poisson_4x4_n11", kind="solve", problem="poisson", nsub=4, nnode=11, npaths=10_000, h=1e-3,
             richardson=False, want_var=False, interiors=0),
        # the reference's recorded problem and path count on its 741-knot layout, with every output that it
        # writes: G's variances and the subdomain interiors
        dict(name="monegros_4x4_n32_var", kind="solve", problem="monegros", nsub=4, nnode=32, npaths=5000, h=5e-3,
             richardson=False, want_var=True, interiors=32),
        # the headline configuration: a production-sized layout at full accuracy
        dict(name="poisson_12x12_n43", kind="solve", problem="poisson", nsub=12, nnode=43, npaths=20_000, h=5e-4,
             richardson=True, want_var=False, interiors=0),
        # the double-precision form that results are checked with
        dict(name="fp64_4x4_n11", kind="estimate", problem="poisson", mode="fp64", nsub=4, nnode=11, npaths=10_000,
             h=1e-3, richardson=False),
        # the bit-exact form that reproduces the CPU restatement
        dict(name="replay_4x4_n11", kind="estimate", problem="poisson", mode="replay", nsub=4, nnode=11,
             npaths=10_000, h=1e-3, richardson=False),
        # coefficients from 1024^2 tables, the default sampler
        dict(name="varcoef_lut_8x8_n31", kind="lut", table=1024, sampler="bspline", nsub=8, nnode=31, npaths=50_000,
             h=5e-4),
        # very uneven path lengths: variance-adaptive paths on the disk
        dict(name="circle_6x16_n11", kind="circle", rings=6, sectors=16, nnode=11, npaths=1000, h=2e-5,
             npaths_max=100_000),
        # a serving batch of independent problems
        dict(name="batch_24", kind="batch", instances=24, npaths=10_000, h=1e-3),
        # two steps of the semilinear loop
        dict(name="semilinear_8x8_n21", kind="semilinear", steps=2, nsub=8, nnode=21, npaths=20_000, h=5e-4, m=32),
        # the interface solve by itself: the default method on the headline layout
        dict(name="gmres_12x12_n43", kind="interface", method="gmres", nsub=12, nnode=43, npaths=2000, h=5e-4),
        # and the reference's method on a medium one
        dict(name="bicgstab_8x8_n31", kind="interface", method="bicgstab", nsub=8, nnode=31, npaths=2000, h=5e-4),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def _knots(nsub, nnode):
    return (nsub - 1) * (nsub * (nnode - 1) + 1) + (nsub - 1) * (nsub * (nnode - 2) + 2)


def draw(rng):
    kind = rng.choice(["knot", "solve", "solve", "fp64", "replay", "lut", "circle", "batch", "semilinear", "interface",
                       "interface"])
    if kind == "knot":
        return dict(kind="knot", problem=rng.choice(["poisson", "helmholtz"]), gap_nodes=rng.randint(6, 32),
                    npaths=int(_log(rng, 256, 20_000)), h=round(_log(rng, 5e-4, 5e-3), 6),
                    richardson=rng.random() < 0.4)
    if kind == "solve":
        while True:
            nsub, nnode = rng.randint(3, 14), rng.randint(8, 43)
            npaths = int(_log(rng, 2000, 20_000))
            if _knots(nsub, nnode) <= 10_989:
                break
        problem = rng.choice(["poisson", "poisson", "monegros", "helmholtz", "varcoef"])
        sub = DOMAIN[problem][0] / nsub  # the step as a share of the subdomain's exit time, as in the listed ones
        rich = rng.random() < 0.6
        return dict(kind="solve", problem=problem, nsub=nsub, nnode=nnode, npaths=npaths,
                    h=float("%.3g" % (sub * sub * _log(rng, 4e-3 if rich else 8e-4, 2e-2))), richardson=rich,
                    want_var=rng.random() < 0.3, interiors=0 if problem == "varcoef" else rng.choice([0, 0, 16, 32]))
    if kind == "fp64":
        nsub, nnode = rng.randint(2, 8), rng.randint(6, 21)
        return dict(kind="estimate", problem=rng.choice(["poisson", "helmholtz", "varcoef"]), mode="fp64", nsub=nsub,
                    nnode=nnode, npaths=max(256, int(_log(rng, 1e5, 2.4e6) / _knots(nsub, nnode))),
                    h=float("%.3g" % ((2.0 / nsub) ** 2 * 4e-3)), richardson=rng.random() < 0.4)
    if kind == "replay":
        nsub, nnode = rng.randint(2, 5), rng.randint(6, 13)
        return dict(kind="estimate", problem=rng.choice(["poisson", "helmholtz", "varcoef"]), mode="replay",
                    nsub=nsub, nnode=nnode, npaths=max(64, min(8000, int(_log(rng, 5e4, 1.2e6) / _knots(nsub, nnode)))),
                    h=float("%.3g" % ((2.0 / nsub) ** 2 * 4e-3)), richardson=False)
    if kind == "lut":
        return dict(kind="lut", table=rng.choice([127, 256, 500, 1024]), sampler=rng.choice(["bspline", "catmull_rom",
                                                                                              "bilinear"]),
                    nsub=rng.randint(4, 8), nnode=rng.randint(9, 31), npaths=int(_log(rng, 2000, 40_000)), h=5e-4)
    if kind == "circle":
        return dict(kind="circle", rings=rng.randint(3, 6), sectors=rng.choice([8, 12, 16]), nnode=rng.randint(7, 11),
                    npaths=rng.choice([512, 1000]), h=float("%.3g" % _log(rng, 2e-5, 5e-4)),
                    npaths_max=rng.choice([20_000, 50_000]))
    if kind == "batch":
        return dict(kind="batch", instances=rng.randint(3, 24), npaths=int(_log(rng, 2000, 10_000)), h=1e-3)
    if kind == "semilinear":
        return dict(kind="semilinear", steps=2, nsub=rng.randint(4, 8), nnode=rng.randint(9, 21),
                    npaths=int(_log(rng, 4000, 20_000)), h=5e-4, m=rng.choice([16, 24, 32]))
    while True:
        nsub, nnode = rng.randint(4, 12), rng.randint(9, 43)
        if 200 <= _knots(nsub, nnode) <= 10_989:
            break
    method = rng.choice(["gmres", "bicgstab"])
    return dict(kind="interface", method=method, nsub=nsub, nnode=nnode, npaths=2000,
                h=float("%.3g" % ((2.0 / nsub) ** 2 * 1.8e-2)))


# --------------------------------------------------------------------------- inputs and passes
def _bvp(name, seed=0):
    return {"poisson": P.BVP.poisson_sincos, "monegros": P.BVP.monegros, "varcoef": P.BVP.varcoef,
            "helmholtz": lambda: P.BVP.helmholtz(2.3, 1.7, -1.5)}[name]()


def _rect(problem, nsub, nnode):
    side, lo = DOMAIN[problem]
    return P.PDDSparseGM((lo, lo), (lo + side, lo + side), nsub, nnode, fac_rule(side, nsub, nnode))


_TABLES = {}  # size -> the file a user would have on disk


def _tables(n):
    if n not in _TABLES:
        _TABLES[n] = varcoef_tables(n)
    return _TABLES[n]


def _knot_stencil(case):
    """A knot on an interface of the 4 x 4 layout of its problem: the two subdomains beside it, side knots at the
    layout's spacing, the sides elongated by half a segment; the south side lies on the boundary."""
    side, lo = DOMAIN[case["problem"]]
    L, n = side / 4.0, case["gap_nodes"]
    gap = L / (n - 1)
    c = fac_rule(side, 4, n)
    rect = (lo + L, lo, lo + 2 * L, lo + 2 * L)
    half = (n // 2) * gap
    index, x, y, base = {}, {}, {}, 100
    for d in "NEW":
        t0, t1 = (rect[0] - half, rect[2] + half) if d == "N" else (rect[1] + gap, rect[3] + half)
        t = t0 + gap * np.arange(int(round((t1 - t0) / gap)) + 1)
        index[d] = np.arange(base, base + len(t), dtype=np.int32)
        base += len(t)
        x[d] = t if d == "N" else np.full(len(t), rect[2] if d == "E" else rect[0])
        y[d] = np.full(len(t), rect[3]) if d == "N" else t
    st = P.Stencil(rect, (lo, lo, lo + side, lo + side)).Init(index, x, y, rect).Compute_ipsi(c)
    x0 = (rect[0] + 0.5 * L, lo + L + 0.3 * gap)
    return st, x0


def prepare(case, seed):
    k = case["kind"]
    s = {"case": case, "seed": 1000 + seed}
    if k == "knot":
        s["stencil"], s["x0"] = _knot_stencil(case)
        s["solver"] = P.EMFKACSolver()
        s["bvp"] = _bvp(case["problem"])
    elif k in ("solve", "estimate"):
        s["bvp"] = _bvp(case["problem"])
        s["pd"] = _rect(case["problem"], case["nsub"], case["nnode"])
    elif k == "lut":
        coef, g, bounds = _tables(case["table"])
        s["bvp"] = P.BVP.lut(coef, g, bounds, sampler=case["sampler"])
        s["pd"] = _rect("varcoef", case["nsub"], case["nnode"])
    elif k == "circle":
        s["bvp"] = P.BVP.circle_poisson()
        s["pd"] = P.PDDSparseGM.circle_mesh(1.0, case["rings"], case["sectors"], case["nnode"])
    elif k == "batch":
        s["batch"] = P.Batch(P.BVP.HELMHOLTZ, batch_instances(case["instances"], seed=1234, scaled_h=case["h"]),
                             order="smallest_first")
    elif k == "semilinear":
        s["pd"] = P.PDDSparseGM((0.0, 0.0), (1.0, 1.0), case["nsub"], case["nnode"],
                                fac_rule(1.0, case["nsub"], case["nnode"]))
    else:
        s["bvp"] = _bvp("poisson")
        s["pd"] = _rect("poisson", case["nsub"], case["nnode"])
        s["est"] = s["pd"].estimate(s["bvp"], case["npaths"], case["h"], seed=s["seed"], **RICH)
    return s


def run(s):
    case, seed = s["case"], s["seed"]
    k = case["kind"]
    rich = RICH if case.get("richardson") else {}
    if k == "knot":
        opts = {"adaptive_h": True, "richardson": True} if rich else {}
        G, _, gj, B, BB = s["solver"].Solve_GPU_Analytic(s["x0"], case["npaths"], case["h"], 0.0, s["bvp"],
                                                         s["stencil"], seed=seed, knot_id=7, **opts)
        return {"G": G, "G_j": gj, "B": B, "BB": BB}
    if k == "solve":
        pd = s["pd"]
        u, est, _ = pd.Solve(s["bvp"], case["npaths"], case["h"], seed=seed, want_var=case["want_var"], **rich)
        out = {"u": u, "G": est.val, "B": est.B, "BB": est.BB}
        if case["want_var"]:
            out["G_var"] = est.var
        if case["interiors"]:
            out["interior"] = pd.subdomain_solve(case["interiors"])[2]
        return out
    if k == "estimate":
        mode = P.MODE_FP64 if case["mode"] == "fp64" else P.MODE_REPLAY_FP64
        est = s["pd"].estimate(s["bvp"], case["npaths"], case["h"], mode=mode, seed=seed, **rich)
        out = {"G": est.val, "B": est.B, "BB": est.BB}
        if case["mode"] == "replay":
            out["G_var"] = est.var
        return out
    if k == "lut":
        est = s["pd"].estimate(s["bvp"], case["npaths"], case["h"], seed=seed, **RICH)
        return {"G": est.val, "B": est.B, "BB": est.BB}
    if k == "circle":
        est = s["pd"].estimate(s["bvp"], case["npaths"], case["h"], seed=seed, adaptive_n=True,
                               npaths_max=case["npaths_max"], target_stderr=1e-3, **RICH)
        u, _ = s["pd"].solve_interface()
        return {"u": u, "G": est.val, "B": est.B, "BB": est.BB, "npaths": est.npaths}
    if k == "batch":
        bt = s["batch"]
        bt.run(case["npaths"], case["h"], seed=seed, richardson=True, dup_sum=True)
        got = [bt.result(i) for i in range(case["instances"])]
        return {"u": np.concatenate([g["u"] for g in got]), "B": np.concatenate([g["B"] for g in got])}
    if k == "semilinear":
        its = s["pd"].solve_semilinear(case["steps"], case["npaths"], case["h"], m=case["m"], seed=seed, **RICH)
        return [{"u": it["u"], "grid": it["grid"][2], "G": it["estimate"].val, "B": it["estimate"].B} for it in its]
    method = P.SOLVE_GMRES_FP32_IR if case["method"] == "gmres" else P.SOLVE_BICGSTAB_FP64
    return s["pd"].solve_interface(method)[0]


# --------------------------------------------------------------------------- what a pass cannot do without
def _tau(L):
    """Mean exit time (diffusion 1/2 sigma^2 = 1) of a layout's stencils, subdomain side L."""
    return 0.085 * L * L


def _steps(case, nsub, side):
    """Path steps per knot path: a Richardson pair takes two fine and one coarse step per h, and the per-knot step
    refines near the sides."""
    s = max(1.0, _tau(side / nsub) / case["h"])
    return 3.0 * s + 18.0 if case.get("richardson") else s


STEP_FLOPS = 60  # Box-Muller, coefficients, state update and exit test of one Euler step


def work(case):
    k = case["kind"]
    if k == "knot":
        n = 3 * case["gap_nodes"] + 3
        steps = case["npaths"] * _steps(case, 4, DOMAIN[case["problem"]][0])
        return {"bytes": 24 * 3 * n + 16 * n, "flops": steps * STEP_FLOPS + case["npaths"] * n * 10 + 3 * n ** 3}
    if k in ("solve", "estimate", "lut", "semilinear", "interface"):
        K = _knots(case["nsub"], case["nnode"])
        nnz = K * 8.5 * case["nnode"]
        if k == "interface":
            return {"bytes": 12 * nnz + 16 * K, "flops": 30 * 2 * nnz}
        side = DOMAIN[case["problem"]][0] if "problem" in case else 1.0
        c = dict(case, richardson=True) if k in ("lut", "semilinear") else case
        flops = K * case["npaths"] * _steps(c, case["nsub"], side) * STEP_FLOPS
        extra = 32 * case["table"] ** 2 if k == "lut" else 0
        if k == "estimate" and case["mode"] == "replay":
            flops += K * case["npaths"] * 2.0 * (2 * case["nnode"]) ** 2
        return {"bytes": 8 * nnz + 24 * K + extra, "flops": case.get("steps", 1) * (flops + 60 * nnz)}
    if k == "circle":
        K = 2 * case["rings"] * case["sectors"] * (case["nnode"] - 2)
        return {"bytes": 8 * K * 8 * case["nnode"] + 24 * K,
                "flops": K * 0.3 * case["npaths_max"] * STEP_FLOPS * 3 * min(400.0, 4e-3 / case["h"])}
    K = 2 * 60 * 25 * case["instances"]
    return {"bytes": 8 * K * 8 * 25 + 24 * K, "flops": K * case["npaths"] * 60.0 * STEP_FLOPS}


# --------------------------------------------------------------------------- the same in 64 bits
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _philox(pair, path, knot, instance, seed):
    """Philox-4x32-10 (Salmon et al., SC'11) on int64 tensors holding 32-bit words."""
    M = 0xFFFFFFFF
    c0 = torch.full_like(path, pair)
    c1, c2, c3 = path.clone(), knot.clone(), torch.full_like(path, instance)
    k0, k1 = seed & M, (seed >> 32) & M
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = ((p1 >> 32) & M) ^ c1 ^ k0, p1 & M, ((p0 >> 32) & M) ^ c3 ^ k1, p0 & M
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return c0, c1, c2, c3


def _normals(a, b):
    u0, u1 = (a.double() + 0.5) * 2.0 ** -32, (b.double() + 0.5) * 2.0 ** -32
    rho = torch.sqrt(-2.0 * torch.log(u0))
    return rho * torch.cos(2 * math.pi * u1), rho * torch.sin(2 * math.pi * u1)


def _problem64(name):
    """(coefficients at (x, y): sigma_x, sigma_y, b_x, b_y, c, f, u_x, u_y; solution) of 1/2 sum (sigma sigma^T)_ij
    u_ij + b.grad u + c u + f = 0."""
    r2 = math.sqrt(2.0)
    if name == "poisson":
        def coef(x, y):
            sx, cx, sy, cy = (torch.sin(math.pi * x), torch.cos(math.pi * x), torch.sin(math.pi * y),
                              torch.cos(math.pi * y))
            return r2, r2, 0.0, 0.0, 0.0, 2 * math.pi ** 2 * sx * cy, math.pi * cx * cy + y, x - math.pi * sx * sy
        return coef, lambda x, y: torch.sin(math.pi * x) * torch.cos(math.pi * y) + x * y
    if name == "helmholtz":
        a, b, c = 2.3, 1.7, -1.5

        def coef(x, y):
            sa, ca, sb, cb = torch.sin(a * x), torch.cos(a * x), torch.sin(b * y), torch.cos(b * y)
            return r2, r2, 0.0, 0.0, c, (a * a + b * b - c) * sa * cb, a * ca * cb, -b * sa * sb
        return coef, lambda x, y: torch.sin(a * x) * torch.cos(b * y)
    if name == "varcoef":
        def coef(x, y):
            s1, s2 = 1 + 0.5 * x * x, 1 + 0.5 * y * y
            e = torch.exp(x)
            ux, uy = e * torch.cos(2 * y), -2 * e * torch.sin(2 * y)
            c = -(1 + x * x + y * y)
            f = -(0.5 * (s1 * s1 * ux - 4 * s2 * s2 * ux) + y * ux - x * uy + c * (ux + 1))
            return s1, s2, y, -x, c, f, ux, uy
        return coef, lambda x, y: torch.exp(x) * torch.cos(2 * y) + 1

    k2, k3, k4, k5, k6, k7, w = 0.01, 0.02, 0.12, 0.05, 0.05, -0.12, 0.333

    def parts(x, y):
        return torch.sqrt(1 + k2 * x * x + k3 * y * y), k4 * x + k5 * y, k6 * x + k7 * y

    def coef(x, y):
        q, A, B = parts(x, y)
        sq, cq, sA, sB = torch.sin(q), torch.cos(q), torch.sin(A), torch.sin(B)
        T = torch.tanh(sA + sB)
        D = 1 - T * T

        def one(k, v, ka, kb):
            p = ka * torch.cos(A) + kb * torch.cos(B)
            first = cq * k * v / q + D * p
            second = (cq * (k / q - k * k * v * v / q ** 3) - sq * k * k * v * v / q ** 2 - 2 * T * D * p * p
                      - D * (ka * ka * sA + kb * kb * sB))
            return w * first, w * second
        ux, uxx = one(k2, x, k4, k6)
        uy, uyy = one(k3, y, k5, k7)
        return r2, r2, 0.0, 0.0, 0.0, -(uxx + uyy), ux, uy
    return coef, lambda x, y: 3 + w * (torch.sin(parts(x, y)[0]) + torch.tanh(torch.sin(parts(x, y)[1])
                                                                                 + torch.sin(parts(x, y)[2])))


def _exact_paths(problem, knots, npaths, h, seed, rich):
    """Every path of the knots: per level the weight, the exit's knot, side (-1: the boundary), side coordinate and
    Y, and per path (pair) its value.  knots: x, y, rect [n, 4], glob [n, 4] (N, S, E, W), word [n]."""
    coef, sol = _problem64(problem)
    t = lambda a, d=torch.float64: torch.as_tensor(np.asarray(a), dtype=d, device=_DEV)  # noqa: E731
    kx, ky, rects, globs, words = t(knots["x"]), t(knots["y"]), t(knots["rect"]), t(knots["glob"], torch.bool), t(
        knots["word"], torch.int64)
    n = len(kx)

    def distance(x, y, r):
        dx = (x - 0.5 * (r[:, 0] + r[:, 2])).abs() - 0.5 * (r[:, 2] - r[:, 0])
        dy = (y - 0.5 * (r[:, 1] + r[:, 3])).abs() - 0.5 * (r[:, 3] - r[:, 1])
        return dx, dy

    hk = torch.full_like(kx, h)
    if rich:  # the per-knot step: (distance / (2 * 0.5826 |N^T sigma|))^2 where that is smaller
        dx, dy = distance(kx, ky, rects)
        d = torch.maximum(dx, dy)
        c = coef(kx, ky)
        sg = torch.where(dx > dy, torch.as_tensor(c[0], device=_DEV), torch.as_tensor(c[1], device=_DEV)).double()
        hk = torch.where(d <= -1e-4, torch.minimum(hk, (d / (sg.abs() * 2 * 0.5826)) ** 2), hk)
    # levels: 0 the path (or the fine one), 1 the coarse one
    weight = [2.0, -1.0] if rich else [1.0]
    total = n * npaths
    value = torch.zeros(total, dtype=torch.float64, device=_DEV)
    exits = []
    ids = torch.arange(total, device=_DEV)
    state = [[ids] + [v.repeat_interleave(npaths) for v in (kx, ky)]
             + [torch.ones(total, dtype=torch.float64, device=_DEV)]
             + [torch.zeros(total, dtype=torch.float64, device=_DEV) for _ in range(2)] for _ in weight]

    def advance(lv, st, dw0, dw1, hh):
        """One step of every path of st, the exits taken out of it."""
        i, x, y, Y, Z, xi = st
        kn = i // npaths
        s0, s1, b0, b1, c, f, g0, g1 = coef(x, y)
        xi = xi - Y * (g0 * s0 * dw0 + g1 * s1 * dw1)
        Z = Z + f * Y * hh
        x = x + b0 * hh + s0 * dw0
        y = y + b1 * hh + s1 * dw1
        Y = Y + c * Y * hh
        r = rects[kn]
        dx, dy = distance(x, y, r)
        c = coef(x, y)
        sg = torch.where(dx > dy, torch.as_tensor(c[0], device=_DEV), torch.as_tensor(c[1], device=_DEV)).abs()
        out = ~(torch.maximum(dx, dy) < -0.5826 * sg * torch.sqrt(hh))
        o = out.nonzero()[:, 0]
        if len(o):
            r, k = r[o], kn[o]
            ex, ey, inx = x[o], y[o], dx[o] > dy[o]
            px = torch.where(inx, torch.where(ex > 0.5 * (r[:, 0] + r[:, 2]), r[:, 2], r[:, 0]),
                             torch.minimum(torch.maximum(ex, r[:, 0]), r[:, 2]))
            py = torch.where(inx, torch.minimum(torch.maximum(ey, r[:, 1]), r[:, 3]),
                             torch.where(ey > 0.5 * (r[:, 1] + r[:, 3]), r[:, 3], r[:, 1]))
            on = torch.stack([py == r[:, 3], py == r[:, 1], px == r[:, 2], px == r[:, 0]], 1)
            glob = (on & globs[k]).any(1)
            side = torch.where(on[:, 1], 1, torch.where(on[:, 0], 0, torch.where(on[:, 3], 3, 2)))
            side = torch.where(glob, torch.full_like(side, -1), side)
            along = torch.where((side == 0) | (side == 1), px, py)
            val = Z[o] + xi[o] + torch.where(glob, Y[o] * sol(px, py), torch.zeros_like(px))
            value.index_add_(0, i[o], weight[lv] * val)
            exits.append((k, side, along, weight[lv] * Y[o]))
        keep = (~out).nonzero()[:, 0]
        return [v[keep] for v in (i, x, y, Y, Z, xi)], keep

    pair = 0
    while any(len(st[0]) for st in state):
        if rich:
            # both levels of a pair read the increments of its block
            for lv in (0, 1):
                st = state[lv]
                if not len(st[0]):
                    continue
                kn = st[0] // npaths
                w = _philox(pair, st[0] % npaths, words[kn], 0, seed)
                hf = 0.5 * hk[kn]
                a, b = _normals(w[0], w[1]), _normals(w[2], w[3])
                sq = torch.sqrt(hf)
                if lv == 0:
                    st, keep = advance(0, st, sq * a[0], sq * a[1], hf)
                    if len(keep):
                        st, _ = advance(0, st, (sq * b[0])[keep], (sq * b[1])[keep], hf[keep])
                else:
                    st, _ = advance(1, st, sq * (a[0] + b[0]), sq * (a[1] + b[1]), 2 * hf)
                state[lv] = st
        else:
            st = state[0]
            kn = st[0] // npaths
            w = _philox(pair, st[0] % npaths, words[kn], 0, seed)
            hh = hk[kn]
            a, b = _normals(w[0], w[1]), _normals(w[2], w[3])
            sq = torch.sqrt(hh)
            st, keep = advance(0, st, sq * a[0], sq * a[1], hh)
            if len(keep):
                st, _ = advance(0, st, (sq * b[0])[keep], (sq * b[1])[keep], hh[keep])
            state[0] = st
        pair += 1
    ex = [torch.cat(v) for v in zip(*exits)]
    return value.reshape(n, npaths), ex


def _exact_rows(knots, npaths, ex, sides):
    """G's side weights per knot: {side: (indices, weights)} in the order N, S, E, W."""
    order = torch.argsort(ex[0], stable=True)
    ex = [v[order] for v in ex]
    bounds = torch.searchsorted(ex[0].contiguous(), torch.arange(len(knots["x"]) + 1, device=_DEV)).tolist()
    inv, rows = {}, []
    for k in range(len(knots["x"])):
        sl = slice(bounds[k], bounds[k + 1])
        sd, al, wy = ex[1][sl], ex[2][sl], ex[3][sl]
        row = []
        for d in range(4):
            idx, t, c = sides[k][d]
            if not len(idx):
                continue
            t = torch.as_tensor(t, dtype=torch.float64, device=_DEV)
            key = (len(t), round(c, 12), round(float(t[-1] - t[0]), 12))
            if key not in inv:
                inv[key] = torch.linalg.inv(torch.exp(-((t[:, None] - t[None, :]) / c) ** 2))
            m = sd == d
            S = (torch.exp(-((t[None, :] - al[m][:, None]) / c) ** 2) * wy[m][:, None]).sum(0)
            row.append((idx, (-(inv[key].T @ S) / npaths).cpu().numpy()))
        rows.append(row)
    return rows


def _exact_layout(case, s):
    """The estimate of a layout's knots: G values on its rows, B and BB."""
    pd, N = s["pd"], case["npaths"]
    side, lo = DOMAIN[case["problem"]]
    hi = lo + side
    dist = np.minimum(np.minimum(pd.x - lo, hi - pd.x), np.minimum(pd.y - lo, hi - pd.y))
    mc = np.flatnonzero(dist > 1e-9 * side)
    knots = {"x": pd.x[mc], "y": pd.y[mc], "word": mc, "rect": [], "glob": []}
    sides = []
    for k in mc:
        rect, kinds, idx = pd.stencil(int(k))
        knots["rect"].append(rect)
        knots["glob"].append([abs(rect[3] - hi) < 1e-9, abs(rect[1] - lo) < 1e-9, abs(rect[2] - hi) < 1e-9,
                              abs(rect[0] - lo) < 1e-9])
        sides.append([(i, (pd.x if d < 2 else pd.y)[i], pd.fac[kinds[d]] if kinds[d] >= 0 else 1.0)
                      for d, i in enumerate(idx)])
    rich = bool(case.get("richardson"))
    value, ex = _exact_paths(case["problem"], knots, N, case["h"], s["seed"], rich)
    val = np.zeros(pd.nnz)
    for k, row in zip(mc, _exact_rows(knots, N, ex, sides)):
        a, b = pd.row_ptr[k], pd.row_ptr[k + 1]
        for idx, w in row:
            at = a + np.searchsorted(pd.col[a:b], idx)
            val[at] = val[at] + w if rich else w  # a knot of two sides: summed, or the last side's
    sol = _problem64(case["problem"])[1]
    B = sol(torch.as_tensor(pd.x), torch.as_tensor(pd.y)).numpy().copy()
    BB = B * B
    B[mc], BB[mc] = value.mean(1).cpu().numpy(), (value ** 2).mean(1).cpu().numpy()
    return val, B, BB


def _dense(pd, val, B):
    A = torch.eye(pd.K, dtype=torch.float64, device=_DEV)
    rows = torch.as_tensor(np.repeat(np.arange(pd.K), np.diff(pd.row_ptr)), device=_DEV)
    A.index_put_((rows, torch.as_tensor(pd.col, device=_DEV).long()), torch.as_tensor(val, device=_DEV), accumulate=True)
    return torch.linalg.solve(A, torch.as_tensor(B, device=_DEV)).cpu().numpy()


def exact(case, seed):
    """What run() returns, in 64 bits: the paths of the same Philox streams, the RBF weights and the interface system
    solved densely.  The tables, the adaptive path counts, the batches, the outer loop and the larger layouts would
    take too long, and G's variances and the interiors are the library's own discretisations: no value for these."""
    k = case["kind"]
    if k == "knot":
        s = prepare(case, seed)
        st, N = s["stencil"], case["npaths"]
        knots = {"x": [s["x0"][0]], "y": [s["x0"][1]], "rect": [st.stencil_parameters],
                 "glob": [[False, True, False, False]], "word": [7]}
        sides = [[(st.index[d], st.x[d] if d in "NS" else st.y[d], st.c2[d]) for d in "NSEW"]]
        value, ex = _exact_paths(case["problem"], knots, N, case["h"], s["seed"], case["richardson"])
        row = _exact_rows(knots, N, ex, sides)[0]
        idx = np.concatenate([r[0] for r in row])
        G = np.concatenate([r[1] for r in row])
        order = np.argsort(idx)
        return {"G": G[order], "G_j": idx[order].astype(np.int32), "B": float(value.mean()),
                "BB": float((value ** 2).mean())}
    if k in ("solve", "estimate"):
        paths = _knots(case["nsub"], case["nnode"]) * case["npaths"]
        if paths > 8e6 or paths * _steps(case, case["nsub"], DOMAIN[case["problem"]][0]) > 6e8:
            return None
        s = prepare(case, seed)
        val, B, BB = _exact_layout(case, s)
        out = {"G": val, "B": B, "BB": BB}
        if k == "solve":
            out["u"] = _dense(s["pd"], val, B)
            out["G_var"] = None
            out["interior"] = None
        else:
            out["G_var"] = None
        return out
    if k == "interface":
        s = prepare(case, seed)
        return _dense(s["pd"], s["est"].val, s["est"].B)
    return None
