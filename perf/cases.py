"""Performance cases of the Feynman-Kac library: what its users call, at the sizes they call it.

A case is one of seven calls:

  points    Context.solve_points / FeynmanKacSolverGPU.Solve_OMP_Analytic: node estimates at given points
  batch     Context.solve_points_multi: many disk problems of uneven path counts and steps in one launch
  assembly  fk_assemble: the G/B system of a square-patch mesh, plain or with the learned control variate
  rounds    fk_assembly_begin / round / end: the adaptive assembly, device-resident sums
  circles   fk_assemble on the reference's circle mesh with pseudospectral interior rows (its serial driver)
  disks     solve_disks_ps: the pseudospectral rows alone
  train     fk_mlp_train + fit_output + build_table: the control variate's network

Sizes are those of the repository's workloads and benchmark, or lie between them.  Every input comes from
the seed: the points, the disks, the Philox key and stream, the training samples.
"""
import math

import numpy as np
import torch

from spac_gb300 import fk

PROBLEM = {"franke": fk.FRANKE, "aniso": fk.ANISO}
KNN, ENLARGE = 20, 0.25
DRIVER_DOM = (0.0, 0.0, 1.25, 1.25)  # the serial driver's square


def listed():
    return [
        # the drop-in call: one node of the reference's loop, its default path count (latency)
        dict(name="point_fp64", kind="points", problem="franke", precision=64, cv="none", n=1, paths=1000, h=1e-3),
        # a few nodes with the exact-gradient control variate, odd counts (checks against an exact solution)
        dict(name="points_cv_fp64", kind="points", problem="aniso", precision=64, cv="exact", n=37, paths=1501, h=5e-4),
        # the pilot of the learned control variate: a collocation lattice of short FP32 solves
        dict(name="points_pilot_fp32", kind="points", problem="aniso", precision=32, cv="none", n=576, paths=300, h=1e-3),
        # 32 x 32 Franke nodes in FP64: the point-solve benchmark
        dict(name="points_grid_fp64", kind="points", problem="franke", precision=64, cv="none", n=1024, paths=10000, h=1e-3),
        # 16 disks of uneven radius, 256 nodes each, paths log-uniform in 1e3..1e5, two steps
        dict(name="batch_disks_fp32", kind="batch", precision=32, n_bvp=16, nodes=256, scale=1.0),
        # the headline: 8 x 8 subdomains, 20000 paths per item
        dict(name="assembly_fp32", kind="assembly", precision=32, cv="none", n_sub=8, side=31, eps=3.0, paths=20000, h=5e-4),
        # the same system in FP64, the reference's arithmetic, fewer paths
        dict(name="assembly_fp64", kind="assembly", precision=64, cv="none", n_sub=8, side=31, eps=1.0, paths=2000, h=5e-4),
        # the learned control variate's run: few paths per item at a small step
        dict(name="assembly_learned_fp32", kind="assembly", precision=32, cv="learned", n_sub=8, side=31, eps=1.0, paths=734, h=5e-5),
        # the adaptive assembly: two pilot rounds and one uneven round, then the rows
        dict(name="rounds_fp32", kind="rounds", n_sub=16, side=31, eps=3.0, paths=256, h=2.5e-4),
        # the reference's serial driver: perimeter circles by paths at h = 1e-5, interior ones by collocation
        dict(name="circles_fp64", kind="circles", n_side=4, nodes=44, n_radial=43, paths=1000, h=1e-5),
        # interior-circle rows of a 32 x 32 circle layout
        dict(name="disks_fp64", kind="disks", problem="franke", n=900, n_circle=44, n_radial=43, n_inner=44, radii="equal"),
        # training, output refit and gradient table of one network
        dict(name="train_table", kind="train", samples=4096, steps=50, batch=4096, table=256),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["points", "points", "points", "batch", "assembly", "assembly", "rounds", "circles", "disks", "train"])
    if kind == "points":
        precision = rng.choice([64, 32])
        n = int(round(_log(rng, 1, 1200)))
        paths = int(round(_log(rng, 100, min(2e4, (6e6 if precision == 64 else 3e7) / n))))
        return dict(kind=kind, problem=rng.choice(["franke", "aniso"]), precision=precision,
                    cv=rng.choice(["none", "none", "exact"]), n=n, paths=paths, h=_log(rng, 3e-4, 4e-3))
    if kind == "batch":
        return dict(kind=kind, precision=rng.choice([64, 32, 32]), n_bvp=rng.randint(2, 16),
                    nodes=int(round(_log(rng, 5, 100))), scale=_log(rng, 0.02, 0.1))
    if kind == "assembly":
        precision, cv = rng.choice([64, 32, 32]), rng.choice(["none", "none", "learned"])
        n_sub, side = rng.randint(2, 8), rng.choice([15, 23, 31])
        budget = 1.5e7 if precision == 64 else 1.5e8
        paths = int(round(_log(rng, 100, max(200, min(2e4, budget / (n_sub * n_sub * 4 * side))))))
        return dict(kind=kind, precision=precision, cv=cv, n_sub=n_sub, side=side, eps=rng.choice([1.0, 3.0]),
                    paths=paths, h=_log(rng, 1e-4, 1e-3))
    if kind == "rounds":
        return dict(kind=kind, n_sub=rng.randint(3, 15), side=rng.choice([23, 31]), eps=rng.choice([1.0, 3.0]),
                    paths=rng.randint(64, 512), h=_log(rng, 1e-4, 1e-3))
    if kind == "circles":
        return dict(kind=kind, n_side=rng.randint(3, 5), nodes=2 * rng.randint(8, 24), n_radial=2 * rng.randint(7, 21) + 1,
                    paths=int(round(_log(rng, 100, 1500))), h=_log(rng, 5e-5, 1e-3))
    if kind == "disks":
        return dict(kind=kind, problem=rng.choice(["franke", "franke", "aniso"]), n=int(round(_log(rng, 1, 400))),
                    n_circle=2 * rng.randint(6, 24), n_radial=2 * rng.randint(4, 21) + 1, n_inner=rng.randint(3, 60),
                    radii=rng.choice(["equal", "uneven"]))
    return dict(kind=kind, samples=int(round(_log(rng, 400, 8000))), steps=int(round(_log(rng, 10, 200))),
                batch=64 * rng.randint(8, 64), table=rng.choice([64, 128, 256]))


# ---------------------------------------------------------------- inputs ----
def _points_in(case, seed):
    rng = np.random.default_rng(seed)
    return np.ascontiguousarray(rng.uniform(0.02, 0.98, (case["n"], 2)))


def _batch_in(case, seed):
    """Disks (radius, cx, cy) 2.5 apart and their nodes: disk of each node, xy, paths, h."""
    rng = np.random.default_rng(seed)
    nb, per = case["n_bvp"], case["nodes"]
    R = rng.uniform(0.25, 1.0, nb)
    disks = np.stack([R, 2.5 * np.arange(nb), np.zeros(nb)], 1)
    of = np.repeat(np.arange(nb), per)
    r = disks[of, 0] * np.sqrt(rng.uniform(0, 1, len(of)))
    t = rng.uniform(0, 2 * np.pi, len(of))
    xy = np.stack([disks[of, 1] + r * np.cos(t), disks[of, 2] + r * np.sin(t)], 1)
    paths = np.maximum(1, np.round(case["scale"] * np.exp(rng.uniform(math.log(1e3), math.log(1e5), len(of)))))
    return disks, of, np.ascontiguousarray(xy), paths.astype(np.uint32), rng.choice([1e-3, 5e-4], len(of))


def _disks_in(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    m = int(math.ceil(math.sqrt(n)))
    H = 1.0 / (m + 1)
    R = np.full(n, H / math.sqrt(2)) if case["radii"] == "equal" else H * rng.uniform(0.4, 0.7, n)
    theta0 = float(rng.uniform(0.05, 0.25))
    out = []
    for d in range(n):
        c = np.array([(d // m + 1) * H, (d % m + 1) * H])
        r = 0.95 * R[d] * np.sqrt(rng.random(case["n_inner"]))
        a = 2 * np.pi * rng.random(case["n_inner"])
        out.append(dict(cx=float(c[0]), cy=float(c[1]), radius=float(R[d]), theta0=theta0, n_circle=case["n_circle"],
                        n_radial=case["n_radial"],
                        periph_theta=theta0 + 2 * np.pi * np.arange(case["n_circle"]) / case["n_circle"],
                        inner_xy=np.stack([c[0] + r * np.cos(a), c[1] + r * np.sin(a)], 1)))
    return out


def _samples_in(n, seed):
    """Training samples of the network: noisy node estimates of u on the unit square."""
    rng = np.random.default_rng(seed)
    xy = rng.uniform(0, 1, (n, 2))
    e = [np.exp(v) for v in _exponents(xy[:, 0], xy[:, 1])]
    u = (0.75 * e[0] + 0.75 * e[1] + 0.5 * e[2] - 0.2 * e[3]) * (1 + xy[:, 0] * xy[:, 1])
    return np.ascontiguousarray(xy), np.ascontiguousarray(u + 0.02 * rng.standard_normal(n))


def _network(ctx, samples, seed, steps, table):
    """A user's learned control variate: one region, trained, refitted and tabulated."""
    rect = np.array([0.0, 0.0, 1.0, 1.0])
    mid = fk.C.c_int()
    ctx.check(ctx.L.fk_mlp_create(ctx.h, 1, rect.ctypes.data_as(fk._dp), 99, fk.C.byref(mid)))
    xy, t = _samples_in(samples, seed)
    _train(ctx, mid.value, xy, t, steps, 4096, table)
    return mid.value


def _train(ctx, mid, xy, t, steps, batch, table):
    px, pt = xy.ctypes.data_as(fk._dp), t.ctypes.data_as(fk._dp)
    ctx.check(ctx.L.fk_mlp_train(ctx.h, mid, len(t), px, pt, None, steps, batch, 1e-2, 5, None))
    ctx.check(ctx.L.fk_mlp_fit_output(ctx.h, mid, len(t), px, pt, None, 1e-6))
    ctx.check(ctx.L.fk_mlp_build_table(ctx.h, mid, table))


def _pinned(n):
    return torch.empty(max(int(n), 1), dtype=torch.float64, pin_memory=True)


class _State:
    def __init__(self, case, seed):
        self.case = case
        self.stream = seed % 1000 + 1
        self.ctx = fk.Context(0, seed=seed + 1000)

    def __del__(self):
        if getattr(self, "ctx", None) is not None:
            self.ctx.close()


def prepare(case, seed):
    s = _State(case, seed)
    ctx, kind = s.ctx, case["kind"]
    s.prec = fk.FP64 if case.get("precision", 64) == 64 else fk.FP32
    if kind == "points":
        s.xy = _points_in(case, seed)
        s.bvp = ctx.register_bvp(PROBLEM[case["problem"]], cv=fk.CV_EXACT if case["cv"] == "exact" else fk.CV_NONE)
        s.solver = fk.FeynmanKacSolverGPU(ctx, s.prec)
    elif kind == "batch":
        disks, of, s.xy, s.paths, s.h = _batch_in(case, seed)
        ids = [ctx.register_bvp(fk.DISK, dom=tuple(d), prob=(d[1], d[2], d[0], 0.0)) for d in disks]
        s.ids = np.array(ids, dtype=np.int32)[of]
    elif kind == "assembly":
        s.mesh = ctx.mesh_square_patches((0, 0, 1, 1), case["n_sub"], case["side"], ENLARGE, case["eps"], KNN)
        info = ctx.mesh_info(s.mesh)
        s.val, s.B = _pinned(info["nnz"]), _pinned(info["n_rows"])
        if case["cv"] == "learned":
            s.bvp = ctx.register_bvp(fk.ANISO, cv=fk.CV_MLP, mlp_id=_network(ctx, 576, seed, 10, 128))
        else:
            s.bvp = ctx.register_bvp(fk.ANISO)
    elif kind == "rounds":
        s.mesh = ctx.mesh_square_patches((0, 0, 1, 1), case["n_sub"], case["side"], ENLARGE, case["eps"], KNN)
        info = ctx.mesh_info(s.mesh)
        n = info["n_items"]
        s.out = {"val": _pinned(info["nnz"]).numpy(), "B": _pinned(info["n_rows"]).numpy(), "item_B": _pinned(n).numpy()}
        s.stats = _pinned(n * len(fk.STAT_FIELDS))
        s.out["item_stats"] = (fk.Stats * n).from_address(s.stats.data_ptr())
        s.plain = ctx.register_bvp(fk.FRANKE)
        s.learned = ctx.register_bvp(fk.FRANKE, cv=fk.CV_MLP, mlp_id=_network(ctx, 1024, seed, 10, 128))
        rng = np.random.default_rng(seed)
        s.pilot = np.full(n, case["paths"], dtype=np.uint32)
        s.of = np.where(rng.random(n) < 0.8, s.learned, s.plain).astype(np.int32)
        s.more = np.round(case["paths"] * np.exp(rng.uniform(-1, 3, n))).astype(np.uint32) * (rng.random(n) < 0.9)
        s.more = s.more.astype(np.uint32)
    elif kind == "circles":
        s.mesh = ctx.mesh_circles(DRIVER_DOM, case["n_side"], 1.0, 0.1428, case["nodes"])
        ctx.mesh_set_disk_solver(s.mesh, case["n_radial"])
        s.bvp = ctx.register_bvp(fk.FRANKE, dom=DRIVER_DOM)
    elif kind == "disks":
        s.disks = _disks_in(case, seed)
        s.bvp = ctx.register_bvp(PROBLEM[case["problem"]])
    else:
        rect = np.array([0.0, 0.0, 1.0, 1.0])
        mid = fk.C.c_int()
        ctx.check(ctx.L.fk_mlp_create(ctx.h, 1, rect.ctypes.data_as(fk._dp), seed, fk.C.byref(mid)))
        s.mid = mid.value
        s.xy, s.t = _samples_in(case["samples"], seed)
        n = fk.C.c_int()
        ctx.check(ctx.L.fk_mlp_num_params(ctx.h, s.mid, fk.C.byref(n)))
        s.p0 = np.zeros(n.value, dtype=np.float32)
        ctx.check(ctx.L.fk_mlp_get_params(ctx.h, s.mid, s.p0.ctypes.data_as(fk._fp)))
        s.p1 = np.zeros_like(s.p0)
        s.tab = np.zeros((case["table"], case["table"], 2), dtype=np.float32)
    return s


def run(s):
    ctx, case, kind = s.ctx, s.case, s.case["kind"]
    ctx.set_stream(s.stream)  # the same random stream every pass
    if kind == "points":
        if case["n"] == 1 and case["cv"] == "none":
            f = s.solver.Solve_OMP_Analytic(s.xy[0], case["paths"], case["h"], 0.0, s.bvp)
            return {k: getattr(f, k) for k in ("phi", "phiphi", "phi_VR", "phiphi_VR", "xi", "xixi", "xiphi", "APL", "RNGC")}
        return ctx.solve_points(s.bvp, s.xy, case["paths"], case["h"], s.prec)
    if kind == "batch":
        return ctx.solve_points_multi(s.ids, s.xy, s.paths, s.h, s.prec)
    if kind == "assembly":
        ptr = [fk.C.cast(t.data_ptr(), fk._dp) for t in (s.val, s.B)]
        ctx.check(ctx.L.fk_assemble(ctx.h, s.mesh, s.bvp, case["paths"], None, case["h"], s.prec, ptr[0], ptr[1], None, None, None))
        return {"val": s.val, "B": s.B}
    if kind == "rounds":
        ctx.assembly_begin(s.mesh)
        v1 = ctx.assembly_round(s.mesh, s.learned, s.pilot, case["h"], fk.FP32)
        v2 = ctx.assembly_round(s.mesh, s.plain, s.pilot, case["h"], fk.FP32)
        v3 = ctx.assembly_round(s.mesh, s.plain, s.more, case["h"], fk.FP32, bvp_of_item=s.of)
        r = ctx.assembly_end(s.mesh, item_G=False, out=s.out)
        return {"val": r["val"], "B": r["B"], "item_B": r["item_B"], "stats": s.stats, "var": [v1, v2, v3]}
    if kind == "circles":
        r = ctx.assemble(s.mesh, s.bvp, case["paths"], case["h"], fk.FP64, items=False)
        return {"val": r["val"], "B": r["B"]}
    if kind == "disks":
        rows = ctx.solve_disks_ps(s.bvp, s.disks)
        return {"G": np.concatenate([g.ravel() for g, _ in rows]), "B": np.concatenate([b for _, b in rows])}
    ctx.check(ctx.L.fk_mlp_set_params(ctx.h, s.mid, s.p0.ctypes.data_as(fk._fp)))
    _train(ctx, s.mid, s.xy, s.t, case["steps"], case["batch"], case["table"])
    ctx.check(ctx.L.fk_mlp_get_params(ctx.h, s.mid, s.p1.ctypes.data_as(fk._fp)))
    g = fk.C.c_int()
    ctx.check(ctx.L.fk_mlp_get_table(ctx.h, s.mid, fk.C.byref(g), s.tab.ctypes.data_as(fk._fp)))
    return {"params": s.p1, "table": s.tab}


# ------------------------------------------------------------------ work ----
# FP operations a path-step cannot do without (FMA = 2): the coefficients at the point, the normal pair,
# the sums, the Euler update and the distance to the boundary.
STEP_FLOPS = {"franke": 110, "aniso": 174}


def _exit_time(xy, rect):
    """Mean exit time of sqrt(2) W from a rectangle (a few terms of its sine series)."""
    ax, ay = rect[2] - rect[0], rect[3] - rect[1]
    u, v = (xy[..., 0] - rect[0]) / ax, (xy[..., 1] - rect[1]) / ay
    t = np.zeros(np.shape(u))
    for i in range(1, 40, 2):
        for j in range(1, 40, 2):
            lam = math.pi ** 2 * ((i / ax) ** 2 + (j / ay) ** 2)
            t += 16 / (math.pi ** 2 * i * j * lam) * np.sin(math.pi * i * u) * np.sin(math.pi * j * v)
    return t


def _steps(t, h):
    # the path overshoots the boundary by about 0.58 sqrt(2 h) and the exit rule shifts it back: at least one step
    return 1.0 + t / h


def work(case):
    kind = case["kind"]
    if kind == "points":
        t = _exit_time(_points_in(case, 1), (0.0, 0.0, 1.0, 1.0))
        return {"bytes": case["n"] * (28 + 128), "flops": STEP_FLOPS[case["problem"]] * case["paths"] * float(_steps(t, case["h"]).sum())}
    if kind == "batch":
        disks, of, xy, paths, h = _batch_in(case, 1)
        r2 = (xy[:, 0] - disks[of, 1]) ** 2 + (xy[:, 1] - disks[of, 2]) ** 2
        return {"bytes": len(of) * (32 + 128), "flops": STEP_FLOPS["franke"] * float((paths * _steps((disks[of, 0] ** 2 - r2) / 4, h)).sum())}
    if kind in ("assembly", "rounds"):
        M = _mesh64(case)
        lo, hi = (np.array(M["rects"])[M["pat"]].reshape(-1, 2, 2)[:, i] for i in (0, 1))
        t = _exit_time((M["xy"][M["row"]] - lo) / (hi - lo), (0.0, 0.0, 1.0, 1.0)) * (hi - lo)[:, 0] ** 2
        paths = case["paths"] * (1 if kind == "assembly" else 2 + 4.1)  # (rounds: the uneven one averages 4.1 pilots)
        return {"bytes": len(t) * 104 + 12 * len(M["val"]),
                "flops": STEP_FLOPS["aniso" if kind == "assembly" else "franke"] * paths * float(_steps(t, case["h"]).sum())}
    if kind == "circles":
        n_side, nodes = case["n_side"], case["nodes"]
        r = 1.25 / (n_side - 1) / math.sqrt(2)
        fk_rows, ps_rows = 4 * (n_side - 1) * nodes * 0.44, (n_side - 2) ** 2 * nodes * 1.0
        return {"bytes": (fk_rows + ps_rows) * nodes * 12,
                "flops": STEP_FLOPS["franke"] * fk_rows * case["paths"] * _steps(r * r / 12, case["h"]) + ps_rows * nodes * nodes * 2}
    if kind == "disks":
        n, nc, half, ni = case["n"], case["n_circle"], (case["n_radial"] + 1) // 2, case["n_inner"]
        rows = n * ni
        one = (nc // 2 + 1) * 2 * half ** 3
        return {"bytes": 8 * rows * (nc + 3), "flops": one * (1 if case["radii"] == "equal" else n) + rows * nc * (nc + 2) * 2}
    per = 2 * (2 * 64 + 2 * 64 * 64 + 64)
    return {"bytes": 24 * case["samples"] + 8 * case["table"] ** 2,
            "flops": 3 * per * case["steps"] * case["batch"] + (per + 2 * 65 * 66 / 2) * case["samples"] + 2 * per * case["table"] ** 2}


# ----------------------------------------------------------------- exact ----
# The same paths in plain 64-bit torch: Philox4x32-10, Box-Muller, Euler steps, the shifted exit rule.
def _exponents(x, y):
    return (-0.25 * ((9 * x - 2) ** 2 + (9 * y - 2) ** 2), -((9 * x + 1) ** 2) / 49 - 0.1 * (9 * y + 1),
            -0.25 * ((9 * x - 7) ** 2 + (9 * y - 3) ** 2), -((9 * x - 4) ** 2) - (9 * y - 7) ** 2)


def _franke64(x, y):
    """u, u_x, u_y and the Laplacian of the Franke function."""
    e = [torch.exp(v) for v in _exponents(x, y)]
    a, b, c = 9 * x - 2, 9 * y - 2, 9 * x + 1
    p, q, r, t = 9 * x - 7, 9 * y - 3, 9 * x - 4, 9 * y - 7
    u = 0.75 * e[0] + 0.75 * e[1] + 0.5 * e[2] - 0.2 * e[3]
    ux = -3.375 * a * e[0] - 27 / 98 * c * e[1] - 2.25 * p * e[2] + 3.6 * r * e[3]
    uy = -3.375 * b * e[0] - 0.675 * e[1] - 2.25 * q * e[2] + 3.6 * t * e[3]
    lap = ((15.1875 * (a * a + b * b) - 60.75) * e[0] + (486 / 4802 * c * c - 243 / 98 + 243 / 400) * e[1] +
           (10.125 * (p * p + q * q) - 40.5) * e[2] + (64.8 - 64.8 * (r * r + t * t)) * e[3])
    return u, ux, uy, lap


def _philox64(k, path, item, stream, key):
    m = 0xFFFFFFFF
    c = [k, path, item, torch.full_like(k, stream)]
    k0, k1 = key & m, (key >> 32) & m
    for _ in range(10):
        a, b = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57  # (the product's 64 bits, in two's complement)
        c = [((b >> 32) & m) ^ c[1] ^ k0, b & m, ((a >> 32) & m) ^ c[3] ^ k1, a & m]
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    return c[0], c[1]


def _rect64(x, y, r):
    """Signed distance to a rectangle and the nearest boundary point."""
    cx, cy = 0.5 * (r[0] + r[2]), 0.5 * (r[1] + r[3])
    hx, hy = r[2] - cx, r[3] - cy
    ox, oy = (x - cx).abs() - hx, (y - cy).abs() - hy
    bx, by = torch.where(x > cx, hx, -hx) + cx, torch.where(y > cy, hy, -hy) + cy
    both = (ox > 0) & (oy > 0)
    side_x = torch.where((ox <= 0) & (oy <= 0), ox > oy, ox > 0)
    d = torch.where(both, torch.sqrt(ox * ox + oy * oy), torch.where(side_x, ox, oy))
    return d, torch.where(side_x | both, bx, x), torch.where(side_x & ~both, y, by)


def _walk64(problem, x0, y0, h, paths, stream, key, cv=False, disk=None, sub=None, dom=(0.0, 0.0, 1.0, 1.0), item0=None):
    """All paths of the items; yields (item, exit x, exit y, Y, Z, xi, steps, domain exit) of those that stopped."""
    dev, f8 = x0.device, torch.float64
    n = len(x0)
    ids = torch.arange(n, device=dev) if item0 is None else item0
    ends = torch.cumsum(paths, 0)
    total, at, room = int(ends[-1]), 0, 6_000_000
    hx, hs = h, torch.sqrt(h)
    it = torch.empty(0, dtype=torch.int64, device=dev)
    pa, k = it.clone(), it.clone()
    x, y, Y, Z, xi = (torch.empty(0, dtype=f8, device=dev) for _ in range(5))
    while at < total or len(it):
        if at < total and len(it) < room // 2:
            g = torch.arange(at, min(total, at + room - len(it)), device=dev)
            at += len(g)
            i = torch.searchsorted(ends, g, right=True)
            one = torch.ones(len(g), dtype=f8, device=dev)
            it, pa, k = torch.cat([it, i]), torch.cat([pa, g - (ends[i] - paths[i])]), torch.cat([k, torch.zeros_like(g)])
            x, y, Y, Z, xi = (torch.cat(v) for v in ((x, x0[i]), (y, y0[i]), (Y, one), (Z, 0 * one), (xi, 0 * one)))
        H, S = hx[it], hs[it]
        w0, w1 = _philox64(k, pa, ids[it], stream, key)
        rad = torch.sqrt(-2.0 * torch.log((w0.to(f8) + 0.5) * 2.0 ** -32))
        ang = 2 * math.pi * ((w1.to(f8) + 0.5) * 2.0 ** -32)
        dx, dy = S * (rad * torch.cos(ang)), S * (rad * torch.sin(ang))
        if problem == "aniso":
            u, ux, uy, lap = _franke64(x, y)
            q = 1 + x * y
            lap = lap * q + 2 * (ux * y + uy * x)
            u, ux, uy = u * q, ux * q + u * y, uy * q + u * x
            a = 1 + 0.5 * torch.sin(2 * math.pi * x) * torch.sin(2 * math.pi * y)
            s, c, bx, by = torch.sqrt(2 * a), -(1 + x * x + y * y), y - 0.5, 0.5 - x
            f = -(a * lap + bx * ux + by * uy + c * u)
        else:
            s, c, bx, by = 1.41421356237, 0.0, 0.0, 0.0
            if disk is None:
                u, ux, uy, lap = _franke64(x, y)
                f = -lap
            else:
                D = disk[it]
                inv = 1 / (2 * D[:, 0])
                f = -_franke64((x - D[:, 1]) * inv + 0.5, (y - D[:, 2]) * inv + 0.5)[3] * inv * inv
        Z = Z + f * Y * H
        if cv:
            xi = xi - Y * s * (ux * dx + uy * dy)
        Y = Y + c * Y * H
        x, y, k = x + (bx * H + s * dx), y + (by * H + s * dy), k + 1
        if disk is None:
            d, ex, ey = _rect64(x, y, dom)
        else:
            D = disk[it]
            r = torch.sqrt((x - D[:, 1]) ** 2 + (y - D[:, 2]) ** 2).clamp_min(5e-4)
            d, ex, ey = r - D[:, 0], (x - D[:, 1]) / r * D[:, 0] + D[:, 1], (y - D[:, 2]) / r * D[:, 0] + D[:, 2]
        won = torch.ones_like(it, dtype=torch.bool)
        if sub is not None:
            e, sx, sy = _rect64(x, y, sub)
            won = d >= e
            d, ex, ey = torch.where(won, d, e), torch.where(won, ex, sx), torch.where(won, ey, sy)
        if problem == "aniso":
            qx, qy = torch.where(d < 0, x, ex), torch.where(d < 0, y, ey)
            s = torch.sqrt(2 + torch.sin(2 * math.pi * qx) * torch.sin(2 * math.pi * qy))
        out = ~(d < -0.5826 * s * S)
        o = out.nonzero()[:, 0]
        if len(o):
            yield it[o], ex[o], ey[o], Y[o], Z[o], xi[o], k[o], won[o]
            i = (~out).nonzero()[:, 0]
            it, pa, k, x, y, Y, Z, xi = (v[i] for v in (it, pa, k, x, y, Y, Z, xi))


def _g64(problem, x, y):
    u = _franke64(x, y)[0]
    return u * (1 + x * y) if problem == "aniso" else u


def _stats64(problem, x0, y0, h, paths, stream, key, cv=False, disk=None):
    n = len(x0)
    S = {k: torch.zeros(n, dtype=torch.float64, device=x0.device) for k in ("s", "s2", "v", "v2", "x", "x2", "xs", "k")}
    for it, ex, ey, Y, Z, xi, k, _ in _walk64(problem, x0, y0, h, paths, stream, key, cv, disk):
        if disk is None:
            g = _g64(problem, ex, ey)
        else:
            D = disk[it]
            g = _g64(problem, (ex - D[:, 1]) / (2 * D[:, 0]) + 0.5, (ey - D[:, 2]) / (2 * D[:, 0]) + 0.5)
        s = Z + Y * g
        for name, v in (("s", s), ("s2", s * s), ("v", s + xi), ("v2", (s + xi) ** 2), ("x", xi), ("x2", xi * xi), ("xs", xi * s), ("k", k.double())):
            S[name].index_add_(0, it, v)
    N = paths.double()
    alias = 2 * (S["x"] + S["x2"]) / N
    return dict(phi=S["s"] / N, phiphi=S["s2"] / N, phi_VR=S["v"] / N, phiphi_VR=S["v2"] / N, xi=alias, xixi=alias, xiphi=S["xs"] / N,
                APL=h * S["k"] / N, RNGC=4 * S["k"], B=S["v"] / N, n_paths=N, n_domain_exits=N, n_capped=0 * N, xi_mean=S["x"] / N,
                xi_sq_mean=S["x2"] / N, mean_steps=S["k"] / N)


def _mesh64(case):
    """The square-patch mesh: rings, items (row, patch) and the CSR pattern with its start values."""
    n, side, H = case["n_sub"], case["side"], 1.0 / case["n_sub"]
    sp = (1 + 2 * ENLARGE) * H / (side + 1)
    q = np.arange(1, side + 1) * sp
    full = np.ones(side)
    rings, rects, closed, first = [], [], [], [0]
    for a in range(n):
        for b in range(n):
            r = ((a - ENLARGE) * H, (b - ENLARGE) * H, (a + 1 + ENLARGE) * H, (b + 1 + ENLARGE) * H)
            ring = np.concatenate([np.stack(v, 1) for v in ((r[0] + q, r[1] * full), (r[2] * full, r[1] + q),
                                                             (r[2] - q, r[3] * full), (r[0] * full, r[3] - q))])
            keep = ((ring > 1e-12) & (ring < 1 - 1e-12)).all(1)
            if not keep.all():
                start = int(np.nonzero(~keep & np.roll(keep, -1))[0][0]) + 1
                ring, keep = np.roll(ring, -start, 0), np.roll(keep, -start)
            rings.append(ring[keep])
            rects.append(r)
            closed.append(bool(keep.all()))
            first.append(first[-1] + int(keep.sum()))
    xy = np.concatenate(rings)
    own = np.repeat(np.arange(n * n), np.diff(first))
    inner = []
    for s, r in enumerate(rects):
        ins = (xy[:, 0] > r[0] + 1e-12) & (xy[:, 0] < r[2] - 1e-12) & (xy[:, 1] > r[1] + 1e-12) & (xy[:, 1] < r[3] - 1e-12)
        inner.append(np.nonzero(ins & (own != s))[0])
    row = np.concatenate(inner)
    pat = np.repeat(np.arange(n * n), [len(v) for v in inner])
    order = np.lexsort((pat, row))
    N = len(xy)
    keys = [np.arange(N) * N + np.arange(N)]
    for s in range(n * n):
        ring = np.arange(first[s], first[s + 1])
        keys += [(inner[s][:, None] * N + ring).ravel(), (ring[:, None] * N + inner[s]).ravel()]
    keys = np.unique(np.concatenate(keys))
    val = np.full(len(keys), 1e-23)
    val[np.searchsorted(keys, np.arange(N) * (N + 1))] = np.bincount(row, minlength=N)
    return dict(xy=xy, rings=rings, rects=rects, closed=closed, first=first, row=row[order], pat=pat[order], keys=keys, val=val, spacing=sp)


def _assembly64(case, stream, key):
    M = _mesh64(case)
    dev, f8, k = "cuda", torch.float64, KNN
    N, paths, h = len(M["xy"]), case["paths"], case["h"]
    val, B = M["val"], np.zeros(N)
    for s, (ring, rect) in enumerate(zip(M["rings"], M["rects"])):
        items = np.nonzero(M["pat"] == s)[0]
        if not len(items):
            continue
        m, rows = len(ring), M["row"][items]
        nw = m if M["closed"][s] else m - k + 1
        nd = torch.tensor(ring, dtype=f8, device=dev)
        win = (torch.arange(nw, device=dev)[:, None] + torch.arange(k, device=dev)) % m
        e2 = (case["eps"] / M["spacing"]) ** 2
        A = torch.exp(-e2 * ((nd[win][:, :, None] - nd[win][:, None]) ** 2).sum(-1))
        t = torch.zeros(len(items) * nw * k, dtype=f8, device=dev)
        b = torch.zeros(len(items), dtype=f8, device=dev)
        x0 = torch.tensor(M["xy"][rows], dtype=f8, device=dev)
        full = torch.full((len(items),), paths, dtype=torch.int64, device=dev)
        for it, ex, ey, Y, Z, _, _, won in _walk64("aniso", x0[:, 0].contiguous(), x0[:, 1].contiguous(), torch.full_like(b, h), full, stream,
                                                  key, sub=rect, item0=torch.tensor(items, device=dev)):
            b.index_add_(0, it, Z + torch.where(won, Y * _g64("aniso", ex, ey), 0 * Z))
            u = (~won).nonzero()[:, 0]
            it, ex, ey, Y = it[u], ex[u], ey[u], Y[u]
            for c in range(0, len(it), 1_000_000):
                i, ix, iy, iY = (v[c:c + 1_000_000] for v in (it, ex, ey, Y))
                d2 = (ix[:, None] - nd[:, 0]) ** 2 + (iy[:, None] - nd[:, 1]) ** 2
                L = torch.maximum(d2[:, win[:, 0]], d2[:, win[:, -1]]).argmin(1)
                w = iY[:, None] * torch.exp(-e2 * d2.gather(1, win[L]))
                t.index_add_(0, ((i * nw + L) * k)[:, None].add(torch.arange(k, device=dev)).ravel(), w.ravel())
        v = torch.linalg.solve(A, t.reshape(len(items), nw, k).permute(1, 2, 0))
        G = torch.zeros(m, len(items), dtype=f8, device=dev)
        G.index_add_(0, win.ravel(), v.reshape(nw * k, len(items)))
        at = np.searchsorted(M["keys"], rows[:, None] * N + np.arange(M["first"][s], M["first"][s + 1]))
        np.add.at(val, at, (-G.T / paths).cpu().numpy())
        np.add.at(B, rows, (b / paths).cpu().numpy())
    return {"val": val, "B": B}


def _disks64(case, seed):
    """Rows of Chebyshev x Fourier collocation disks: per angular frequency a dense solve in the radius."""
    nc, nr = case["n_circle"], case["n_radial"]
    half, nh = (nr + 1) // 2, nc // 2
    m = 2 * half
    if case["problem"] != "franke":
        return None  # (c varies: no closed form per frequency)
    i = np.arange(nr + 1)
    cw = np.where((i == 0) | (i == nr), 2.0, 1.0) * (-1.0) ** i
    dl = 2 * np.pi * np.arange(nc) / nc
    a = np.array([-(np.pi * nc / (2 * np.pi)) ** 2 / 3 - 1 / 6] + [0.5 * (-1.0) ** (l + 1) / np.sin(l * np.pi / nc) ** 2 for l in range(1, nc)])
    mu = np.array([(a * np.cos(k * dl)).sum() for k in range(nc)])
    bw = (-1.0) ** np.arange(m) * np.sin(np.pi * (1.0 / m + 2.0 / m * np.arange(m)) / 2)
    G, B = [], []
    known = {}
    for d in _disks_in(case, seed):
        R = d["radius"]
        if R not in known:
            r = R * np.cos(np.pi * i / nr)
            D = np.outer(cw, 1 / cw) / (r[:, None] - r + np.eye(nr + 1))
            D -= np.diag(D.sum(1))
            op = D @ D + D / r[:, None]
            A1, A2 = op[:half, :half], op[:half, ::-1][:, :half]
            Mk = A1[None] + (-1.0) ** np.arange(nc)[:, None, None] * A2[None] + mu[:, None, None] * np.diag(1 / r[:half] ** 2)[None]
            Mk[:, 0] = np.eye(half)[0]
            known[R] = np.linalg.inv(Mk), r[:half]
        inv, r = known[R]
        th = dl + d["theta0"]
        f = np.zeros((half, nc))
        x, y = torch.tensor(r[1:, None] * np.cos(th) + d["cx"]), torch.tensor(r[1:, None] * np.sin(th) + d["cy"])
        f[1:] = _franke64(x, y)[3].numpy()
        ph = d["periph_theta"]
        k = np.arange(-(len(ph) // 2), len(ph) // 2)
        card = np.cos(k[:, None, None] * (th - ph[:, None])).sum(0) / len(k)
        z = np.zeros((1 + len(ph), half, nc))
        z[0] = np.real(np.fft.ifft(np.einsum("kij,jk->ik", inv, np.fft.fft(f, axis=1)), axis=1))
        z[1:] = np.real(np.fft.ifft(np.einsum("ki,pk->pik", inv[:, :, 0], np.fft.fft(card, axis=1)), axis=2))
        rel = d["inner_xy"] - np.array([d["cx"], d["cy"]])
        rp, tp = np.hypot(rel[:, 0], rel[:, 1]) / R, np.arctan2(rel[:, 1], rel[:, 0])
        w = bw / (rp[:, None] - np.concatenate([-r, r[::-1]]) / R)
        kk = np.arange(-nh, nh)
        ang = kk[:, None, None] * (tp[:, None] - th)
        F, F2 = np.cos(ang).sum(0), (np.cos(ang) * np.cos(kk * np.pi)[:, None, None]).sum(0)
        v = (np.einsum("sjl,pl,pj->ps", z, F, w[:, ::-1][:, :half], optimize=True) +
             np.einsum("sjl,pl,pj->ps", z, F2, w[:, :half], optimize=True)) / nc / w.sum(1)[:, None]
        G.append(-v[:, 1:].ravel())
        B.append(v[:, 0])
    return {"G": np.concatenate(G), "B": np.concatenate(B)}


def exact(case, seed):
    kind, key, stream = case["kind"], seed + 1000, seed % 1000 + 1
    if kind == "disks":
        return _disks64(case, seed)
    if kind == "assembly" and case["cv"] == "none":
        return _assembly64(case, stream, key)
    if kind not in ("points", "batch"):
        return None  # (the 16-bit network and what uses it; the circle stencil's inverse, condition 1e10; three streams of uneven rounds)
    t = lambda v, d=torch.float64: torch.tensor(np.asarray(v), dtype=d, device="cuda")  # noqa: E731
    if kind == "points":
        xy = _points_in(case, seed)
        n = case["n"]
        S = _stats64(case["problem"], t(xy[:, 0]), t(xy[:, 1]), t(np.full(n, case["h"])), t(np.full(n, case["paths"]), torch.int64), stream, key,
                     cv=case["cv"] == "exact")
        if n == 1 and case["cv"] == "none":
            return {k: float(S[k][0]) for k in ("phi", "phiphi", "phi_VR", "phiphi_VR", "xi", "xixi", "xiphi", "APL", "RNGC")}
        return S
    disks, of, xy, paths, h = _batch_in(case, seed)
    if float((paths * h ** -1.0).sum()) > 3e11:
        return None  # (more than 20 seconds)
    return _stats64("franke", t(xy[:, 0]), t(xy[:, 1]), t(h), t(paths.astype(np.int64), torch.int64), stream, key, disk=t(disks[of]))
