"""Workloads of the colour-gradient LBM framework, as a user's program runs them.

A pass of a `single` case is one interval of a simulation: `steps` time steps, the diagnostic row of
the last one (what Imm_OPS / Imm_INCL print every 500 steps) and the per-node fields of that step
(what they write as vel_*.vtk / rho_*.vtk or perfil.dat); the next pass continues the same
simulation.  A pass of a `batch` case is a whole sweep through the batch engine: every case
submitted, advanced to its last step with its diagnostics, its final fields read and its memory
released.  Box sides, operators and ranges of tau, sigma, chi and v0 are those of the reference's
stored sweeps (40 to 200 nodes a side, FP64) and of this repository's benchmark mix (64 to 512) and
large single drops.
"""
import importlib
import math
import random

import numpy as np
import torch

lbm = importlib.import_module("interfacial-tension-operators-lbm_b200")

OPS = {"P1": lbm.OP_P1, "P3": lbm.OP_P3, "F1": lbm.OP_F1, "F2": lbm.OP_F2, "F3": lbm.OP_F3}
PREC = {"f64": lbm.PREC_F64, "f32": lbm.PREC_F32, "fold": lbm.PREC_F32_FOLD}
STATE_BYTES = {"f64": 304, "f32": 152, "fold": 72}  # populations of one node
MOST_UPDATES = 2048 * 2048 * 500                      # node updates of the largest listed case
XI = 1.569988


def single(name, nx, ny, op, prec, steps, geometry="drop", v0=0.0):
    c = {"kind": "single", "nx": nx, "ny": ny, "op": op, "prec": prec, "steps": steps, "geometry": geometry, "v0": v0}
    return {"name": name, **c} if name else c


def batch(name, count, lo, hi, prec, steps, strips):
    c = {"kind": "batch", "count": count, "lo": lo, "hi": hi, "prec": prec, "steps": steps, "strips": strips}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the smallest box of the sweeps, a row every ten steps: a program that watches a small drop
        single("drop40_rows", 40, 40, "P3", "f64", 10),
        # the box of the reference's E2 and E4 sweeps, one diagnostic interval
        single("drop100", 100, 100, "P3", "f64", 500),
        # the inclined-interface box of its E3 sweep, curvature force
        single("strip200", 200, 200, "F1", "f64", 500, geometry="strip"),
        # a translating drop with the capillary-stress force
        single("drop256_moving", 256, 256, "F2", "f64", 500, v0=0.05),
        # a box beyond the caches in the bit-exact precision
        single("drop1024x768", 1024, 768, "P1", "f64", 500),
        # FP32 storage on a box with odd sides
        single("drop333x207", 333, 207, "F2", "f32", 500),
        # the translating drop of the precision study
        single("drop512_moving", 512, 512, "P3", "f32", 500, v0=0.1),
        # the large single drop
        single("drop2048", 2048, 2048, "P3", "f32", 500),
        # the folded storage, chemical-potential force
        single("fold300", 300, 300, "F3", "fold", 500),
        # the folded storage on a large ragged box, curvature force
        single("fold1500x1100", 1500, 1100, "F1", "fold", 500),
        # a sweep of equal 100-node boxes in FP64, as the reference's batch script runs its E2 folder
        batch("sweep_e2", 42, 100, 100, "f64", 501, 0.0),
        # a mixed sweep of the benchmark's sizes in FP32, drops and strips, all operators
        batch("sweep_mix", 32, 64, 512, "f32", 501, 0.2),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    prec = rng.choice(["f64", "f64", "f32", "fold"])
    if rng.random() < 0.2:
        lo = side(40, 128)
        return batch(None, rng.randint(6, 32), lo, min(512, int(lo * rng.uniform(1.0, 4.0))), prec, 501,
                     rng.choice([0.0, 0.2]))
    while True:
        nx = side(40, 2048)
        ny = nx if rng.random() < 0.5 else max(40, min(2048, int(nx * rng.uniform(0.5, 1.5))))
        steps = rng.choice([10, 100, 500, 500])
        bytes_per_update = 1 if prec != "f64" else 2
        if nx * ny * steps * bytes_per_update <= MOST_UPDATES:
            break
    op = rng.choice(sorted(OPS))
    strip = nx == ny and rng.random() < 0.3
    return single(None, nx, ny, op, prec, steps, geometry="strip" if strip else "drop",
                  v0=0.0 if strip else rng.choice([0.0, 0.0, 0.05, 0.1]))


def physics(r, nx, ny, op, geometry, v0):
    """Physical parameters of one case: those of the sweeps, drawn by r."""
    sigma = r.uniform(0.03, 0.1)
    tau = r.uniform(0.7, 1.1)
    m = min(nx, ny)
    p, q = (r.randint(1, 4), r.randint(1, 4)) if geometry == "strip" else (1, 0)
    return {"nx": nx, "ny": ny, "op": op, "chi": r.choice([0.5, 2.0]), "tau": tau, "beta": 0.8,
            "A": 9.0 * sigma / (4.0 * tau) if op in ("P1", "P3") else sigma,
            "radius": m * r.uniform(0.2, 0.26), "k": 2.0 * math.log(9.0) / 3.45, "v0": v0,
            "geometry": geometry, "p": p, "q": q}


def members(case, seed):
    """The physical parameters of the simulations of a case, one or many."""
    r = random.Random(seed)
    if case["kind"] == "single":
        return [physics(r, case["nx"], case["ny"], case["op"], case["geometry"], case["v0"])]
    sizes = random.Random(7 * case["count"] + case["lo"] + case["hi"])  # the sweep's boxes: not the seed's
    got = []
    for _ in range(case["count"]):
        nx = int(round(math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        geometry = "strip" if sizes.random() < case["strips"] else "drop"
        got.append(physics(r, nx, nx, sizes.choice(sorted(OPS)), geometry, 0.0))
    return got


def desc(m, prec):
    return lbm.desc(m["nx"], m["ny"], lbm.make_op(OPS[m["op"]], m["chi"], XI), tau=m["tau"], beta=m["beta"],
                    A_fact=m["A"], geometry=lbm.GEOM_STRIP if m["geometry"] == "strip" else lbm.GEOM_DROP,
                    radius=m["radius"], k_profile=m["k"], v0=m["v0"], p=m["p"], q=m["q"], precision=PREC[prec])


def prepare(case, seed):
    ms = members(case, seed)
    if case["kind"] == "single":
        return {"case": lbm.Case(desc(ms[0], case["prec"])), "steps": case["steps"], "done": 0,
                "strip": case["geometry"] == "strip"}
    b = lbm.Batch()
    b.hold_finished(True)
    return {"batch": b, "descs": [desc(m, case["prec"]) for m in ms], "steps": case["steps"]}


def row(d):
    """A diagnostic row as two arrays: its measures and its counts."""
    v = d.as_dict()
    return {"measures": np.array([x for x in v.values() if isinstance(x, float)]),
            "counts": np.array([x for x in v.values() if isinstance(x, int)], dtype=np.int64)}


def run(state):
    if "case" in state:
        c = state["case"]
        c.step(state["steps"], keep_aux=True)
        state["done"] += state["steps"]
        last = state["done"] - 1
        if state["strip"]:
            return {"row": row(c.diag_strip(last)), "fields": c.read_profile()}
        return {"row": row(c.diag_drop(last)), "fields": c.read_fields()}
    b, descs = state["batch"], state["descs"]
    for tag, d in enumerate(descs):
        b.submit(d, state["steps"], tag)
    rows, fields = {}, {}
    while len(fields) < len(descs):
        b.advance()
        for e in b.poll():
            if e.kind == lbm.EV_DIAG:
                rows[(e.tag, e.step)] = row(e.strip if e.geometry == lbm.GEOM_STRIP else e.drop)
            else:
                d = descs[e.tag]
                form = lbm.FIELDS_PROFILE if e.geometry == lbm.GEOM_STRIP else lbm.FIELDS_VTK
                fields[e.tag] = b.read_fields(e.tag, d.nx * d.ny, form)
                b.release(e.tag)
    keys, tags = sorted(rows), range(len(descs))
    return {"measures": np.concatenate([rows[k]["measures"] for k in keys]),
            "counts": np.concatenate([rows[k]["counts"] for k in keys]),
            "fields": {f: np.concatenate([fields[t][f] for t in tags]) for f in ("rho_R", "rho_B", "ux", "uy")}}


# Additions, multiplications, divisions and roots of one node update: the colour sums and moments of
# the 2 x 19 (or 2 x 9) populations, the colour gradient, equilibrium and relaxation by direction,
# the operator, and the recolouring split.
FLOPS = {"P1": 560, "P3": 560, "F1": 640, "F2": 680, "F3": 620}
FLOPS_FOLD = {"P1": 290, "P3": 290, "F1": 370, "F2": 400, "F3": 340}


def work(case):
    per = FLOPS_FOLD if case["prec"] == "fold" else FLOPS
    nbytes = flops = 0
    for m in members(case, 0):
        n = m["nx"] * m["ny"]
        # a single case reads its populations and writes them; a sweep starts from descriptions;
        # the fields are five numbers a node (four in perfil.dat)
        nbytes += n * 8 * (4 if m["geometry"] == "strip" else 5)
        if case["kind"] == "single":
            nbytes += 2 * n * STATE_BYTES[case["prec"]]
        flops += n * case["steps"] * per[m["op"]]
    return {"bytes": nbytes, "flops": flops}


# --- the same physics in plain 64-bit torch -------------------------------------------------------

CX = [0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0]
CY = [0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, -1, 1, -1, 1]
CZ = [0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, -1, 1, 1, -1]


def exact(case, seed):
    if case["kind"] != "single" or case["nx"] * case["ny"] * case["steps"] > 8_000_000:
        return None
    m = members(case, seed)[0]
    f64 = torch.float64
    nx, ny = m["nx"], m["ny"]
    c = torch.tensor([CX, CY, CZ], dtype=f64)
    cc = c.square().sum(0)
    w = torch.where(cc == 0, 1.0 / 3.0, torch.where(cc == 1, 1.0 / 18.0, 1.0 / 36.0)).to(f64)
    wv, norm = w[:, None, None], cc.clamp(min=1.0).sqrt()[:, None, None]
    cv = [c[a][:, None, None] for a in range(3)]

    def along(u):  # c_i . u
        return cv[0] * u[0] + cv[1] * u[1] + cv[2] * u[2]

    def equilibrium(rho, u):
        cu = along(u)
        return wv * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2))

    def moved(a, dx, dy):  # a(x + dx, y + dy)
        return torch.roll(a, (-dy, -dx), (0, 1))

    def gradient(a):  # 3 sum_i w_i c_i a(x + c_i)
        g = torch.zeros(3, ny, nx, dtype=f64)
        for i in range(1, 19):
            s = 3.0 * w[i] * moved(a, CX[i], CY[i])
            g[0] += CX[i] * s
            g[1] += CY[i] * s
        return g

    yy, xx = torch.meshgrid(torch.arange(ny), torch.arange(nx), indexing="ij")
    u0 = torch.zeros(3, ny, nx, dtype=f64)
    if m["geometry"] == "drop":
        r = ((xx - nx // 2).to(f64) ** 2 + (yy - ny // 2).to(f64) ** 2).sqrt()
        red = 1.0 / (1.0 + torch.exp((m["k"] * (r - m["radius"])).clamp(-60.0, 60.0)))
        u0[0] = m["v0"]
    else:
        s = torch.remainder(m["p"] * xx + m["q"] * yy, nx).to(f64)
        length = math.sqrt(m["p"] ** 2 + m["q"] ** 2)
        near = torch.where(2 * s < nx, torch.minimum(s, 0.5 * nx - s), -torch.minimum(s - 0.5 * nx, nx - s)) / length
        red = 1.0 / (1.0 + torch.exp(-(2.0 * math.log(9.0) / 3.45) * near))
    fR, fB = equilibrium(red, u0), equilibrium(1.0 - red, u0)

    tau, A, op = m["tau"], m["A"], m["op"]
    if op == "P1":
        B = w / 3.0
    else:
        chi = m["chi"]
        den = 6.0 * chi + 24.0
        B = torch.where(cc == 0, -(2.0 + 2.0 * chi) / (3.0 * chi + 12.0),
                        torch.where(cc == 1, chi / den, 1.0 / den)).to(f64)
    for _ in range(case["steps"]):
        rR, rB = fR.sum(0), fB.sum(0)
        rho = rR + rB
        phi = (rR - rB) / rho
        g = gradient(phi)
        size = (g[0] ** 2 + g[1] ** 2).sqrt()
        F = torch.zeros(3, ny, nx, dtype=f64)
        if op == "F1":
            n = g * torch.where(size > 1e-12, 1.0 / size, torch.zeros_like(size))
            F = 0.5 * A * -(gradient(n[0])[0] + gradient(n[1])[1]) * g
        elif op == "F2":
            inv = torch.where(size > 1e-30, 1.0 / size, torch.zeros_like(size))
            txx, tyy = 0.5 * A * (size - g[0] ** 2 * inv), 0.5 * A * (size - g[1] ** 2 * inv)
            gxy = gradient(-0.5 * A * g[0] * g[1] * inv)
            F[0], F[1] = gradient(txx)[0] + gxy[1], gxy[0] + gradient(tyy)[1]
        elif op == "F3":
            lap = sum(6.0 * w[i] * (moved(phi, CX[i], CY[i]) - phi) for i in range(1, 19))
            F = (4.0 * (3.0 * A / (8.0 * XI)) * phi * (phi * phi - 1.0) - 0.75 * A * XI * lap) * g
        f = fR + fB
        u = torch.stack([(cv[a] * f).sum(0) for a in range(3)]) / rho + 0.5 * F / rho
        cu, cF = along(u), along(F)
        uF = u[0] * F[0] + u[1] * F[1] + u[2] * F[2]
        f = f + (equilibrium(rho, u) - f) / tau + (1.0 - 0.5 / tau) * wv * 3.0 * (cF + 3.0 * cF * cu - uF)
        cg = along(g)
        if op in ("P1", "P3"):
            inv2 = torch.where(size * size > 1e-60, 1.0 / (size * size), torch.zeros_like(size))
            f = f + A * size * (wv * cg * cg * inv2 - B[:, None, None])
        cos = -cg * torch.where(size > 0.0, 1.0 / size, torch.zeros_like(size)) / norm
        cR = rR / rho
        t = m["beta"] * cR * (1.0 - cR) * wv * rho * cos
        fR, fB = cR * f - t, (1.0 - cR) * f + t
        last = fR, fB, F
        fR = torch.stack([moved(fR[i], -CX[i], -CY[i]) for i in range(19)])
        fB = torch.stack([moved(fB[i], -CX[i], -CY[i]) for i in range(19)])
    fR, fB, F = last
    rR, rB = fR.sum(0), fB.sum(0)
    u = (torch.stack([(cv[a] * (fR + fB)).sum(0) for a in range(3)]) - 0.5 * F) / (rR + rB)
    fields = {"rho_R": rR, "rho_B": rB, "ux": u[0], "uy": u[1]}
    if m["geometry"] == "drop":
        fields["uz"] = None  # zero by symmetry: what a run prints there is round-off
    return {"row": None, "fields": {k: v if v is None else v.reshape(-1) for k, v in fields.items()}}
