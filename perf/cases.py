"""The planner's work as its users call it: cases for timing and for comparing outputs.

A case names a call of the public Python front end (``e2e_gpu_dp_b200.api`` and
``e2e_gpu_dp_b200.envgen``) and its sizes.  The sizes are those of the named
workloads, of the batched form's size ranges and of the parity problems, with
ragged ones between them.  Inputs are synthesised here from a seed in the
reference's layout: a double-gyre mean flow, low-frequency Fourier modes,
Gaussian mode coefficients independent over (t, realisation, mode), and a few
per cent of obstacle cells.

kinds
  plan     build_model, then the layered solve: what a planner run is
  build    build_model alone (the ``build_model`` executable's work)
  fused    build_solve: value and policy without a stored model
  fleet    build_models of uneven problems, then solve_batch of all of them
  layered  the layered solve of a model that is there already (re-solves)
  jacobi   the reference's own schedule (the ``spvi_2`` executable's work)
  env      the environment generator
  rollout  a policy followed through every realisation
"""
import math

import numpy as np
import torch

from e2e_gpu_dp_b200 import api, envgen
from e2e_gpu_dp_b200.problem import REWARD_TYPES, Problem

DEV = "cuda"
PROBLEM_KEYS = ("gsize", "nt", "nrzns", "nmodes", "num_ac_speeds", "num_ac_angles", "F", "dt", "dx", "dy",
                "r_outbound", "r_terminal", "i_term", "j_term", "term_subgrid_size", "neighb_gsize",
                "prob_type", "alpha")


def _case(name, kind, g, nt, nrzns, nm, angles, **more):
    """A case of a grid problem; the target at 9/10 and 1/2 of the grid, the
    neighbourhood 21 cells or the largest odd number that the grid holds."""
    c = dict(kind=kind, gsize=g, nt=nt, nrzns=nrzns, nmodes=nm, num_ac_speeds=1, num_ac_angles=angles, F=1.0,
             dt=1.0, dx=1.0, dy=1.0, r_outbound=-100.0, r_terminal=100.0, i_term=(9 * g) // 10, j_term=g // 2,
             term_subgrid_size=1, neighb_gsize=min(21, g if g % 2 else g - 1), prob_type="time", alpha=0.0,
             gyre=1.0, sigma0=0.3, sigma_base=math.sqrt(2.0), obstacles=0.03, scalar=0.0, where="device")
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a smoke-sized problem from host arrays: launches, synchronisations and allocations count
        _case("plan_16", "plan", 16, 8, 96, 3, 8, gyre=0.6, sigma_base=2.0, obstacles=0.08, neighb_gsize=11,
              where="host"),
        # the CPU-runnable workload, 50x50x30, from host arrays as a planning program holds them
        _case("plan_50", "plan", 50, 30, 500, 4, 8, gyre=0.5, sigma_base=2.0, obstacles=0.05, where="host"),
        # the headline workload: 200x200x120, 16 headings, 5000 realisations, 10 modes
        _case("plan_200", "plan", 200, 120, 5000, 10, 16),
        # the large-grid workload's rows (300x300, 2000 realisations, 8 modes) over 40 steps
        _case("build_300", "build", 300, 40, 2000, 8, 16),
        # odd everything: grid side, realisations, modes; two speeds, the energy/time mix, a 2x2 target
        _case("build_137_ragged", "build", 137, 53, 777, 7, 12, num_ac_speeds=2, F=1.5, term_subgrid_size=2,
              prob_type="custom1", alpha=0.05, r_outbound=-1000.0),
        # half-cell spacing with a scalar field: the radiation reward
        _case("plan_120_half", "plan", 120, 40, 500, 6, 8, dx=0.5, dy=0.5, dt=0.5, gyre=0.4, sigma_base=2.0,
              scalar=0.4, prob_type="energy2"),
        # one backward pass without a stored model
        _case("fused_100", "fused", 100, 60, 1000, 6, 16),
        # a fleet of uneven problems (grid 32-160, 20-100 steps, 200-2000 realisations, 4-8 modes)
        dict(name="fleet_12", kind="fleet", n=12, sizes=2024),
        # re-solving a resident model, both schedules
        _case("layered_200", "layered", 200, 120, 500, 10, 16),
        _case("jacobi_200", "jacobi", 200, 120, 500, 10, 16),
        # the environment generator with the reference script's parameters
        dict(name="env_25x8", kind="env", init_gsize=25, nt=10, n_wsamples=1000, interpolate_degree=8, n_modes=3,
             obstacle="dynamic"),
        # a policy evaluated over all 5000 realisations of the headline workload
        _case("rollout_200", "rollout", 200, 120, 5000, 10, 16, interpolate=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plan", "plan", "build", "build", "fused", "fleet", "layered", "jacobi", "env", "rollout"])
    if kind == "fleet":
        return dict(kind="fleet", n=rng.randint(2, 12), sizes=rng.randint(0, 1 << 20))
    if kind == "env":
        return dict(kind="env", init_gsize=rng.randint(9, 25), nt=rng.randint(4, 12), n_wsamples=_log(rng, 60, 1000),
                    interpolate_degree=rng.randint(2, 8), n_modes=rng.randint(2, 4),
                    obstacle=rng.choice(["none", "static", "dynamic"]))
    while True:
        c = _case(None, kind, _log(rng, 16, 300), _log(rng, 6, 120), _log(rng, 90, 5000), rng.randint(2, 10),
                  rng.choice([8, 12, 16]), gyre=rng.uniform(0.4, 1.0), sigma_base=rng.choice([2.0, math.sqrt(2.0)]),
                  obstacles=rng.uniform(0.0, 0.08), where=rng.choice(["device", "device", "host"]))
        c["i_term"], c["j_term"] = rng.randrange(c["gsize"] - 1), rng.randrange(c["gsize"] - 1)
        form = rng.choice(["time", "time", "time", "speeds", "half"])
        if form == "speeds":
            c.update(num_ac_speeds=2, F=1.5, prob_type=rng.choice(["custom1", "energy1"]), alpha=0.05,
                     term_subgrid_size=2)
        elif form == "half":
            c.update(dx=0.5, dy=0.5, dt=0.5, sigma_base=2.0, gyre=0.4, scalar=0.4,
                     prob_type=rng.choice(["time", "energy2", "energy3"]))
        if kind == "rollout":
            c["interpolate"] = rng.choice([False, True])
        rows = c["gsize"] ** 2 * c["nt"] * c["num_ac_speeds"] * c["num_ac_angles"]
        dear = 4 if form == "half" else 1  # a case costs no more than the largest listed one
        if rows <= 60_000_000 and rows * c["nrzns"] * dear <= 150_000_000_000:
            return c


# ---- inputs ---------------------------------------------------------------------------


def _problem(c):
    return Problem(**{k: c[k] for k in PROBLEM_KEYS}, prob_name="case")


def _mode(rng, X, Y, L):
    acc = np.zeros_like(X)
    for _ in range(3):
        kx, ky = rng.integers(1, 4, size=2)
        px, py = rng.uniform(0, 2 * math.pi, size=2)
        acc += rng.uniform(0.5, 1.0) * np.cos(2 * math.pi * kx * X / L + px) * np.cos(2 * math.pi * ky * Y / L + py)
    return acc / max(float(np.abs(acc).max()), 1e-9)


def _pieces(c, seed):
    """The time-invariant fields and the coefficients of every step."""
    g, nt, nm, nr, dx = c["gsize"], c["nt"], c["nmodes"], c["nrzns"], c["dx"]
    rng = np.random.default_rng([int(seed), g, nt, nr])
    x = dx / 2 + dx * np.arange(g)
    X, Y = np.meshgrid(x, x[::-1])
    L = g * dx
    p = {"u": -c["gyre"] * np.sin(math.pi * X / L) * np.cos(math.pi * Y / L),
         "v": c["gyre"] * np.cos(math.pi * X / L) * np.sin(math.pi * Y / L),
         "ui": np.stack([_mode(rng, X, Y, L) for _ in range(nm)]),
         "vi": np.stack([_mode(rng, X, Y, L) for _ in range(nm)]),
         "s": np.full((g, g), c["scalar"]) + (c["scalar"] * _mode(rng, X, Y, L) if c["scalar"] else 0.0)}
    p = {k: v.astype(np.float32) for k, v in p.items()}
    mask = (rng.random((g, g)) < c["obstacles"]).astype(np.int32)
    n = c["term_subgrid_size"]
    mask[c["i_term"]:c["i_term"] + n, c["j_term"]:c["j_term"] + n] = 0
    p["mask"] = mask
    sig = np.array([c["sigma0"] / c["sigma_base"] ** k for k in range(nm)], dtype=np.float32)
    p["Yi"] = rng.standard_normal((nt, nr, nm), dtype=np.float32) * sig
    return p


def _fields(c, seed, where):
    p, nt = _pieces(c, seed), c["nt"]
    if where == "host":
        return {k: v if k == "Yi" else np.ascontiguousarray(np.broadcast_to(v, (nt,) + v.shape))
                for k, v in p.items()}
    out = {}
    for k, v in p.items():
        t = torch.from_numpy(v).to(DEV)
        out[k] = t if k == "Yi" else t.expand(nt, *v.shape).contiguous()
    return out


class _View:
    """A device array of a model, for torch.as_tensor; it keeps the model."""

    def __init__(self, model, ptr, n, typestr):
        self.model = model
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": typestr, "data": (int(ptr), False),
                                         "version": 3}


def _view(model, ptr, n, typestr):
    return torch.as_tensor(_View(model, ptr, n, typestr), device=DEV)


def _entry_arrays(rows):
    """The caller's own arrays for a model's entries: room for 8 next states a
    row, zeros behind the last one."""
    return (torch.zeros(8 * rows, dtype=torch.int32, device=DEV), torch.zeros(8 * rows, dtype=torch.int16, device=DEV))


def _model_arrays(m, keep):
    """The model: row pointers and rewards where they lie, and next states and
    counts copied into the caller's arrays."""
    i = m.info()
    n = i["nnz"]
    keep[0][:n].copy_(_view(m, i["col"], n, "<i4"))
    keep[1][:n].copy_(_view(m, i["cnt"], n, "<i2"))
    return {"row_ptr": _view(m, i["row_ptr"], i["n_rows"] + 1, "<i4" if i["index_bits"] == 32 else "<i8"),
            "R": _view(m, i["R"], i["ns"] * i["num_actions"], "<f4"), "col": keep[0], "cnt": keep[1]}


def _outputs(ns):
    return (torch.empty(ns, dtype=torch.float32, device=DEV), torch.empty(ns, dtype=torch.int32, device=DEV))


def _fleet(c):
    """The sizes of a fleet, from the case alone."""
    rng = np.random.default_rng(c["sizes"])
    out = []
    for _ in range(c["n"]):
        g = int(rng.integers(32, 161))
        out.append(_case(None, "plan", g, int(rng.integers(20, 101)), int(rng.integers(200, 2001)),
                         int(rng.integers(4, 9)), int(rng.choice([8, 16])), i_term=int(rng.integers(g)),
                         j_term=int(rng.integers(g)), obstacles=float(rng.uniform(0.0, 0.05))))
    return out


def _toward_target(c):
    """The heading closest to the target's direction in every cell: a policy to
    evaluate, free of any solver."""
    g, na = c["gsize"], c["num_ac_angles"]
    i, j = np.meshgrid(np.arange(g), np.arange(g), indexing="ij")
    ang = np.arctan2(-(c["i_term"] - i), c["j_term"] - j)
    a = np.rint(ang / (2 * math.pi / na)).astype(np.int64) % na + na * (c["num_ac_speeds"] - 1)
    return np.ascontiguousarray(np.broadcast_to(a.astype(np.int32), (c["nt"], g, g))).reshape(-1)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "env":
        rng = np.random.default_rng([int(seed), 17])
        obst = {"none": ("None",), "static": ("static",), "dynamic": None}[c["obstacle"]]
        G = c["init_gsize"] * c["interpolate_degree"]
        if obst is None:
            obst = (0.4 * G, 0.6 * G, 0.15 * G, (-0.01 * G, 0.005 * G), "dynamic")
        args = dict(init_gsize=c["init_gsize"], nt=c["nt"], dt=10.0 / c["nt"], dxy=2.0 / c["init_gsize"],
                    A=float(rng.uniform(0.4, 0.6)), A_sc=3, eps=float(rng.uniform(0.08, 0.12)), op_nrzns=10,
                    n_wsamples=c["n_wsamples"], w_range=(math.pi / 10, 8 * math.pi / 10), wx=math.pi,
                    interpolate_degree=c["interpolate_degree"], n_modes=c["n_modes"], dyn_obstacle_data=obst)
        return {"kind": kind, "args": args}
    if kind == "fleet":
        cs = _fleet(c)
        probs = [_problem(x) for x in cs]
        return {"kind": kind, "probs": probs, "fields": [_fields(x, seed + 31 * k, "device") for k, x in enumerate(cs)],
                "out": [_outputs(p.ns) for p in probs], "entries": [_entry_arrays(_rows(x)) for x in cs]}
    p = _problem(c)
    s = {"kind": kind, "prob": p, "fields": _fields(c, seed, c["where"] if kind in ("plan", "build", "fused") else "device")}
    if c["where"] == "device" or kind in ("layered", "jacobi"):
        s["out"] = _outputs(p.ns)
    if kind in ("plan", "build"):
        s["entries"] = _entry_arrays(_rows(c))
    if kind in ("layered", "jacobi"):
        s["model"] = api.build_model(p, s.pop("fields"))
    if kind == "rollout":
        s["policy"] = torch.from_numpy(_toward_target(c)).to(DEV)
        s["start"] = (c["gsize"] // 8, c["gsize"] // 2)
        s["interpolate"] = c["interpolate"]
    return s


# ---- one pass ---------------------------------------------------------------------------


def run(state):
    s, kind = state, state["kind"]
    if kind in ("plan", "build"):
        m = api.build_model(s["prob"], s["fields"])
        out = _model_arrays(m, s["entries"])
        if kind == "plan":
            v, pi = s.get("out", (None, None))
            out["value"], out["policy"], _ = m.solve(method="layered", value=v, policy=pi)
        return out
    if kind == "fused":
        v, pi = s.get("out", (None, None))
        v, pi, _ = api.build_solve(s["prob"], s["fields"], value=v, policy=pi)
        return {"value": v, "policy": pi}
    if kind in ("layered", "jacobi"):
        v, pi, st = s["model"].solve(method=kind, value=s["out"][0], policy=s["out"][1])
        return {"value": v, "policy": pi, "iterations": st["iterations"], "residual": st["residual"]}
    if kind == "fleet":
        models = api.build_models(s["probs"], s["fields"])
        api.solve_batch(models, [o[0] for o in s["out"]], [o[1] for o in s["out"]])
        arrays = [_model_arrays(m, e) for m, e in zip(models, s["entries"])]
        return [{"col": a["col"], "cnt": a["cnt"], "R": a["R"], "value": o[0], "policy": o[1]}
                for a, o in zip(arrays, s["out"])]
    if kind == "env":
        out = envgen.build_environment_DG_with_westward_clouds(**s["args"], device=True)
        del out["stats"]
        return out
    r = api.rollout(s["prob"], s["fields"], s["policy"], s["start"], interpolate=s["interpolate"])
    del r["stats"]
    return r


# ---- what a pass cannot do without ---------------------------------------------------------


def _field_bytes(c):
    return 4 * c["nt"] * (c["gsize"] ** 2 * (4 + 2 * c["nmodes"]) + c["nrzns"] * c["nmodes"])


def _rows(c):
    return c["gsize"] ** 2 * (c["nt"] - 1) * c["num_ac_speeds"] * c["num_ac_angles"]


def _entries(c):
    # about 3.5 next states a row, as the headline workload has
    return 3.5 * _rows(c)


def work(case):
    """Fields read once, the model (row pointers, entries of 6 bytes, rewards),
    values and policy written once; the velocity of every (cell, realisation),
    one landing test of it, and a multiply-add per entry backed up."""
    c, kind = case, case["kind"]
    if kind == "env":
        n, G2 = c["init_gsize"] ** 2, (c["init_gsize"] * c["interpolate_degree"]) ** 2
        r, nws, nt = c["n_modes"], c["n_wsamples"], c["nt"]
        # fields out, coefficients out; six products of the centred matrices with r columns
        return {"bytes": nt * (4.0 * G2 * (5 + 3 * r) + 8.0 * nws * r) + 36.0 * G2,
                "flops": nt * (3.0 * n * nws * (2 * 6 * r + 40))}
    if kind == "fleet":
        parts = [work(x) for x in _fleet(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    cells, na = c["gsize"] ** 2, c["num_ac_speeds"] * c["num_ac_angles"]
    rows, ns, e = _rows(c), cells * c["nt"], _entries(c)
    samples = float(cells) * (c["nt"] - 1) * c["nrzns"]
    model = 4.0 * rows + 6.0 * e + 4.0 * ns * na
    if kind == "rollout":
        steps = float(c["nrzns"]) * c["nt"] / 2
        return {"bytes": steps * 4 * (3 * c["nmodes"] + 4) + 25.0 * c["nrzns"], "flops": steps * (4 * c["nmodes"] + 20)}
    if kind == "layered":
        return {"bytes": model + 8.0 * ns, "flops": 2 * e + 2 * rows}
    if kind == "jacobi":
        # a layer is final after as many sweeps as layers follow it
        half = c["nt"] / 2.0
        return {"bytes": half * (model + 8.0 * ns), "flops": half * (2 * e + 2 * rows)}
    w = {"bytes": float(_field_bytes(c)), "flops": samples * (4 * c["nmodes"] + 10)}
    if kind in ("plan", "build"):
        w["bytes"] += model
    if kind in ("plan", "fused"):
        w["bytes"] += 8.0 * ns
        w["flops"] += 2 * e + 2 * rows
    return w


# ---- 64-bit values ---------------------------------------------------------------------------


def _override(c, mask):
    """[cell, 13 (di + 6) + dj + 6]: does the way from a cell to (di, dj) beyond it pass an obstacle?"""
    g, D = c["gsize"], 6
    ob = np.zeros((g + 4 * D, g + 4 * D), bool)
    ob[2 * D:-2 * D, 2 * D:-2 * D] = mask == 1
    out = np.zeros((g, g, 2 * D + 1, 2 * D + 1), bool)
    diag = 1.414213 * c["dx"]
    for di in range(-D, D + 1):
        for dj in range(-D, D + 1):
            for a in range(min(di, 0), max(di, 0) + 1):
                for b in range(min(dj, 0), max(dj, 0) + 1):
                    if a == 0 and b == 0:
                        continue
                    near = True
                    if di and dj:  # distance of (b, -a) from the line through (0, 0) and (dj, -di)
                        A = -di / dj
                        near = abs(A * b + a) * c["dx"] / math.hypot(A, 1.0) < diag
                    if near:
                        out[:, :, di + D, dj + D] |= ob[2 * D + a:2 * D + a + g, 2 * D + b:2 * D + b + g]
    return out.reshape(g * g, -1)


def _plan64(c, seed):
    """Values of the layered solve in 64 bits: per (cell, action) the mean over
    the realisations of reward + value of the landing cell."""
    dev = DEV if torch.cuda.is_available() else "cpu"
    p, g, nt, nr = _pieces(c, seed), c["gsize"], c["nt"], c["nrzns"]
    f = {k: torch.from_numpy(v).to(dev).double() for k, v in p.items()}
    nc, dx, dt, D = g * g, c["dx"], c["dt"], (c["neighb_gsize"] - 1) // 2
    ovr = torch.from_numpy(_override(c, p["mask"])).to(dev)
    i = torch.arange(nc, device=dev) // g
    j = torch.arange(nc, device=dev) % g
    obst, sc = f["mask"].reshape(-1) == 1, f["s"].reshape(-1)
    n = c["term_subgrid_size"]

    def terminal(a, b):
        return (a >= c["i_term"]) & (a < c["i_term"] + n) & (b >= c["j_term"]) & (b < c["j_term"] + n)

    ns, na = c["num_ac_speeds"], c["num_ac_angles"]
    acts = [(np.float32(c["F"]) if ns == 1 else np.float32(k + 1) * (np.float32(c["F"]) / np.float32(ns)),
             np.float32(h * (2 * math.pi) / na)) for k in range(ns) for h in range(na)]
    kind = REWARD_TYPES[c["prob_type"]]
    V = torch.zeros(nt, nc, dtype=torch.float64, device=dev)
    ui, vi = f["ui"].reshape(-1, nc), f["vi"].reshape(-1, nc)
    per = max(1, 4_000_000 // nr)
    for t in range(nt - 2, -1, -1):
        for lo in range(0, nc, per):
            k = slice(lo, min(lo + per, nc))
            vx = f["u"].reshape(-1)[k, None] + ui[:, k].T @ f["Yi"][t].T
            vy = f["v"].reshape(-1)[k, None] + vi[:, k].T @ f["Yi"][t].T
            best = None
            for F, th in acts:
                F, cs, sn = float(F), float(np.cos(th)), float(np.sin(th))
                ax = j[k, None] * dx + (F * cs + vx) * dt
                ay = i[k, None] * dx - (F * sn + vy) * dt
                top = (g - 1) * dx
                clamps = ((ax < 0) | (ax > top)).double() + ((ay < 0) | (ay > top)).double()
                j2 = torch.floor(ax.clamp(0, top) / dx + 0.5).long()
                i2 = torch.floor(ay.clamp(0, top) / dx + 0.5).long()
                edge = ((i2 == 0) | (i2 == g - 1) | (j2 == 0) | (j2 == g - 1)).double()
                term = terminal(i2, j2)
                r = c["r_outbound"] * (clamps + edge)
                r = r + torch.where(term, c["r_terminal"], 0.05 * c["r_outbound"] if t > nt - 20 else 0.0)
                rad = (sc[k, None] + sc[i2 * g + j2]) / 2
                a = np.float32(c["alpha"])
                r = r + dt * {0: -1.0, 1: -(F * F + 0.01), 2: rad - F * F - 0.01, 3: rad - 0.01,
                              4: float(-a * F * F - (1 - a))}[kind]
                di, dj = i2 - i[k, None], j2 - j[k, None]
                o = ovr[k].gather(1, (di.clamp(-6, 6) + 6) * 13 + dj.clamp(-6, 6) + 6)
                r = torch.where(o, torch.as_tensor(c["r_outbound"], dtype=r.dtype, device=dev), r)
                inside = (di.abs() <= D) & (dj.abs() <= D)
                q = (r + torch.where(inside, V[t + 1][i2 * g + j2], 0.0)).mean(1)
                best = q if best is None else torch.maximum(best, q)
            still = terminal(i[k], j[k])
            stay = V[t + 1][k] + torch.where(still, 0.0, c["r_outbound"])
            V[t][k] = torch.where(still | obst[k], stay, best)
    return V.reshape(-1).cpu().numpy()


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "env":
        svals = []
        a = prepare(c, seed)["args"]
        x = (0.5 + np.arange(c["init_gsize"])) * a["dxy"]
        X, Y = np.meshgrid(x, x[::-1])
        w = a["w_range"][0] + np.arange(c["n_wsamples"]) / (c["n_wsamples"] - 1) * (a["w_range"][1] - a["w_range"][0])
        for t in range(c["nt"]):
            e = a["eps"] * np.sin(w * (t * a["dt"]))[:, None]
            xx, yy = X.reshape(1, -1), Y.reshape(1, -1)
            h = e * xx * xx + (1 - 2 * e) * xx
            hx = 2 * e * (xx - 1) + 1
            wy = math.pi / 2
            vx = -0.5 * a["A"] * math.pi * np.sin(a["wx"] * h) * np.cos(wy * yy)
            vy = a["A"] * math.pi * np.sin(wy * yy) * hx * np.cos(a["wx"] * h)
            ph = a["A"] * np.sin(math.pi * h) * np.sin(wy * yy)
            svals.append([np.linalg.svd(m - m.mean(0), compute_uv=False)[:c["n_modes"]]
                          for m in (np.concatenate([vx, vy], 1), ph)])
        sv = np.array(svals)
        names = list(envgen.FILES)
        return {**{k: None for k in names}, "svals_vel": sv[:, 0], "svals_phi": sv[:, 1]}
    if kind in ("plan", "fused"):
        samples = float(c["gsize"]) ** 2 * c["nt"] * c["nrzns"] * c["num_ac_speeds"] * c["num_ac_angles"]
        if samples > (1e10 if torch.cuda.is_available() else 3e8):
            return None
        out = {"value": _plan64(c, seed), "policy": None}
        return out if kind == "fused" else {"row_ptr": None, "col": None, "cnt": None, "R": None, **out}
    # a stored model's solves and a trajectory are functions of counts and
    # cells that rounding decides: no 64-bit value of their own
    return None
