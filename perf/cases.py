"""The work that is timed: flow solves, transport solves, batches and geometry walks.

Every case goes through the package's Python entry points, with host arrays
in and host arrays out, as a program that calls `stokes_d3q19`, `solve_adr`,
`solve_batch` or `prep.inlet_walk` does.  Time loops run for a fixed
number of iterations (`tol=0`, `steps=n`), so that the work of a case is known;
solves in real use run for 1 000 to 100 000 of the same iterations.

`exact` restates the algorithms in 64 bits with plain torch: lattice
Boltzmann TRT with Guo forcing and node bounce-back, and the finite-volume
transport with minmod-limited advection, dual-Monod or sorption terms.
"""

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "prt-deeponet-gui_b200"))

from prtlb_gpu import (Chemistry, coat_with_biofilm, default_chemistry,  # noqa: E402
                       first_order_chemistry, monod_chemistry, prep, random_pack,
                       reversible_sorption_chemistry, solve_adr, stokes_d2q9, stokes_d3q19)
from prtlb_gpu.batch import Request, solve_batch  # noqa: E402

PORE = 2
BIOFILM = 3
FORCE = 2e-6
STORED = {"fp64": 8, "fp32": 4, "fp32f": 4, "fp16": 2}

# chemicals by kinetics, and how many of them are transported
SPECIES = {"monod": 1, "first_order": 1, "sorption": 2, "dual": 2, "default4": 4, "biofilm4": 4}
MOVING = {"monod": 1, "first_order": 1, "sorption": 1, "dual": 2, "default4": 3, "biofilm4": 3}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def flow(name, shape, porosity, precision, nit):
    s = list(shape) + [1] * (3 - len(shape))
    return {"name": name, "kind": "flow", "nd": len(shape), "nx": s[0], "ny": s[1], "nz": s[2],
            "porosity": porosity, "precision": precision, "nit": nit}


def transport(name, shape, porosity, kinetics, pe, da, steps, n_t=5):
    s = list(shape) + [1] * (3 - len(shape))
    return {"name": name, "kind": "transport", "nd": len(shape), "nx": s[0], "ny": s[1],
            "nz": s[2], "porosity": porosity, "kinetics": kinetics, "pe": pe, "da": da,
            "steps": steps, "n_t": n_t}


def batch(name, count, lo, hi, nit, steps):
    return {"name": name, "kind": "batch", "count": count, "lo": lo, "hi": hi, "nit": nit,
            "steps": steps}


def walk(name, shape, porosity):
    return {"name": name, "kind": "walk", "nd": len(shape), "nx": shape[0], "ny": shape[1],
            "nz": shape[2] if len(shape) == 3 else 1, "porosity": porosity}


def listed():
    return [
        # the smallest rocks of the request sets, in the default precision:
        # launches and the call's own cost count most
        flow("flow3d_24_fp64", (24, 24, 24), 0.45, "fp64", 600),
        # the plain 2D configuration: 128 x 128 disks, D2Q9, 1350 iterations
        flow("flow2d_128_fp64", (128, 128), 0.6, "fp64", 1350),
        # the plain 3D configuration: the 64^3 pack in float32
        flow("flow3d_64_fp32f", (64, 64, 64), 0.45, "fp32f", 6000),
        # a rock cut from an image: three unequal odd edges, default precision
        flow("flow3d_113x80x97_fp64", (113, 80, 97), 0.4, "fp64", 1000),
        # the precision sweep's packs, beyond the L2 cache
        flow("flow3d_128_fp32", (128, 128, 128), 0.45, "fp32", 1000),
        flow("flow3d_192_fp16", (192, 192, 192), 0.45, "fp16", 1000),
        # the plain configurations' transport: Monod at 64^3, first order in 2D
        transport("adr3d_64_monod", (64, 64, 64), 0.45, "monod", 10.0, 1.0, 10000),
        transport("adr2d_128_first_order", (128, 128), 0.6, "first_order", 10.0, 1.0, 4000),
        # the built-in four-chemical chemistry on a large pack
        transport("adr3d_128_default4", (128, 128, 128), 0.45, "default4", 10.0, 1.0, 3000),
        # biofilm with its own diffusivities and coupled biomass, unequal edges
        transport("adr3d_131x96x71_biofilm4", (131, 96, 71), 0.5, "biofilm4", 30.0, 3.0, 3000),
        # the batched configuration's small rocks, all kinetics, flow then transport
        batch("batch_16_small", 16, 24, 48, 600, 800),
        # the walk behind keep_inlet_connected and the distance columns
        walk("walk3d_128", (128, 128, 128), 0.45),
    ]


def _edge(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flow"] * 3 + ["transport"] * 3 + ["batch", "walk"])
    if kind == "batch":
        lo = rng.randint(24, 40)
        c = batch("", rng.randint(4, 16), lo, rng.randint(lo + 2, 56), 50 * rng.randint(4, 12),
                  rng.randint(200, 800))
    else:
        if rng.random() < 0.75:
            base = _edge(rng, 24, 150)
            shape = [min(160, max(20, int(round(base * rng.uniform(0.75, 1.3))))) for _ in range(3)]
            porosity = rng.uniform(0.35, 0.6)
        else:
            shape = [_edge(rng, 48, 700) for _ in range(2)]
            porosity = rng.uniform(0.5, 0.7)
        porosity = round(porosity, 3)
        n = math.prod(shape)
        if kind == "flow":
            nit = max(200, min(3000, int(1.2e9 / n)))
            c = flow("", shape, porosity, rng.choice(["fp64", "fp32", "fp32f", "fp16"]), nit)
        elif kind == "transport":
            kinetics = rng.choice(sorted(SPECIES))
            steps = max(300, min(8000, int(6.0e9 / n / MOVING[kinetics])))
            c = transport("", shape, porosity, kinetics, round(10.0 ** rng.uniform(0.0, 2.0), 2),
                          round(10.0 ** rng.uniform(-1.0, 1.0), 3), steps, rng.randint(2, 6))
        else:
            c = walk("", shape, porosity)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _shape(case):
    return (case["nx"], case["ny"], case["nz"])[:case["nd"]]


def _rock(case, seed):
    """A random sphere pack (radius 4-7) or disk pack (radius 4-8)."""
    shape = _shape(case)
    return random_pack(shape, case["porosity"], 4.0, 8.0 if len(shape) == 2 else 7.0,
                       seed=int(seed))


def _field(g, seed):
    """A velocity with a flow field's features, float32 (3,) + grid: fast in
    the wide pores and slow at the walls (the pore mask blurred over a few
    voxels), with transverse parts that change sign along the grid."""
    dev = _device()
    m = torch.from_numpy(g == PORE).to(dev).double()
    a = m
    for ax in range(g.ndim):
        a = (a.roll(2, ax) + 2 * a.roll(1, ax) + 3 * a + 2 * a.roll(-1, ax) + a.roll(-2, ax)) / 9.0
    ph = np.random.default_rng(seed).uniform(0.0, 2.0 * math.pi, 4)
    x = [torch.arange(n, device=dev, dtype=torch.float64).reshape([-1 if b == ax else 1
         for b in range(g.ndim)]) for ax, n in enumerate(g.shape)]
    v = torch.zeros((3,) + g.shape, device=dev, dtype=torch.float64)
    v[0] = 2e-4 * a * a * (1.0 + 0.3 * torch.sin(x[1] * 0.21 + ph[0]))
    v[1] = 8e-5 * a * a * torch.sin(x[0] * 0.37 + ph[1] + x[1] * 0.11)
    if g.ndim == 3:
        v[2] = 8e-5 * a * a * torch.sin(x[0] * 0.29 + ph[2] + x[2] * 0.17)
    return (v * m).float().cpu().numpy()


def _chemistry(kinetics, da):
    if kinetics == "monod":
        return monod_chemistry(0.5)
    if kinetics == "first_order":
        return first_order_chemistry()
    if kinetics == "sorption":
        return reversible_sorption_chemistry(0.5, da)
    if kinetics == "dual":
        return default_chemistry(2)
    if kinetics == "default4":
        return default_chemistry(4)
    return Chemistry(names=["Ac", "A", "P", "Bio"], inlet=[1.0, 1.0, 0.0, np.nan],
                     c_init=[0.0, 0.0, 0.0, 0.1], d_rel=[1.0, 0.8, 1.2, 0.0],
                     immobile=[False, False, False, True], ks_donor=0.2, ks_acceptor=0.15,
                     d_biofilm_rel=[0.6, 0.5, 0.7, 0.0], decay_lattice=0.002,
                     biofilm_code=BIOFILM, seed_in_biofilm=True, biomass_coupled=True)


def _batch_draws(case, seed):
    """Parameters of a batch's requests: the edges spread over the case's
    range, Pe, Da and kinetics mixed."""
    rng = np.random.default_rng(seed)
    span, draws = case["hi"] - case["lo"] + 1, []
    for k in range(case["count"]):
        e = [case["lo"] + (7 * k + 3 * a * a) % span for a in range(3)]
        draws.append({"nd": 3, "nx": e[0], "ny": e[1], "nz": e[2],
                      "porosity": float(rng.uniform(0.4, 0.6)),
                      "pe": float(10.0 ** rng.uniform(0.0, 2.0)),
                      "da": float(10.0 ** rng.uniform(-2.0, 1.0)),
                      "kinetics": ("monod", "first_order", "sorption")[k % 3],
                      "seed": int(rng.integers(0, 2 ** 31 - 1))})
    return draws


def prepare(case, seed):
    if case["kind"] == "batch":
        reqs = []
        for d in _batch_draws(case, seed):
            reqs.append(Request(_rock(d, d["seed"]),
                                flow=dict(nit=case["nit"], tol=0.0, force=FORCE, precision="fp32"),
                                adr=dict(pe=d["pe"], da=d["da"], n_t=5,
                                         n_species=SPECIES[d["kinetics"]], steps=case["steps"],
                                         chem=_chemistry(d["kinetics"], d["da"])),
                                keep_velocity=True))
        return {"case": case, "requests": reqs}
    g = _rock(case, seed)
    if case["kind"] in ("flow", "walk"):
        return {"case": case, "g": g}
    v = _field(g, seed)
    if case["kinetics"] == "biofilm4":
        g = coat_with_biofilm(g, BIOFILM, layers=1)[0]
    return {"case": case, "g": g, "v": v, "chem": _chemistry(case["kinetics"], case["da"])}


def run(state):
    case = state["case"]
    if case["kind"] == "flow":
        info = {}
        solve = stokes_d3q19 if case["nd"] == 3 else stokes_d2q9
        vel = solve(state["g"], nit=case["nit"], force=FORCE, tol=0.0, info=info,
                    precision=case["precision"])
        return {"vel": vel, "permeability": info["permeability"], "iters": info["flow_iters"]}
    if case["kind"] == "transport":
        out, t_norm = solve_adr(state["g"], state["v"], case["pe"], case["da"], case["n_t"],
                                n_species=SPECIES[case["kinetics"]], steps=case["steps"],
                                chem=state["chem"])
        return {"out": out, "t_norm": t_norm}
    if case["kind"] == "batch":
        found = []
        for r in solve_batch(state["requests"], quiet=True):
            if r.error is not None:
                raise r.error
            found.append({"vel": r.vel, "out": r.out})
        return found
    steps, n_reached, n_pore = prep.inlet_walk(state["g"])
    return {"steps": steps, "n_reached": n_reached, "n_pore": n_pore}


def work(case):
    """Bytes and operations of the whole time loop: per flow iteration every
    population of a pore voxel read and written once; per transport step every
    concentration of a solute voxel read and written once and its face
    velocities read once; plus the call's own inputs and outputs."""
    if case["kind"] == "batch":
        n = ((case["lo"] + case["hi"]) / 2.0) ** 3 * case["count"]
        nf = 0.5 * n
        per_it, per_step = nf * 2 * 19 * 4, nf * (8 * 4.0 / 3.0 + 12)
        own = n * (1 + 12 + 20 * 4.0 / 3.0)
        return {"bytes": case["nit"] * per_it + case["steps"] * per_step + own,
                "flops": nf * (case["nit"] * 330.0 + case["steps"] * 130.0)}
    n = float(math.prod(_shape(case)))
    nf = case["porosity"] * n
    if case["kind"] == "walk":
        return {"bytes": n * (1 + 4), "flops": 6 * nf}
    if case["kind"] == "flow":
        q = 19 if case["nd"] == 3 else 9
        return {"bytes": case["nit"] * nf * 2 * q * STORED[case["precision"]] + n * (1 + 12),
                "flops": case["nit"] * nf * (330.0 if q == 19 else 150.0)}
    ns, mv, nd = SPECIES[case["kinetics"]], MOVING[case["kinetics"]], case["nd"]
    own = n * (1 + 12 + 4 * ns * case["n_t"])
    return {"bytes": case["steps"] * nf * (8.0 * ns + 4.0 * nd) + own,
            "flops": case["steps"] * nf * (mv * nd * 36.0 + 10.0 * ns)}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
E3 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0),
      (-1, -1, 0), (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1),
      (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1)]
W3 = [1 / 3.] + [1 / 18.] * 6 + [1 / 36.] * 12
E2 = [(0, 0), (1, 0), (0, 1), (-1, 0), (0, -1), (1, 1), (-1, 1), (-1, -1), (1, -1)]
W2 = [4 / 9.] + [1 / 9.] * 4 + [1 / 36.] * 4


def _exact_flow(g, nit, force, tau=0.8, magic=3.0 / 16.0):
    """(velocity, permeability) after nit iterations, float64."""
    dev = _device()
    E, W = (E3, W3) if g.ndim == 3 else (E2, W2)
    nd, n, q = g.ndim, g.size, len(W)
    opp = torch.tensor([E.index(tuple(-c for c in e)) for e in E], device=dev)
    Ef = torch.tensor(E, dtype=torch.float64, device=dev)
    w = torch.tensor(W, dtype=torch.float64, device=dev).reshape(-1, 1)
    pore = torch.from_numpy(g == PORE).to(dev).reshape(-1)
    at = torch.arange(n, device=dev).reshape(g.shape)
    pull = torch.stack([i * n + at.roll(e, tuple(range(nd))).reshape(-1)
                        for i, e in enumerate(E)]).reshape(-1)
    om_p = 1.0 / tau
    om_m = 1.0 / (magic / (tau - 0.5) + 0.5)
    guo = w * (1 - 0.5 * om_m) * 3.0 * force * Ef[:, :1]
    half = torch.zeros((nd, 1), dtype=torch.float64, device=dev)
    half[0] = 0.5 * force
    f = w.expand(q, n).contiguous()
    for _ in range(nit):
        rho = f.sum(0)
        u = (Ef.T @ f + half) / rho * pore
        eu = Ef @ u
        feq = w * rho * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * (u * u).sum(0))
        fo, d = f[opp], f - feq
        do = d[opp]
        post = f - (0.5 * om_p) * (d + do) - (0.5 * om_m) * (d - do) + guo
        f = torch.where(pore, post, fo).reshape(-1)[pull].reshape(q, n)
    v = torch.zeros((3, n), dtype=torch.float64, device=dev)
    v[:nd] = (Ef.T @ f + half) / f.sum(0) * pore
    k = (tau - 0.5) / 3.0 * float(v[0].mean()) / force
    return v.reshape((3,) + g.shape).cpu().numpy(), k


def _take(a, ax, off):
    """`a` shifted by `off` along an axis, its edge values repeated."""
    n = a.shape[ax]
    return a.index_select(ax, (torch.arange(n, device=a.device) + off).clamp(0, n - 1))


def _limited(up, upup, down):
    d1, d2 = down - up, up - upup
    return up + 0.25 * (torch.sign(d1) + torch.sign(d2)) * torch.minimum(d1.abs(), d2.abs())


def _wanted(total, n_t):
    if n_t == 1:
        return [total]
    if n_t == 2:
        return [0, total]
    tail = np.geomspace(max(total // 400, 1), max(total, 1), n_t - 1)
    return [int(v) for v in np.round(np.concatenate([[0.0], tail]))]


def _picked(steps, n_t, ratio=1.12):
    """The step numbers of the n_t snapshots kept of a run of `steps` steps."""
    kept, nxt = [0], 1
    while nxt <= steps:
        kept.append(nxt)
        nxt = max(nxt + 1, int(math.ceil(nxt * ratio)))
    if kept[-1] != steps:
        kept.append(steps)
    used, got = set(), []
    for want in _wanted(steps, n_t):
        i = int(np.abs(np.asarray(kept) - want).argmin())
        for d in range(len(kept)):
            free = [j for j in (i - d, i + d) if 0 <= j < len(kept) and j not in used]
            if free:
                i = free[0]
                break
        used.add(i)
        got.append(kept[i])
    return got


def _exact_transport(g, vel, case, chem):
    """(snapshots, their normalised times) of a fixed-step run, float64."""
    dev = _device()
    nd, ns = g.ndim, SPECIES[case["kinetics"]]
    grid = torch.from_numpy(g).to(dev)
    bf = grid == (chem.biofilm_code if chem.biofilm_code is not None else 255)
    m = (grid == PORE) | bf
    v = torch.from_numpy(np.asarray(vel)).to(dev).double()[:nd]
    axial, speed = float(v[0][m].mean()), float((v * v).sum(0).sqrt()[m].mean())
    u = v / (axial if axial > 0.1 * speed else speed) * m
    l_ref = float(g.shape[0])
    D, k = l_ref / case["pe"], case["da"] / l_ref
    kd = chem.decay_for(l_ref)
    still = [bool(b) for b in chem.immobile]
    dp = [0.0 if still[j] else float(chem.d_rel[j]) * D for j in range(ns)]
    db = [0.0 if still[j] else float(chem.d_biofilm_rel[j]) * D for j in range(ns)]
    worst = max([p / D for p in dp] + ([p / D for p in db] if bool(bf.any()) else []) + [1.0])
    umax = sum(float(u[a].abs().max()) for a in range(nd))
    half = [chem.ks_donor] + ([chem.ks_acceptor] if ns > 1 else [])
    k_lin = max([k] + [k / ks for ks in half if ks > 0])
    sorp = chem.sorption
    if sorp is not None:
        ksorp = sorp.da / l_ref
        k_lin += ksorp * (1.0 + 1.0 / sorp.kd)
    dt = 0.4 / (umax + 2.0 * nd * D * worst + k_lin + kd)
    moving = [j for j in range(ns) if not still[j]]
    faces = []
    for a in range(nd):
        ol, oh = m & _take(m, a, -1), m & _take(m, a, 1)
        fl, fh = ol & _take(m, a, -2), oh & _take(m, a, 2)
        ul = torch.where(ol, 0.5 * (u[a] + _take(u[a], a, -1)), 0.0)
        uh = torch.where(oh, 0.5 * (u[a] + _take(u[a], a, 1)), 0.0)
        dd = []
        for j in moving:
            here = torch.where(bf, db[j], dp[j]).double()
            lo, hi = _take(here, a, -1), _take(here, a, 1)
            dd.append((torch.where(ol, 2 * here * lo / (here + lo), 0.0),
                       torch.where(oh, 2 * here * hi / (here + hi), 0.0)))
        faces.append((ol, oh, fl, fh, ul, uh, ul >= 0, uh >= 0, dd))
    divu = sum(f[5] - f[4] for f in faces)

    def moved(C, p):
        out = C * divu
        for a in range(nd):
            ol, oh, fl, fh, ul, uh, pl, ph, dd = faces[a]
            m1, p1 = torch.where(ol, _take(C, a, -1), C), torch.where(oh, _take(C, a, 1), C)
            m2, p2 = torch.where(fl, _take(C, a, -2), m1), torch.where(fh, _take(C, a, 2), p1)
            out = out + dd[p][1] * (p1 - C) + dd[p][0] * (m1 - C)
            hi = _limited(torch.where(ph, C, p1), torch.where(ph, m1, p2), torch.where(ph, p1, C))
            lo = _limited(torch.where(pl, m1, C), torch.where(pl, m2, p1), torch.where(pl, C, m1))
            out = out - (uh * hi - ul * lo)
        return out

    def reacted(C):
        dC = [torch.zeros_like(C[0]) for _ in range(ns)]
        if chem.biotic_on:
            R = k * C[0] / (chem.ks_donor + C[0]) if chem.ks_donor > 0 else k * C[0]
            if ns > 1:
                R = R * (C[1] / (chem.ks_acceptor + C[1]) if chem.ks_acceptor > 0 else C[1])
            if chem.biomass_coupled and ns > 3:
                R = R * C[3] / float(chem.c_init[3])
            lim = C[0] / dt
            if ns > 1 and chem.alpha > 0:
                lim = torch.minimum(lim, C[1] / (chem.alpha * dt))
            R = torch.minimum(R, 0.5 * lim)
            dC[0] = -R
            if ns > 1:
                dC[1] = -chem.alpha * R
            if ns > 2:
                dC[2] = (1.0 - (chem.yield_ if ns > 3 else 0.0)) * R
            if ns > 3:
                dC[3] = chem.yield_ * R - kd * C[3]
        if sorp is not None:
            c, s = C[sorp.dissolved], C[sorp.sorbed]
            r = torch.minimum(ksorp * (c - s / sorp.kd), 0.5 * c / dt)
            r = torch.maximum(r, -0.5 * s / dt)
            dC[sorp.dissolved] = dC[sorp.dissolved] - r
            dC[sorp.sorbed] = dC[sorp.sorbed] + r
        return dC

    C = []
    for j in range(ns):
        start = float(np.float32(chem.c_init[j]))
        where = bf if (j == 3 and chem.seed_in_biofilm and bool(bf.any()) and still[j]) else m
        C.append(torch.where(where, start, 0.0).double())
    got = _picked(case["steps"], case["n_t"])
    snaps = {0: torch.stack(C)}
    for n in range(1, case["steps"] + 1):
        for j in moving:
            if chem.inlet[j] == chem.inlet[j]:
                C[j][0] = torch.where(m[0], float(chem.inlet[j]), C[j][0])
        dC = reacted(C)
        for p, j in enumerate(moving):
            dC[j] = dC[j] + moved(C[j], p)
        C = [torch.where(m, (C[j] + dt * dC[j]).clamp(min=0.0), 0.0) for j in range(ns)]
        if n in got:
            snaps[n] = torch.stack(C)
    out = torch.stack([snaps[n] for n in got])
    return out.cpu().numpy(), np.asarray(got, np.float64) / max(case["steps"], 1)


def exact(case, seed):
    state = prepare(case, seed)
    if case["kind"] == "flow":
        vel, k = _exact_flow(state["g"], case["nit"], FORCE)
        return {"vel": vel, "permeability": k, "iters": None}
    if case["kind"] == "transport":
        out, t_norm = _exact_transport(state["g"], state["v"], case, state["chem"])
        return {"out": out, "t_norm": t_norm}
    if case["kind"] == "batch":
        found = []
        for r in state["requests"]:
            vel, _ = _exact_flow(r.mat, case["nit"], FORCE)
            d = {"pe": r.adr["pe"], "da": r.adr["da"], "n_t": 5, "steps": case["steps"],
                 "kinetics": {"monod": "monod", "first order": "first_order"}.get(
                     r.adr["chem"].source, "sorption")}
            found.append({"vel": vel, "out": _exact_transport(r.mat, vel, d, r.adr["chem"])[0]})
        return found
    return None  # whole numbers
