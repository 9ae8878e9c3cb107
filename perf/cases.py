"""Timed cases: what a program that uses this framework has it do.

A case is a dict of plain values.  Its "kind" is one of the framework's entry
points and the pattern a program calls it in:

  sedov     Domain: reset, step(cycles), read back the state the cycle carries
            (the reference's main run, and one point of a parameter study)
  restart   Domain: upload a mid-run state, step(cycles), read the state back
            (checkpoint / restart, and coupling to a host code)
  ensemble  Ensemble: reset, step(cycles), read every member's state
  energy    autograd.TerminalEnergy: objective and both gradients
  field     autograd.FinalEnergyField: final energy field, then the gradients
            of a loss of it (forward run, checkpointed reverse sweep)
  halo      HaloPlan: pack and unpack of one rank's messages

The sizes are those of the command line's default (s=30), the benchmark
(s=150, s=192, s=30, 64-problem ensembles of s=16..64), the tests (s=8..64)
and odd sizes between them.
"""
import math

import numpy as np
import torch

import lulesh_gb300 as lg
from lulesh_gb300 import autograd as lga

CARRIED = ("x", "y", "z", "xd", "yd", "zd", "e", "p", "q", "v", "ss")
NODAL = frozenset(CARRIED[:6])
EXTENT = 1.125  # edge of the Sedov box


def listed():
    return [
        # a small run of the tests and of interactive use: launches and latency
        {"name": "sedov-s10-fp64", "kind": "sedov", "nx": 10, "regions": 11, "balance": 1,
         "cost": 1, "precision": "fp64", "cycles": 100},
        # the command line's default problem and arithmetic
        {"name": "sedov-s30-fp64", "kind": "sedov", "nx": 30, "regions": 11, "balance": 1,
         "cost": 1, "precision": "fp64", "cycles": 100},
        # the same problem in the benchmark's arithmetic
        {"name": "sedov-s30-fma", "kind": "sedov", "nx": 30, "regions": 11, "balance": 1,
         "cost": 1, "precision": "fp64-fma", "cycles": 100},
        # a checkpoint picked up mid-run on an odd mesh, few cycles between checkpoints
        {"name": "restart-s45-fma", "kind": "restart", "nx": 45, "regions": 11, "balance": 1,
         "cost": 1, "precision": "fp64-fma", "cycles": 20},
        # the same on a larger mesh in the uncontracted arithmetic
        {"name": "restart-s80-fp64", "kind": "restart", "nx": 80, "regions": 16, "balance": 2,
         "cost": 4, "precision": "fp64", "cycles": 10},
        # the benchmark's headline problem
        {"name": "sedov-s150-fma", "kind": "sedov", "nx": 150, "regions": 11, "balance": 1,
         "cost": 1, "precision": "fp64-fma", "cycles": 20},
        # the benchmark's mixed-precision problem: costly regions, the largest mesh
        {"name": "sedov-s192-mixed", "kind": "sedov", "nx": 192, "regions": 16, "balance": 2,
         "cost": 4, "precision": "mixed", "cycles": 20},
        # mixed precision mid-run on a mid-sized odd mesh
        {"name": "restart-s71-mixed", "kind": "restart", "nx": 71, "regions": 16, "balance": 2,
         "cost": 4, "precision": "mixed", "cycles": 30},
        # an ensemble study's batch
        {"name": "ensemble-16-fma", "kind": "ensemble", "members": 16, "low": 16, "high": 40,
         "precision": "fp64-fma", "cycles": 60},
        # one gradient of the terminal energy (default arithmetic)
        {"name": "energy-s32-fp64", "kind": "energy", "nx": 32, "regions": 11, "cycles": 40,
         "ckpt": 10, "precision": "fp64"},
        # one step of an inversion of the final energy field
        {"name": "field-s20-fma", "kind": "field", "nx": 20, "regions": 11, "cycles": 25,
         "ckpt": 5, "precision": "fp64-fma"},
        # force exchange of an interior rank of a 3 x 3 x 3 decomposition
        {"name": "halo-sbn-s150", "kind": "halo", "exchange": "sbn", "nx": 150, "fields": 3},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


# element-cycles per microsecond on this part, to keep a drawn pass below the
# largest listed one
_RATE = {"fp64": 150.0, "fp64-fma": 250.0, "mixed": 450.0}


def draw(rng):
    kind = rng.choice(("sedov", "sedov", "restart", "restart", "ensemble", "energy", "field",
                       "halo"))
    if kind in ("sedov", "restart"):
        precision = rng.choice(("fp64", "fp64-fma", "mixed"))
        nx = _log_int(rng, 8, 160 if precision == "mixed" else 120)
        top = int(120e3 * _RATE[precision] / nx ** 3)
        return {"kind": kind, "nx": nx, "regions": rng.choice((1, 4, 11, 16)),
                "balance": rng.choice((1, 2)), "cost": rng.choice((1, 1, 4)),
                "precision": precision, "cycles": max(1, min(_log_int(rng, 3, 120), top))}
    if kind == "ensemble":
        low = rng.randint(8, 24)
        members, high = rng.randint(3, 24), low + rng.randint(4, 24)
        return {"kind": kind, "members": members, "low": low, "high": high,
                "precision": rng.choice(("fp64", "fp64-fma", "fp64-fma", "mixed")),
                "cycles": max(1, min(rng.randint(5, 80), int(12e6 / (members * high ** 3))))}
    if kind in ("energy", "field"):
        return {"kind": kind, "nx": _log_int(rng, 6, 32), "regions": rng.choice((4, 11)),
                "cycles": rng.randint(4, 40), "ckpt": rng.randint(2, 12),
                "precision": rng.choice(("fp64", "fp64-fma"))}
    exchange = rng.choice(("sbn", "sync_pos_vel", "monoq"))
    return {"kind": kind, "exchange": exchange, "nx": _log_int(rng, 8, 200),
            "fields": {"sbn": rng.choice((1, 3)), "sync_pos_vel": 6, "monoq": 3}[exchange]}


def _rng(seed):
    return np.random.default_rng([7, seed])


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def _carried_buffers(nodes, elems):
    return {f: _pinned(nodes if f in NODAL else elems) for f in CARRIED}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _sedov_choice(seed):
    """hgcoef and energy factor in the ranges of the ensemble study."""
    r = _rng(seed)
    return float(r.uniform(1.0, 3.0)), float(2.0 ** r.uniform(-1.0, 1.0))


def _members(case, seed):
    r = _rng(seed)
    # mesh sizes and regions by the case, so that every seed does the same work
    shape = np.random.default_rng([case["members"], case["low"], case["high"]])
    out = []
    for _ in range(case["members"]):
        out.append({"nx": int(shape.integers(case["low"], case["high"] + 1)),
                    "numReg": int(shape.integers(4, 17)), "balance": 1, "cost": 1,
                    "its": 10 ** 9, "hgcoef": float(r.uniform(1.0, 3.0)),
                    "einit_factor": float(2.0 ** r.uniform(-1.0, 1.0))})
    return out


def _lattice(nx, device):
    g = EXTENT * torch.arange(nx + 1, dtype=torch.float64, device=device) / nx
    z, y, x = torch.meshgrid(g, g, g, indexing="ij")
    return x.reshape(-1).clone(), y.reshape(-1).clone(), z.reshape(-1).clone()


def _mid_run(nx, seed, device):
    """A blast partway through the box: nodes displaced and moving outward,
    energy behind the front, the rest of the mesh at rest."""
    r = _rng(seed)
    gen = torch.Generator().manual_seed(int(r.integers(1 << 40)))
    front, push, speed, heat = (float(r.uniform(*b)) for b in
                                ((0.45, 0.8), (0.15, 0.3), (20.0, 60.0), (500.0, 4000.0)))
    X, Y, Z = _lattice(nx, device)
    R = torch.sqrt(X * X + Y * Y + Z * Z)
    s = torch.clamp(R / front, max=1.0)
    inside = (s < 1.0).double()
    stretch = 1.0 + push * (1.0 - s) * inside
    noise = [1.0 + 0.05 * torch.rand(X.shape, generator=gen, dtype=torch.float64).to(device)
             for _ in range(3)]
    m = _mesh([nx], device)
    st = {}
    for f, c, w in zip("xyz", (X, Y, Z), noise):
        st[f] = c * stretch
        st[f + "d"] = speed * s * inside * w * c / torch.clamp(R, min=1e-12)
    h = EXTENT / nx
    xc, yc, zc = (st[f][m["corner"]] for f in "xyz")
    st["v"] = _volume(xc, yc, zc) / h ** 3
    st["v"] = torch.where((st["v"] - 1.0).abs() < 1e-10, torch.ones_like(st["v"]), st["v"])
    centre = torch.sqrt(xc.mean(0) ** 2 + yc.mean(0) ** 2 + zc.mean(0) ** 2)
    hot = (centre < front).double()
    wave = torch.rand(centre.shape, generator=gen, dtype=torch.float64).to(device)
    st["e"] = heat * hot * (1.2 - centre / front) * (1.0 + 0.02 * wave)
    st["p"] = (2.0 / 3.0) * st["e"] / st["v"]
    st["q"] = 0.05 * st["p"] * wave
    st["ss"] = torch.sqrt(torch.clamp((2.0 / 3.0) * st["e"] + st["v"] ** 2 * (2.0 / 3.0) /
                                      st["v"] * st["p"], min=.1111111e-36))
    dt = 0.1 * h / (speed + math.sqrt(1.2 * heat))
    t = {"time": 1e-3, "deltatime": dt, "dtcourant": 2.0 * dt, "dthydro": 1e20, "cycle": 100}
    return st, t


def _study(case, seed):
    """Initial energies with noise, hgcoef, constant time steps and the
    element mask of a gradient study."""
    r = _rng(seed)
    nx = case["nx"]
    E = nx ** 3
    e = np.zeros(E)
    e[0] = 3.948746e+7 * (nx / 45.0) ** 3
    at = r.permutation(E)[: max(1, min(E // 4, 1000))]
    e[at] += 1e-4 * e[0] * r.uniform(0.2, 1.0, at.size)
    dt = 0.25 * (EXTENT / nx) / math.sqrt(2.0 * e[0])
    c = (np.arange(nx) + 0.5) / nx
    mask = (c[:, None, None] ** 2 + c[None, :, None] ** 2 + c[None, None, :] ** 2 < 0.2).reshape(-1)
    return e, float(r.uniform(1.5, 3.0)), np.full(case["cycles"], dt), mask


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("sedov", "restart"):
        nx = case["nx"]
        hg, factor = _sedov_choice(seed)
        d = lg.Domain(nx, case["regions"], case["balance"], case["cost"], its=10 ** 9,
                      precision=case["precision"], hgcoef=hg, einit_factor=factor)
        st = {"case": case, "dom": d, "out": _carried_buffers(d.numNode, d.numElem)}
        if kind == "restart":
            fields, st["time"] = _mid_run(nx, seed, "cuda")
            st["in"] = _carried_buffers(d.numNode, d.numElem)
            for f in CARRIED:
                st["in"][f][:] = fields[f].cpu().numpy()
        return st
    if kind == "ensemble":
        members = _members(case, seed)
        return {"case": case, "members": members,
                "ens": lg.Ensemble(members, precision=case["precision"])}
    if kind in ("energy", "field"):
        e, hg, dts, mask = _study(case, seed)
        prob = lga.TerminalEnergyProblem(case["nx"], case["regions"], case["cycles"],
                                         case["ckpt"], e_base=e, precision=case["precision"],
                                         dts=dts, mask=mask)
        weight = torch.from_numpy(_rng(seed + 1).uniform(0.5, 1.5, e.size))
        return {"case": case, "prob": prob, "e0": torch.from_numpy(e),
                "hg": torch.tensor(hg, dtype=torch.float64), "weight": weight}
    plan = lg.HaloPlan(case["exchange"], case["nx"], 3, 13, case["fields"])  # the centre rank
    info = plan.info()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    length = info["field_length"]

    def values(n):
        return torch.rand(n, generator=gen, dtype=torch.float64, device="cuda")
    return {"case": case, "plan": plan, "fields": [values(length) for _ in range(case["fields"])],
            "send": torch.zeros(info["buffer_doubles"], dtype=torch.float64, device="cuda"),
            "recv": values(info["buffer_doubles"]),
            "base": [values(length) for _ in range(case["fields"])]}


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind in ("sedov", "restart"):
        d = st["dom"]
        if kind == "sedov":
            d.reset()
        else:
            for f in CARRIED:
                d.set_field(f, st["in"][f])
            for k, v in st["time"].items():
                d.set_scalar(k, v)
        d.step(case["cycles"], check=True)
        return {f: d.field(f, out=st["out"][f]) for f in CARRIED}
    if kind == "ensemble":
        en = st["ens"]
        en.reset()
        en.step(case["cycles"])
        n = len(st["members"])
        return {f: np.concatenate([en.field(i, f) for i in range(n)]) for f in CARRIED}
    if kind in ("energy", "field"):
        e0 = st["e0"].clone().requires_grad_(True)
        hg = st["hg"].clone().requires_grad_(True)
        if kind == "energy":
            out = lga.TerminalEnergy.apply(e0, hg, st["prob"])
            out.backward()
        else:
            out = lga.FinalEnergyField.apply(e0, hg, st["prob"])
            (out * st["weight"]).sum().backward()
        return {"value": out.detach(), "grad_e": e0.grad, "grad_hgcoef": hg.grad}
    fields = st["fields"]
    for f, b in zip(fields, st["base"]):
        f.copy_(b)
    stream = torch.cuda.current_stream().cuda_stream or None
    st["plan"].pack(fields, st["send"], stream)
    st["plan"].unpack(fields, st["recv"], stream)
    return {"send": st["send"], "fields": fields}


def work(case):
    """Bytes: the carried state and constants of each cycle read and written
    once (266 B per element-cycle), and the state's way to the host.  Flops:
    the cycle's operations with every term formed once."""
    kind = case["kind"]
    if kind == "halo":
        surface = 6 * (case["nx"] + 1) ** 2 * case["fields"]
        return {"bytes": 8.0 * surface * 4, "flops": float(surface)}
    if kind == "ensemble":
        elems = sum(m["nx"] ** 3 for m in _members(case, 0))
    else:
        elems = case["nx"] ** 3
    cycles = case["cycles"] * (3 if kind in ("energy", "field") else 1)
    reps = 3.0 if case.get("cost", 1) == 1 else 8.0  # average EOS repetitions
    return {"bytes": 266.0 * elems * cycles + 88.0 * elems,
            "flops": (1500.0 + 70.0 * reps) * elems * cycles}


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch
# ---------------------------------------------------------------------------
_FACES = ((0, 1, 2, 3), (0, 4, 5, 1), (1, 5, 6, 2), (2, 6, 7, 3), (3, 7, 4, 0), (4, 7, 6, 5))
_GAMMA = ((1, 1, -1, -1, -1, -1, 1, 1), (1, -1, -1, 1, -1, 1, 1, -1),
          (1, -1, 1, -1, 1, -1, 1, -1), (-1, 1, -1, 1, 1, -1, 1, -1))
_VOLU = ((1, 2, 3, 4, 5, 7), (2, 3, 0, 5, 6, 4), (3, 0, 1, 6, 7, 5), (0, 1, 2, 7, 4, 6),
         (7, 6, 5, 0, 3, 1), (4, 7, 6, 1, 0, 2), (5, 4, 7, 2, 1, 3), (6, 5, 4, 3, 2, 0))


def _mesh(sizes, device):
    """Topology of meshes of the given edges laid end to end."""
    corner, face = [], {k: [] for k in ("xim", "xip", "etam", "etap", "zetam", "zetap")}
    openp = {k: [] for k in ("xip", "etap", "zetap")}
    symm, eown, nown = {k: [] for k in "xyz"}, [], []
    noff = eoff = 0
    for i, nx in enumerate(sizes):
        n = nx + 1
        k = torch.arange(nx, device=device)
        pl, ro, co = torch.meshgrid(k, k, k, indexing="ij")
        pl, ro, co = pl.reshape(-1), ro.reshape(-1), co.reshape(-1)
        base = noff + (pl * n + ro) * n + co
        corner.append(torch.stack([base, base + 1, base + n + 1, base + n, base + n * n,
                                   base + n * n + 1, base + n * n + n + 1, base + n * n + n]))
        el = eoff + (pl * nx + ro) * nx + co
        for key, c, d in (("xi", co, 1), ("eta", ro, nx), ("zeta", pl, nx * nx)):
            face[key + "m"].append(torch.where(c > 0, el - d, el))
            face[key + "p"].append(torch.where(c < nx - 1, el + d, el))
            openp[key + "p"].append(c == nx - 1)
        k = torch.arange(n, device=device)
        pz, ry, cx = torch.meshgrid(k, k, k, indexing="ij")
        for key, c in (("x", cx), ("y", ry), ("z", pz)):
            symm[key].append((c == 0).reshape(-1))
        eown.append(torch.full((nx ** 3,), i, device=device))
        nown.append(torch.full((n ** 3,), i, device=device))
        noff += n ** 3
        eoff += nx ** 3
    m = {"corner": torch.cat(corner, 1), "eown": torch.cat(eown), "nown": torch.cat(nown),
         "nodes": noff, "elems": eoff, "count": len(sizes)}
    for k, v in face.items():
        m[k] = torch.cat(v)
    for k, v in openp.items():
        m["free_" + k] = torch.cat(v)
    for k, v in symm.items():
        m["symm_" + k] = torch.cat(v)
    return m


def _volume(x, y, z):
    def tri(a, b, c):
        return (a[0] * (b[1] * c[2] - b[2] * c[1]) + a[1] * (b[2] * c[0] - b[0] * c[2]) +
                a[2] * (b[0] * c[1] - b[1] * c[0]))

    def d(i, j):
        return (x[i] - x[j], y[i] - y[j], z[i] - z[j])

    def add(a, b):
        return tuple(p + q for p, q in zip(a, b))
    return (tri(add(d(3, 1), d(7, 2)), d(6, 3), d(2, 0)) +
            tri(add(d(4, 3), d(5, 7)), d(6, 4), d(7, 0)) +
            tri(add(d(1, 4), d(2, 5)), d(6, 1), d(5, 0))) / 12.0


def _cross(a, b):
    return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])


def _forces(m, s, hg):
    """Nodal stress and hourglass forces."""
    pos = [s[f][m["corner"]] for f in "xyz"]
    vel = [s[f + "d"][m["corner"]] for f in "xyz"]
    sig = -s["p"] - s["q"]
    normal = [[0.0] * 8 for _ in range(3)]
    for a, b, c, d in _FACES:
        u = [0.5 * (p[d] + p[c] - p[b] - p[a]) for p in pos]
        w = [0.5 * (p[c] + p[b] - p[d] - p[a]) for p in pos]
        for k, area in enumerate(_cross(u, w)):
            for j in (a, b, c, d):
                normal[k][j] = normal[k][j] + 0.25 * area
    det = s["volo"] * s["v"]
    x, y, z = pos
    dv = [[], [], []]
    for n0, n1, n2, n3, n4, n5 in _VOLU:
        for k, (a, b) in enumerate(((y, z), (z, x), (x, y))):
            dv[k].append(((a[n1] + a[n2]) * (b[n0] + b[n1]) - (a[n0] + a[n1]) * (b[n1] + b[n2]) +
                          (a[n0] + a[n4]) * (b[n3] + b[n4]) - (a[n3] + a[n4]) * (b[n0] + b[n4]) -
                          (a[n2] + a[n5]) * (b[n3] + b[n5]) + (a[n3] + a[n5]) * (b[n2] + b[n5]))
                         / 12.0)
    coef = -hg * 0.01 * s["ss"] * s["elemMass"] / det.pow(1.0 / 3.0)
    force = [[-(sig * normal[k][j]) for j in range(8)] for k in range(3)]
    for g in _GAMMA:
        mode = [sum(g[j] * p[j] for j in range(8)) / det for p in pos]
        h = [g[j] - (dv[0][j] * mode[0] + dv[1][j] * mode[1] + dv[2][j] * mode[2])
             for j in range(8)]
        for k in range(3):
            amp = coef * sum(h[j] * vel[k][j] for j in range(8))
            for j in range(8):
                force[k][j] = force[k][j] + amp * h[j]
    total = []
    for k in range(3):
        t = torch.zeros(m["nodes"], dtype=torch.float64, device=sig.device)
        for j in range(8):  # the nodes of one corner number are distinct
            t[m["corner"][j]] += force[k][j]
        total.append(t)
    return total


def _limiter(m, dv, key):
    norm = 1.0 / (dv + 1e-36)
    lo = dv[m[key + "m"]] * norm
    hi = torch.where(m["free_" + key + "p"], torch.zeros_like(dv), dv[m[key + "p"]]) * norm
    phi = torch.minimum(torch.minimum(0.5 * (lo + hi), 2.0 * lo), 2.0 * hi)
    return phi.clamp(0.0, 1.0)


def _cut(a, eps):
    return torch.where(a.abs() < eps, torch.zeros_like(a), a)


def _pressure(e, comp):
    b = (2.0 / 3.0) * (comp + 1.0)
    return _cut(b * e, 1e-7).clamp(min=0.0), b


def _sound(e, v, b, p):
    c = (2.0 / 3.0) * e + v * v * b * p
    return torch.where(c <= .1111111e-36, torch.full_like(c, .3333333e-18),
                       torch.sqrt(c.clamp(min=.1111111e-36)))


def _cycle(m, s, hg, dt):
    """One cycle in place; dt per member.  Returns the Courant and hydro
    limits per member."""
    dtn, dte = dt[m["nown"]], dt[m["eown"]]
    for f, F in zip("xyz", _forces(m, s, hg)):
        a = F / s["nodalMass"]
        a = torch.where(m["symm_" + f], torch.zeros_like(a), a)
        s[f + "d"] = _cut(s[f + "d"] + a * dtn, 1e-7)
        s[f] = s[f] + s[f + "d"] * dtn
    pos = [s[f][m["corner"]] for f in "xyz"]
    vel = [s[f + "d"][m["corner"]] for f in "xyz"]
    vol = _volume(*pos)
    vnew = vol / s["volo"]
    delv = vnew - s["v"]
    big = torch.zeros_like(vol)
    for a, b, c, d in ((0, 1, 2, 3), (4, 5, 6, 7), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6),
                       (3, 0, 4, 7)):
        n = _cross([p[c] - p[a] for p in pos], [p[d] - p[b] for p in pos])
        big = torch.maximum(big, 4.0 * (n[0] ** 2 + n[1] ** 2 + n[2] ** 2))
    arealg = 4.0 * vol / torch.sqrt(big)

    def dirs(c):
        a, b, d, e = c[6] - c[0], c[5] - c[3], c[7] - c[1], c[4] - c[2]
        return (a + b - d - e, a - b + d - e, a + b + d + e)
    P = [dirs(c) for c in pos]  # [coordinate][direction]
    V = [dirs(c) for c in vel]
    half = [[P[k][i] - 0.5 * dte * V[k][i] for i in range(3)] for k in range(3)]
    col = [[half[k][i] for k in range(3)] for i in range(3)]
    vcol = [[V[k][i] for k in range(3)] for i in range(3)]
    pcol = [[P[k][i] for k in range(3)] for i in range(3)]
    cof = [_cross(col[1], col[2]), _cross(col[2], col[0]), _cross(col[0], col[1])]
    det = sum(cof[0][k] * col[0][k] for k in range(3))
    vdov = sum(cof[i][k] * vcol[i][k] for i in range(3) for k in range(3)) / det
    vabs = s["volo"] * vnew
    norm = 1.0 / (vabs + 1e-36)
    delx, dvel = [], []
    for i in range(3):
        a = _cross([0.25 * w for w in pcol[(i + 1) % 3]], [0.25 * w for w in pcol[(i + 2) % 3]])
        delx.append(vabs / torch.sqrt(a[0] ** 2 + a[1] ** 2 + a[2] ** 2 + 1e-36))
        dvel.append(norm * 0.25 * sum(a[k] * vcol[i][k] for k in range(3)))
    rho = s["elemMass"] / vabs
    ql = qq = 0.0
    for i, key in enumerate(("xi", "eta", "zeta")):
        phi = _limiter(m, dvel[i], key)
        d = (dvel[i] * delx[i]).clamp(max=0.0)
        ql = ql + d * (1.0 - phi)
        qq = qq + d * d * (1.0 - phi * phi)
    still = vdov > 0.0
    ql = torch.where(still, torch.zeros_like(rho), -0.5 * rho * ql)
    qq = torch.where(still, torch.zeros_like(rho), (2.0 / 3.0) * rho * qq)

    comp, vhalf = 1.0 / vnew - 1.0, vnew - 0.5 * delv
    chalf = 1.0 / vhalf - 1.0
    e0, p0, q0, grow = s["e"], s["p"], s["q"], delv > 0.0
    zero = torch.zeros_like(e0)
    e = (e0 - 0.5 * delv * (p0 + q0)).clamp(min=-1e15)
    ph, b = _pressure(e, chalf)
    w = 1.0 / (1.0 + chalf)
    q = torch.where(grow, zero, _sound(e, w, b, ph) * ql + qq)
    e = e + 0.5 * delv * (3.0 * (p0 + q0) - 4.0 * (ph + q))
    e = _cut(e, 1e-7).clamp(min=-1e15)
    p, b = _pressure(e, comp)
    qt = torch.where(grow, zero, _sound(e, vnew, b, p) * ql + qq)
    e = e - (7.0 * (p0 + q0) - 8.0 * (ph + q) + (p + qt)) * delv / 6.0
    e = _cut(e, 1e-7).clamp(min=-1e15)
    p, b = _pressure(e, comp)
    q = torch.where(grow, q, _cut(_sound(e, vnew, b, p) * ql + qq, 1e-7))
    s["p"], s["e"], s["q"], s["ss"] = p, e, q, _sound(e, vnew, b, p)
    s["v"] = torch.where((vnew - 1.0).abs() < 1e-10, torch.ones_like(vnew), vnew)

    c = s["ss"] ** 2 + torch.where(vdov < 0.0, 256.0 * arealg ** 2 * vdov ** 2, zero)
    rest = vdov == 0.0  # an element at rest constrains nothing
    far = torch.full_like(c, 1e20)
    limits = []
    for w in (torch.where(rest, far, arealg / torch.sqrt(c)),
              torch.where(rest, far, 0.1 / (vdov.abs() + 1e-20))):
        lim = torch.full((m["count"],), 1e20, dtype=torch.float64, device=c.device)
        limits.append(lim.scatter_reduce(0, m["eown"], w, "amin"))
    return limits


def _next_dt(dt, time, courant, hydro, first):
    new = dt.clone()
    if not first:
        g = torch.full_like(dt, 1e20)
        g = torch.where(courant < g, courant / 2.0, g)
        g = torch.where(hydro < g, hydro * 2.0 / 3.0, g)
        ratio = g / dt
        new = torch.where((ratio >= 1.0) & (ratio < 1.1), dt,
                          torch.where(ratio > 1.2, dt * 1.2, g)).clamp(max=1e-2)
    target = 1e-2 - time
    target = torch.where((target > new) & (target < 4.0 * new / 3.0), 2.0 * new / 3.0, target)
    return torch.minimum(new, target)


def exact(case, seed):
    kind = case["kind"]
    if kind == "halo":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "ensemble":
        members = _members(case, seed)
    elif kind in ("energy", "field"):
        e, hg, dts, mask = _study(case, seed)
        members = [{"nx": case["nx"], "hgcoef": hg, "einit_factor": 1.0}]
    else:
        hg, factor = _sedov_choice(seed)
        members = [{"nx": case["nx"], "hgcoef": hg, "einit_factor": factor}]
    sizes = [q["nx"] for q in members]
    m = _mesh(sizes, dev)
    grids = [_lattice(n, dev) for n in sizes]
    s = {f: torch.cat([g[i] for g in grids]) for i, f in enumerate("xyz")}
    s["volo"] = _volume(*(s[f][m["corner"]] for f in "xyz"))
    s["elemMass"] = s["volo"]
    s["nodalMass"] = torch.zeros(m["nodes"], dtype=torch.float64, device=dev)
    for j in range(8):
        s["nodalMass"][m["corner"][j]] += s["volo"] / 8.0
    for f in ("xd", "yd", "zd"):
        s[f] = torch.zeros_like(s["x"])
    for f in ("e", "p", "q", "ss"):
        s[f] = torch.zeros_like(s["volo"])
    s["v"] = torch.ones_like(s["volo"])
    at, dt = 0, []
    for q in members:
        e0 = 3.948746e+7 * (q["nx"] / 45.0) ** 3 * q["einit_factor"]
        s["e"][at] = e0
        dt.append(0.5 * float(s["volo"][at]) ** (1.0 / 3.0) / math.sqrt(2.0 * e0))
        at += q["nx"] ** 3
    dt = torch.tensor(dt, dtype=torch.float64, device=dev)
    hgc = torch.tensor([q["hgcoef"] for q in members], dtype=torch.float64, device=dev)[m["eown"]]
    time, courant, hydro, first = torch.zeros_like(dt), dt * 0 + 1e20, dt * 0 + 1e20, True
    if kind in ("energy", "field"):
        s["e"] = torch.from_numpy(e).to(dev)
    if kind == "restart":
        fields, t = _mid_run(case["nx"], seed, dev)
        s.update(fields)
        time, courant, hydro, first = (dt * 0 + t["time"], dt * 0 + t["dtcourant"],
                                       dt * 0 + t["dthydro"], False)
        dt = dt * 0 + t["deltatime"]
    for c in range(case["cycles"]):
        dt = dt * 0 + float(dts[c]) if kind in ("energy", "field") else \
            _next_dt(dt, time, courant, hydro, first)
        courant, hydro = _cycle(m, s, hgc, dt)
        time, first = time + dt, False
    if kind == "field":
        return {"value": s["e"].cpu(), "grad_e": None, "grad_hgcoef": None}
    if kind == "energy":
        return {"value": (s["e"] * s["volo"])[torch.from_numpy(mask).to(dev)].sum().cpu(),
                "grad_e": None, "grad_hgcoef": None}
    return {f: s[f] for f in CARRIED}
