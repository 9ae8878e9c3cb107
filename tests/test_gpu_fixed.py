"""The FMA build's fixed-point kernels and their FP64 route for elements the
formats do not hold, against the strict build's IEEE kernels on the same state:
meshes of one element up to sizes that are no multiple of a block, regular,
worn, flattened, far from unit scale, at rest, and inverted."""
import numpy as np
import pytest

from paritylib import field_rel_err

pytestmark = pytest.mark.gpu

H = 1.125


def _state(nx, kind, seed=3):
    r = np.random.default_rng(seed)
    g = H * np.arange(nx + 1) / nx
    z, y, x = (a.reshape(-1).copy() for a in np.meshgrid(g, g, g, indexing="ij"))
    n, E = x.size, nx ** 3
    jit = {"worn": 0.2, "bent": 0.08}.get(kind, 0.02) * H / nx
    scale = {"huge": 2.0 ** 62, "tiny": 2.0 ** -40}.get(kind, 1.0)
    flat = 1e-3 if kind == "flat" else 1.0
    s = {}
    for f, c, a in (("x", x, 1.0), ("y", y, 1.0), ("z", z, flat)):
        on = c > 0  # the symmetry planes stay planes
        s[f] = (c + np.where(on, jit * r.uniform(-1, 1, n), 0.0)) * a * scale
        s[f + "d"] = np.where(on, 30.0 * c + r.uniform(-1, 1, n), 0.0) * a
    if kind == "still":
        for f in ("xd", "yd", "zd"):
            s[f][:] = 0.0
    if kind == "inverted":
        s["x"][1], s["x"][0] = s["x"][0], s["x"][1] + 0.5 * H / nx
    heat = 1e3 * flat ** 2
    s["e"] = r.uniform(0.5, 1.0, E) * heat
    s["v"] = np.ones(E)
    s["p"] = 2.0 / 3.0 * s["e"]
    s["q"] = r.uniform(0, 0.1, E) * s["p"]
    if kind == "still":
        for f in ("e", "p", "q"):
            s[f][:] = 0.0
    s["ss"] = np.sqrt(10.0 / 9.0 * s["e"] + 1e-30)
    vol = (H / nx) ** 3 * flat * scale ** 3
    s["volo"] = np.full(E, vol * (1e10 if kind == "squeezed" else 1.0))
    s["elemMass"] = np.full(E, vol)
    s["dt"] = 1e-3 * (H / nx) / 60.0 * min(scale, 1.0)
    return s


def _run(lg, precision, nx, kind):
    s = _state(nx, kind)
    d = lg.Domain(nx, numReg=5, its=10 ** 9, precision=precision,
                  hgcoef=0.0 if kind == "nohourglass" else 2.5)
    mass = d.field("nodalMass") / d.field("volo")[0] * s["elemMass"][0]
    d.set_field("nodalMass", mass)
    dt = s.pop("dt")
    for f, v in s.items():
        d.set_field(f, v)
    d.set_scalar("deltatime", dt)
    status = [d.phase(1), d.phase(2), d.phase(3)]
    out = {f: d.field(f) for f in ("fx", "fy", "fz", "x", "y", "z", "xd", "yd", "zd", "vnew",
                                   "arealg", "vdov", "delx_xi", "delx_eta", "delx_zeta", "delv_xi",
                                   "delv_eta", "delv_zeta", "e", "p", "q", "ss", "v")}
    out["dtcourant"] = np.array([d.scalar("dtcourant")])
    return status, out


KINDS = ["regular", "bent", "worn", "flat", "huge", "tiny", "still", "nohourglass", "squeezed",
         "inverted"]


@pytest.mark.parametrize("nx", [1, 5, 11])
@pytest.mark.parametrize("kind", KINDS)
def test_fma_build_matches_strict(native_lib, kind, nx):
    import lulesh_gb300 as lg
    st0, a = _run(lg, "fp64", nx, kind)
    st1, b = _run(lg, "fp64-fma", nx, kind)
    assert st0 == st1
    if any(st0):
        return
    worst = {}
    for f, want in a.items():
        # A relative error on the field's own scale.  Both builds round each
        # term at 2^-53; coordinates of magnitude nx edges and the cancelling
        # sums of a worn element raise that by a few hundred.
        scale = np.max(np.abs(want))
        worst[f] = field_rel_err(b[f], want, floor=1e-3) if scale else float(np.max(np.abs(b[f])))
    print(kind, nx, max(worst.items(), key=lambda kv: kv[1]))
    assert max(worst.values()) <= 1e-10, worst
