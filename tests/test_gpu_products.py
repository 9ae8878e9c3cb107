"""The strict build's forces and kinematics with their products and coordinate sums on the
integer pipes, by one thread and by three for each element, and their FP64 route for
elements the integers do not hold (the batched kernels), against the eight-lane
kernels' FP64 arithmetic: the same bits, on regular, worn, flattened, resting,
far-scaled and special meshes, at element counts that leave a warp incomplete."""
import numpy as np
import pytest

from test_gpu_fixed import _state

pytestmark = pytest.mark.gpu

FIELDS = ["fx", "fy", "fz", "x", "y", "z", "xd", "yd", "zd", "vnew", "v", "vdov", "arealg",
          "delv", "e", "p", "q", "ss"]


def _special(nx, kind):
    s = _state(nx, kind if kind in ("bent", "worn", "flat", "huge", "tiny", "still") else "worn")
    # powers of two outside the products' range in part (volumes) or altogether
    f = {"vast": 2.0 ** 190, "faint": 2.0 ** -190, "vanishing": 2.0 ** -300}.get(kind, 1.0)
    for c in "xyz":
        s[c] *= f
        if kind == "slow":  # velocities below the range beside ordinary ones
            s[c + "d"][::3] *= 2.0 ** -600
        if kind == "offset":  # coordinates of very different exponents in one element
            s[c] = np.where(s[c] == 0.0, 2.0 ** -40, s[c])
    if kind in ("vast", "faint"):
        s["volo"] = s["volo"] * f * f * f
        s["elemMass"] = s["elemMass"] * f * f * f
    if kind == "nan":
        s["xd"][-1] = np.nan
    return s


# the size of a second member: three threads for each element with the small one, one
# thread with the large one, whose members together take more than a wave of blocks
@pytest.mark.parametrize("fill", [4, 34])
@pytest.mark.parametrize("nx", [1, 3, 7, 11])
@pytest.mark.parametrize("kind", ["bent", "worn", "flat", "huge", "tiny", "still", "vast", "faint",
                                  "vanishing", "slow", "offset", "nan"])
def test_products_equal_fp64(native_lib, kind, nx, fill):
    import lulesh_gb300 as lg
    d = lg.Domain(nx, 5, 1, 1, its=10 ** 9, hgcoef=2.5)
    opts = dict(numReg=5, balance=1, cost=1, its=10 ** 9, hgcoef=2.5)
    e = lg.Ensemble([dict(nx=nx, **opts), dict(nx=fill, **opts)])
    s = _special(nx, kind)
    del s["dt"]
    for f, v in s.items():
        d.set_field(f, v)
        e.set_field(0, f, v)
    # the set-up's time step is far too long for some of these: the cycle's forces
    # are there all the same
    st = d.step(1)
    assert e.step(1) == st
    for f in FIELDS:
        a, b = d.field(f), e.field(0, f)
        same = (a.view(np.int64) == b.view(np.int64)) | (np.isnan(a) & np.isnan(b))
        assert same.all(), (f, int((~same).sum()))
