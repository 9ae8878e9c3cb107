"""The FMA build's velocity rates where the velocity components differ in size: a stream
or a shear in x beside a compression of 1e-3 to 1e-8 of it in y, on a regular mesh, where
the rates are quotients of differences.  A tilt below the fixed-point cofactors' 2^-24
takes the FP64 form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [1, 5])
@pytest.mark.parametrize("ratio", [1e-3, 1e-8])
@pytest.mark.parametrize("flow", ["stream", "shear", "tilted stream"])
def test_rates_of_unlike_components(native_lib, flow, ratio, nx):
    import lulesh_gb300 as lg
    d = lg.Domain(nx, numReg=3, its=10 ** 9, precision="fp64-fma")
    n = nx + 1
    x, y = d.field("x"), d.field("y")
    if flow == "tilted stream":  # planes of constant y stay, the others lean
        x = x + 2.0 ** -31 * y
        d.set_field("x", x)
    yd = -ratio * y
    d.set_field("xd", y.copy() if flow == "shear" else np.full_like(x, 3.0))
    d.set_field("yd", yd)
    d.set_field("zd", np.zeros_like(x))
    d.set_scalar("deltatime", 1e-4)
    assert d.phase(2) == 0
    L = np.longdouble
    Y, V = (a.reshape(n, n, n)[:-1, :, :-1].astype(L) for a in (y, yd))
    dy, dv = Y[:, 1:] - Y[:, :-1], V[:, 1:] - V[:, :-1]
    for f, want in (("vdov", dv / (dy - L(0.5e-4) * dv)), ("delv_eta", dv / dy)):
        got = np.abs(d.field(f)).reshape(nx, nx, nx)
        # about 16 roundings of 2^-53
        assert np.max(np.abs(got - np.abs(want)) / np.abs(want)) <= 16 * 2.0 ** -53, f
