"""The FMA build's time limits are the quotients of its fields, rounded once: the hydro
limit dvovmax / |vdov| and the Courant limit arealg / sqrt(...) of every cycle of a run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [6, 13])
def test_time_limits_are_quotients(native_lib, nx):
    import lulesh_gb300 as lg
    d = lg.Domain(nx, numReg=3, its=10 ** 9, precision="fp64-fma")
    L = np.longdouble
    hydro, courant = [], []
    for _ in range(60):
        assert d.step(1) == 0
        vdov, ss, length = (d.field(f) for f in ("vdov", "ss", "arealg"))
        m = vdov != 0
        if not m.any():  # the first cycles' velocities may be below the cut-off
            continue
        rate = (np.abs(vdov[m]) + 1e-20).astype(L)  # 1e-20 changes no such rate
        want = np.min(L(0.1) / rate)
        hydro.append(abs(L(d.scalar("dthydro")) - want) / want)
        v, s, a = vdov[m].astype(L), ss[m].astype(L), length[m].astype(L)
        want = np.min(a / np.sqrt(s * s + np.where(v < 0, 256 * a * a * v * v, 0)))
        courant.append(abs(L(d.scalar("dtcourant")) - want) / want)
    assert len(hydro) > 40
    # one rounding; the corrected quotient's own error is below 2^-59
    assert max(hydro) <= 1.02 * 2.0 ** -53
    # four or five operations under the root (half of their roundings counts), the root
    # and the product
    assert max(courant) <= 5 * 2.0 ** -53
