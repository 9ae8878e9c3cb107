"""The energy floor emin in the FMA and mixed builds, whose EOS repetitions run on the
integer pipes without it: elements whose energy falls below it, and the ordinary ones
beside them, against the strict build on the same state."""
import numpy as np
import pytest

from paritylib import field_rel_err

pytestmark = pytest.mark.gpu


def _material(lg, precision, nx):
    d = lg.Domain(nx, numReg=3, its=10 ** 9, precision=precision)
    E = nx ** 3
    far = np.arange(E) % 3 == 0
    # resting elements of relative volume 64 that came from 121 or from 33 (the change
    # is -57 or 31), or from 60
    d.set_field("volo", d.field("volo") / 64.0)
    d.set_field("v", np.where(far, np.where(np.arange(E) % 2, 121.0, 33.0), 60.0))
    d.set_field("p", np.where(far, 1.4e14, 1.0e4))
    for f in ("xd", "yd", "zd", "e", "q"):
        d.set_field(f, np.zeros_like(d.field(f)))
    d.set_scalar("deltatime", 1e-9)
    status = d.phase(2)
    return status, {f: d.field(f) for f in ("e", "p", "q", "ss", "v")}


@pytest.mark.parametrize("nx", [1, 5])
@pytest.mark.parametrize("precision", ["fp64-fma", "mixed"])
def test_energy_floor_matches_strict(native_lib, precision, nx):
    import lulesh_gb300 as lg
    st0, a = _material(lg, "fp64", nx)
    st1, b = _material(lg, precision, nx)
    assert st0 == st1 == 0
    assert a["e"].max() > 1e14  # the clamped energy, not the one below the floor
    for f in a:
        # about a hundred operations of 2^-53 in a row, on terms at most 100 times the
        # result: 1e-12
        assert field_rel_err(b[f], a[f], floor=1e-3) <= 1e-12, f
