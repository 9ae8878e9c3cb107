"""The strict build's kernels with eight lanes for each element (meshes too small
to fill the SMs) against the batched kernels, one thread for each element: the
same bits, at element counts that leave a warp's last lanes without one, on both
sides of the size where the choice changes, and with and without hourglass
forces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["x", "y", "z", "xd", "yd", "zd", "fx", "fy", "fz", "e", "p", "q", "v", "ss", "vnew",
          "delv", "vdov", "arealg"]


@pytest.mark.parametrize("nx", [1, 3, 5, 10, 19, 20])
@pytest.mark.parametrize("hgcoef", [2.7, 0.0])
def test_lanes_equal_batched_kernels(native_lib, nx, hgcoef):
    import lulesh_gb300 as lg
    opts = dict(nx=nx, numReg=7, balance=1, cost=1, its=10 ** 9, hgcoef=hgcoef, einit_factor=1.3)
    d = lg.Domain(nx, 7, 1, 1, its=10 ** 9, hgcoef=hgcoef, einit_factor=1.3)
    e = lg.Ensemble([opts])
    assert d.step(25) == e.step(25) == 0
    for f in FIELDS:
        a, b = d.field(f), e.field(0, f)
        assert np.array_equal(a.view(np.int64), b.view(np.int64)), f
