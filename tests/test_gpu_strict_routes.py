"""The strict build's three forms of forces and kinematics -- eight lanes for each element,
three warps for 32, one thread -- on both sides of the sizes where a Domain changes from
one to the next, against one thread for each element (an ensemble too large for the other
two): the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["x", "y", "z", "xd", "yd", "zd", "fx", "fy", "fz", "e", "p", "q", "v", "ss", "vnew",
          "delv", "vdov", "arealg"]


def _root(elements):
    nx = round(elements ** (1 / 3)) + 1
    while nx ** 3 > elements:
        nx -= 1
    return nx


@pytest.mark.parametrize("hgcoef", [2.7, 0.0])
@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("elements", [32, 192])  # for each SM: the last of lanes, of warps
def test_forms_agree_where_the_choice_changes(native_lib, elements, side, hgcoef):
    import torch
    import lulesh_gb300 as lg
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nx, fill = _root(elements * sms) + side, _root(192 * sms) + 3
    opts = dict(numReg=7, balance=1, cost=1, its=10 ** 9)
    d = lg.Domain(nx, 7, 1, 1, its=10 ** 9, hgcoef=hgcoef, einit_factor=1.3)
    e = lg.Ensemble([dict(nx=nx, hgcoef=hgcoef, einit_factor=1.3, **opts), dict(nx=fill, **opts)])
    assert d.step(25) == e.step(25) == 0
    for f in FIELDS:
        a, b = d.field(f), e.field(0, f)
        assert np.array_equal(a.view(np.int64), b.view(np.int64)), f
