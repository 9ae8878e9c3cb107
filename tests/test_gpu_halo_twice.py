"""lg_halo_unpack with one array given for several fields: each field's messages are
applied in the order of the fields, all of them added (sbn) or the last one kept."""
import numpy as np
import pytest

from halolib import field_length

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,order", [("sbn", "aba"), ("sbn", "aa"), ("sbn", "abcd"),
                                        ("sync_pos_vel", "abbaab"), ("monoq", "aab")])
@pytest.mark.parametrize("nx,rank", [(1, 0), (6, 13)])
def test_one_array_for_several_fields(native_lib, kind, order, nx, rank):
    import torch
    import lulesh_gb300 as lg
    p = lg.HaloPlan(kind, nx, 3, rank, len(order))
    rng = np.random.default_rng(nx)
    host = {c: rng.standard_normal(field_length(kind, nx)) for c in sorted(set(order))}
    buf = rng.standard_normal(p.info()["buffer_doubles"])
    dev = {c: torch.from_numpy(a).cuda() for c, a in host.items()}
    p.unpack([dev[c] for c in order], torch.from_numpy(buf).cuda())
    torch.cuda.synchronize()
    e = p.entries("recv")
    want = {c: a.copy() for c, a in host.items()}
    for f, c in enumerate(order):
        for i, b, s in zip(e["index"], e["bufpos"], e["stride"]):
            v = buf[b + f * s]
            want[c][i] = want[c][i] + v if kind == "sbn" else v
    for c in want:
        assert np.array_equal(dev[c].cpu().numpy().view(np.int64), want[c].view(np.int64)), c
    p.close()
