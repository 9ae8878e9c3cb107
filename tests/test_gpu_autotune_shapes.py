"""lg_ensemble_autotune leaves the kernels alone whose launches take no block size and no
grid (forces and kinematics of small strict ensembles): their entries stay the defaults
instead of the winner among equal candidates."""
import pytest

pytestmark = pytest.mark.gpu


def test_kernels_of_one_shape_are_not_tuned(native_lib):
    import lulesh_gb300 as lg
    opts = dict(numReg=5, balance=1, cost=1, its=10 ** 9)
    for _ in range(4):
        e = lg.Ensemble([dict(nx=9, **opts), dict(nx=6, **opts)])
        choice = e.autotune(1)
        for k in ("k_forces", "k_kinematics"):
            assert choice[k] == {"block": 128, "persistent": True}, (k, choice)
        e.close()
