"""The fine-grained passes in every accepted order: idpd_bonded between pass 1
and pass 2, or between two calls of pass 2, leaves the pair forces what they
are without it, also of particles whose pass-1 lists overflowed."""
import numpy as np
import pytest

from helpers import FORCE_TOL, mdpd_params, mixed_system, oracle_forces, rel_force_err
from implicit_dpd_gb300 import configs
from implicit_dpd_gb300.engine import Engine

pytestmark = pytest.mark.gpu

ORDERS = [("density", "bonded", "force"), ("density", "force", "bonded", "force"),
          ("density", "bonded", "bonded", "force", "bonded", "force")]


def _pair_passes(p, st, n_amp, reach, skin, calls):
    e = Engine()
    e.set_params(p)
    e.upload(st)
    if n_amp:
        e.build_topology(n_amp, [0])
    e.set_tuning(reach, skin)
    for c in calls:
        getattr(e, c)()
    got = e.download()["acc"], e.download_aux(press=True)["press"]
    e.close()
    return got


@pytest.mark.parametrize("reach,skin", [(1, 0.0), (2, 0.0), (1, 0.2)])
@pytest.mark.parametrize("dense", [False, True])
def test_bonded_between_the_pair_passes_leaves_their_forces(reach, skin, dense):
    if dense:  # rho 400: every pass-1 list (512 entries) overflows
        box = np.full(3, 6.1 if skin else 5.0)  # idpd_density wants 5 cells of 1 + skin
        st, n_amp = configs.liquid(box, 400.0, seed=40, prop=1), 0
        p = mdpd_params(box, time=5)
    else:
        box, st, n_amp = mixed_system(seed=44)
        p = mdpd_params(box, time=5)
    want = _pair_passes(p, st, n_amp, reach, skin, ("density", "force"))
    acc = oracle_forces(p, st)[3]
    assert rel_force_err(want[0], acc)[0] < FORCE_TOL
    for calls in ORDERS:
        got = _pair_passes(p, st, n_amp, reach, skin, calls)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), calls
