"""Parameters set between idpd_step_host calls (time step, coefficients, pair
form, step counter) hold from the next call on, as for the three calls that it
stands for."""
import numpy as np
import pytest

from helpers import mdpd_params, mixed_system, pairwise_params, warren_params
from implicit_dpd_gb300.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skin", [0.0, 0.2])
def test_parameters_changed_between_host_steps(skin):
    box, st, n_amp = mixed_system(seed=52)
    sets = [mdpd_params(box, time=5), mdpd_params(box, time=6, dt=0.002), warren_params(box, time=7),
            pairwise_params(box, time=8), mdpd_params(box, time=150, seed=9)]
    a, b = Engine(), Engine()
    rows = [[np.array(st[k], np.float64) for k in ("pos", "vel", "acc")] for _ in range(2)]
    for e in (a, b):
        e.set_params(sets[0])
        e.upload(st)
        e.build_topology(n_amp, [0, 3])
        e.set_tuning(1, skin)
    for p in sets:
        for e in (a, b):
            e.set_params(p)
        for _ in range(2):
            a.set_dynamics(*rows[0])
            a.step(1)
            a.download_dynamics(*rows[0])
            b.step_host(*rows[1])
            for x, y, name in zip(*rows, ("pos", "vel", "acc")):
                assert np.array_equal(x, y), (name, p.form, p.time)
        assert a.get_params().time == b.get_params().time == p.time + 2
    a.close()
    b.close()
