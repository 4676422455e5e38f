"""idpd_step's runs of steps are captured as calls come to need them: whatever the
lengths of the calls and their order, the state is that of one launch per step."""
import numpy as np
import pytest

from helpers import mdpd_params, mixed_system
from implicit_dpd_gb300.abi import CFG_PLAIN_GRAPHS
from implicit_dpd_gb300.engine import Engine

pytestmark = pytest.mark.gpu

CALLS = [[2, 2, 2], [3, 3], [4, 4, 4], [8, 8, 8], [9, 4, 9, 4], [16], [22, 22], [1, 40, 2, 15],
         [130]]


def _run(flags, skin, calls):
    box, st, n_amp = mixed_system(seed=91, box=(7.0, 8.0, 7.5), n_amp=200)
    e = Engine(flags=flags, sort_period=31)
    e.set_params(mdpd_params(box, time=63))
    e.upload(st)
    e.build_topology(n_amp, [0, 3])
    e.set_tuning(1, skin)
    out = []
    for k in calls:
        e.step(k)
        out.append(e.download())
        assert e.last_step_ms() > 0.0
    t = e.get_params().time
    e.set_tuning(1, skin, lanes=8)  # the runs are captured anew
    e.step(6)
    out.append(e.download())
    e.close()
    return out, t


@pytest.mark.parametrize("calls", CALLS, ids=str)
@pytest.mark.parametrize("skin", [0.0, 0.2])
def test_calls_of_any_length_equal_single_steps(skin, calls):
    a, ta = _run(0, skin, calls)
    b, tb = _run(CFG_PLAIN_GRAPHS, skin, calls)
    assert ta == tb == 63 + sum(calls)
    for x, y in zip(a, b):
        for k in ("pos", "vel", "acc"):
            assert np.array_equal(x[k], y[k]), k
