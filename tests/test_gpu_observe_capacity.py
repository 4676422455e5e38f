"""idpd_set_observe with a capacity that cannot be allocated ends in an error and
leaves the observation as it was."""
import numpy as np
import pytest

from helpers import mdpd_params, mixed_system
from implicit_dpd_gb300.engine import Engine, EngineError

pytestmark = pytest.mark.gpu


def test_observation_goes_on_after_a_refused_capacity():
    got = []
    for refused in (False, True):
        box, st, n_amp = mixed_system(seed=61)
        e = Engine()
        e.set_params(mdpd_params(box, time=4))
        e.upload(st)
        e.build_topology(n_amp, [0])
        e.set_observe(2, 64)
        e.step(5)
        if refused:
            with pytest.raises(EngineError):
                e.set_observe(3, 2 ** 31 - 1)  # more than the device's memory
        e.step(5)
        obs = e.observations()
        e.set_observe(2, 16)
        e.step(4)
        got.append((obs, e.observations(), e.download()))
        e.close()
    for a, b in zip(got[0][:2], got[1][:2]):
        assert [o["time"] for o in a] == [o["time"] for o in b] and len(a) > 0
        for x, y in zip(a, b):
            for k in x:
                assert np.array_equal(np.asarray(x[k]), np.asarray(y[k])), k
    for k in ("pos", "vel", "acc"):
        assert np.array_equal(got[0][2][k], got[1][2][k]), k
