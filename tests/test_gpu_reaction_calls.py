"""Steps with the reaction, one call each or many to a call, with observations
switched on between calls (the step counters are not read before): the same
state and the same records, in the loop graph and in plain graphs."""
import numpy as np
import pytest

import pyoracle as O
from implicit_dpd_gb300 import configs
from implicit_dpd_gb300.abi import CFG_PLAIN_GRAPHS, IdpdChemParams
from implicit_dpd_gb300.engine import Engine

pytestmark = pytest.mark.gpu


def _run(flags, chunks, more):
    box = np.array([10.0, 10.0, 10.0])
    n_amp = 600
    st = configs.flat_bilayers(box, n_amp, seed=5, jitter=0.05)
    core = [0, 1, 7]
    core_ptcl = [int(st["id"][(st["amp_id"] == a) & (st["unit"] == 0)][0]) for a in core]
    p = O.derive_params(configs.run_param(box, cf_b_rigid=20.0))
    p.seed, p.time = 1, 5
    cp = IdpdChemParams(p_thresld=0.05, eps=0.2, influ_rad=2.0, influ_hei=0.8, influ_dep=4.0,
                        influ_grd=-0.5, amp_num=n_amp, max_amp_num=100000)
    e = Engine(flags=flags, sort_period=4)
    e.set_params(p)
    e.upload(st)
    e.build_topology(n_amp, core)
    e.set_chem(cp, 1234, core_ptcl, 6000, beg_chem=10)
    for k in chunks:
        e.step(k)
    e.set_observe(3)
    for k in more:
        e.step(k)
    out, obs, t = e.download(), e.observations(), e.get_params().time
    e.set_observe(0)
    e.step(2)
    last = e.download()
    e.close()
    return out, obs, t, last


def test_reaction_steps_by_call_and_with_observations():
    want = _run(0, [9], [10])
    assert want[2] == 5 + 19 and [o["time"] for o in want[1]] == [15, 18, 21]
    assert len(want[0]["pos"]) > 2400
    for flags, chunks, more in ((0, [1] * 9, [1] * 10), (0, [2, 7], [4, 1, 5]),
                                (CFG_PLAIN_GRAPHS, [9], [10]),
                                (CFG_PLAIN_GRAPHS, [1] * 9, [3, 7])):
        got = _run(flags, chunks, more)
        assert got[2] == want[2]
        for a, b in ((got[0], want[0]), (got[3], want[3])):
            for k in ("pos", "vel", "acc", "id", "prop", "amp_id", "unit"):
                assert np.array_equal(a[k], b[k]), k
        assert len(got[1]) == len(want[1])
        for x, y in zip(got[1], want[1]):
            for k in x:
                assert np.array_equal(np.asarray(x[k]), np.asarray(y[k])), k
