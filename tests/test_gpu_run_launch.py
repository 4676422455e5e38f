"""Steps without the reaction go out eight in one graph launch, the rest one by one; a
step that removes the centre-of-mass drift (every 100 steps of some replica) or observes
is a launch of its own graph, picked from the host's copy of the step counters. Bit for
bit the state, the counters and the records of one launch per step with every kernel in
it, for run lengths around eight, for replicas whose counters differ, across a counter
set in between and across a step on host arrays."""
import numpy as np
import pytest

from helpers import mdpd_params, mixed_system, warren_params
from implicit_dpd_gb300 import configs
from implicit_dpd_gb300.abi import CFG_PLAIN_GRAPHS, FORM_WARREN
from implicit_dpd_gb300.engine import Engine, derive_params

pytestmark = pytest.mark.gpu


def _run(flags, skin, times, period, chunks):
    e = Engine(n_replicas=len(times), flags=flags, sort_period=37)
    for r, t in enumerate(times):
        box, st, n_amp = mixed_system(seed=50 + r)
        # a common drift, so that a removal left out or done twice shows
        st["vel"] = st["vel"] + np.array([0.3, -0.2, 0.1])
        e.set_params(mdpd_params(box, time=t), r)
        e.upload(st, r)
        e.build_topology(n_amp, [0, 3], r)
    e.set_tuning(1, skin)
    if period:
        e.set_observe(period)
    for k in chunks:
        e.step(k)
    p = e.get_params(0)
    p.time = 95
    e.set_params(p, 0)
    e.step(11)
    out = [e.download(replica=r) for r in range(len(times))]
    t = [e.get_params(r).time for r in range(len(times))]
    obs = e.observations() if period and len(times) == 1 else []
    e.close()
    return out, t, obs


@pytest.mark.parametrize("skin", [0.0, 0.25])
@pytest.mark.parametrize("times,period", [((93,), 0), ((1,), 0), ((88, 195), 0), ((90,), 5)])
def test_runs_of_steps_equal_single_steps(skin, times, period):
    chunks = [7, 8, 9, 1, 2, 17, 70]
    a, ta, oa = _run(0, skin, times, period, chunks)
    b, tb, ob = _run(CFG_PLAIN_GRAPHS, skin, times, period, chunks)
    assert ta == tb == [106] + [t + sum(chunks) + 11 for t in times[1:]]
    for x, y in zip(a, b):
        for k in ("pos", "vel", "acc", "id", "prop"):
            assert np.array_equal(x[k], y[k]), k
    assert len(oa) == len(ob)
    for x, y in zip(oa, ob):
        for k in x:
            assert np.array_equal(np.asarray(x[k]), np.asarray(y[k])), k


@pytest.mark.parametrize("rho", [5.9, 6.0])
def test_rebuild_in_an_if_node_or_in_every_step(rho):
    # 396,716 rows, below the line where the rebuild's kernels go into an IF node, and
    # 403,440, above it; against one launch per step, which has no such node
    box = np.array([41.0, 41.0, 40.0])
    st = configs.liquid(box, rho, seed=71)
    q = derive_params(configs.run_param(box, dt=0.005, cf_r=3.0))
    q.seed, q.time, q.form = 5, 95, FORM_WARREN
    q.warren_a, q.warren_b, q.warren_rd = -40.0, 25.0, 0.75

    def run(flags):
        e = Engine(flags=flags)
        e.set_params(q)
        e.upload(st)
        e.set_tuning(1, 0.2)
        e.step(20)
        out, n = e.download(), e.list_rebuilds()
        e.close()
        return out, n

    (a, na), (b, nb) = run(0), run(CFG_PLAIN_GRAPHS)
    assert na == nb and 1 < na < 20  # steps with and without a rebuild
    for k in ("pos", "vel", "acc", "id"):
        assert np.array_equal(a[k], b[k]), k


def test_host_array_steps_remove_the_drift_when_due():
    box, st, n_amp = mixed_system(seed=61)
    st["vel"] = st["vel"] + np.array([0.3, -0.2, 0.1])

    def run(on_host):
        e = Engine()
        e.set_params(mdpd_params(box, time=98))
        e.upload(st)
        e.build_topology(n_amp, [0, 3])
        out = {k: np.array(st[k], np.float64) for k in ("pos", "vel", "acc")}
        for _ in range(4):
            if on_host:
                e.step_host(out["pos"], out["vel"], out["acc"])
            else:
                e.set_dynamics(out["pos"], out["vel"], out["acc"])
                e.step(1)
                out = e.download()
        t = e.get_params().time
        e.close()
        return out, t

    (a, ta), (b, tb) = run(True), run(False)
    assert ta == tb == 102
    for k in ("pos", "vel", "acc"):
        assert np.array_equal(a[k], b[k]), k


def test_a_change_of_the_pair_form_between_steps():
    # the captured steps hold one form's passes: after the change, as a fresh handle
    box, st, n_amp = mixed_system(seed=91)

    def engine(p, state):
        e = Engine()
        e.set_params(p)
        e.upload(state)
        e.build_topology(n_amp)
        return e

    e = engine(mdpd_params(box, time=3), st)
    e.step(5)
    mid = e.download()
    q = warren_params(box, time=8)
    e.set_params(q)
    e.step(5)
    a = e.download()
    e.close()
    e = engine(q, mid)
    e.step(5)
    b = e.download()
    e.close()
    for k in ("pos", "vel", "acc"):
        assert np.array_equal(a[k], b[k]), k
