"""The walk buffers of a handle outlive a change of its observation capacity: a
dispatch in flight keeps its results, later ones work, and the handle closes."""
import numpy as np
import pytest

from helpers import mdpd_params
from implicit_dpd_gb300.abi import WALK_DENSITY, WALK_FORCE
from implicit_dpd_gb300.engine import WALK_DTYPES, Engine

pytestmark = pytest.mark.gpu

BOX = np.array([6.0, 6.0, 6.0])


def _records(kind, sizes):
    rng = np.random.default_rng(9)
    out = ([], [])
    for counts in sizes:
        for side, n in enumerate(counts):
            a = np.zeros(n, WALK_DTYPES[kind][side])
            a["prop"], a["pos"] = rng.integers(0, 3, n), rng.random((n, 3)) * 2.0
            if kind == WALK_FORCE:
                a["id"] = rng.permutation(1000)[:n] + 1000 * side
                a["vel"], a["dens"] = rng.normal(size=(n, 3)), rng.random((n, 3))
            out[side].append(a)
    return out


def _engine():
    e = Engine()
    e.set_params(mdpd_params(BOX, time=3))
    return e


def _same(a, b):
    return all(np.array_equal(x[k], y[k], equal_nan=True)
               for x, y in zip(a, b) for k in x.dtype.names)


@pytest.mark.parametrize("kind", [WALK_DENSITY, WALK_FORCE])
def test_walks_across_a_change_of_the_observation_capacity(kind):
    epi, epj = _records(kind, [(40, 90), (3, 0), (20, 33)])
    e = _engine()
    e.dispatch_walks(kind, epi, epj)
    want = e.retrieve_walks(kind)
    e.close()
    e = _engine()
    e.dispatch_walks(kind, epi, epj)
    e.set_observe(10, 64)
    assert _same(e.retrieve_walks(kind), want)
    for capacity in (128, 16):
        e.set_observe(5, capacity)
        e.dispatch_walks(kind, epi, epj)
        assert _same(e.retrieve_walks(kind), want)
    e.close()
