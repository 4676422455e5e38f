"""Walks of many records go to the device in pieces of 2,048 words: sizes around a
piece and its multiples give the results of the host's copy (unaligned records)
bit for bit."""
import numpy as np
import pytest

from helpers import mdpd_params
from implicit_dpd_gb300.engine import WALK_DTYPES, Engine

pytestmark = pytest.mark.gpu

PIECE = 2048 * 8


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("pieces", [1, 3])
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_pieces_of_a_walk(kind, pieces, extra):
    got = []
    for offset in (0, 4):
        rng = np.random.default_rng(5)
        epi, epj = [], []
        sizes = [(7, 0), (0, 0), (pieces * PIECE // WALK_DTYPES[kind][0].itemsize + extra,
                                  pieces * PIECE // WALK_DTYPES[kind][1].itemsize + extra), (3, 20)]
        for counts in sizes:
            for side, n in enumerate(counts):
                dt = WALK_DTYPES[kind][side]
                a = np.frombuffer(np.zeros(n * dt.itemsize + 16, np.uint8).data, dt, n, offset=offset)
                a["prop"], a["pos"] = rng.integers(0, 3, n), rng.random((n, 3)) * 8.0
                if kind:
                    a["id"] = rng.permutation(100000)[:n] + 100000 * side
                    a["vel"], a["dens"] = rng.normal(size=(n, 3)), rng.random((n, 3))
                (epj if side else epi).append(a)
        e = Engine()
        e.set_params(mdpd_params(np.array([8.0, 8.0, 8.0]), time=3))
        e.dispatch_walks(kind, epi, epj)
        for a in epi + epj:
            a[...] = 0
        got.append(np.concatenate(e.retrieve_walks(kind)))
        e.close()
    assert len(got[0]) == sum(ni for ni, _ in sizes)
    for name in got[0].dtype.names:
        assert np.array_equal(got[1][name], got[0][name], equal_nan=True), name
