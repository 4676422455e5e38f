"""The walks' records are read from the caller's memory by the device where they are
aligned, and copied by the host where they are not: the same results bit for bit, with
empty walks, one record and more than a CTA's threads hold, and with the records
overwritten as soon as the dispatch returns."""
import numpy as np
import pytest

from helpers import mdpd_params
from implicit_dpd_gb300.engine import WALK_DTYPES, Engine

pytestmark = pytest.mark.gpu

BOX = np.array([6.0, 6.0, 6.0])
SIZES = [(1, 1), (0, 5), (3, 0), (17, 40), (260, 300), (2, 33)]


def _records(kind, offset):
    rng = np.random.default_rng(5)
    out = ([], [])
    for ni, nj in SIZES:
        pos = rng.random((ni + nj, 3)) * 2.0
        for side, (dt, p) in enumerate(zip(WALK_DTYPES[kind][:2], (pos[:ni], pos[ni:]))):
            n = len(p)
            buf = np.zeros(n * dt.itemsize + 16, np.uint8)
            a = np.frombuffer(buf.data, dt, n, offset=offset)
            a["prop"], a["pos"] = rng.integers(0, 3, n), p
            if kind:
                a["id"] = rng.permutation(1000)[:n] + 1000 * side
                a["vel"], a["dens"] = rng.normal(size=(n, 3)), rng.random((n, 3))
            out[side].append(a)
    return out


@pytest.mark.parametrize("kind", [0, 1])
def test_aligned_and_unaligned_records(kind):
    got = []
    for offset in (0, 8, 4):  # 4: unaligned
        e = Engine()
        e.set_params(mdpd_params(BOX, time=3))
        epi, epj = _records(kind, offset)
        e.dispatch_walks(kind, epi, epj)
        for a in epi + epj:
            a[...] = 0
        got.append(np.concatenate(e.retrieve_walks(kind)))
        e.close()
    assert len(got[0]) == sum(ni for ni, _ in SIZES)
    for g in got[1:]:
        for name in g.dtype.names:
            assert np.array_equal(g[name], got[0][name], equal_nan=True), name
