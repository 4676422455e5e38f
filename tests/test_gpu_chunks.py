"""Rows per warp of the pair passes: the launches halve a warp's 32-row chunk
while the handle is small, so the same system runs in chunks of another size
inside a larger batch. Its results must be those of the handle alone, bit for
bit, whatever the chunk, its remainder and the lanes per particle."""
import numpy as np
import pytest

from helpers import FORCE_TOL, mdpd_params, mixed_system, oracle_forces, rel_force_err, warren_params
from implicit_dpd_gb300 import configs
from implicit_dpd_gb300.engine import Engine

pytestmark = pytest.mark.gpu


def _run(systems, lanes, dens_lanes, skin):
    e = Engine(n_replicas=len(systems))
    for r, (p, st, n_amp) in enumerate(systems):
        e.set_params(p, r)
        e.upload(st, r)
        if n_amp:
            e.build_topology(n_amp, replica=r)
    e.set_tuning(1, skin, lanes=lanes, dens_lanes=dens_lanes)
    e.step(4)
    out = e.download()
    pairs = e.pair_count()
    e.close()
    return out, pairs


def _at_rest(side):
    """A filler that never moves (a lattice of spacing 1.1 at rest, no pair
    within the cutoff): the rebuild decision of a handle is taken over all its
    replicas, so a moving one would change the rebuilds of the other."""
    box = np.array([1.1 * side] * 3)
    k = np.arange(side ** 3)
    st = configs.liquid(box, len(k) / box.prod(), seed=side)
    st["pos"] = np.stack([k % side, k // side % side, k // side ** 2], axis=1) * 1.1 + 0.5
    st["vel"][:] = 0.0
    return st, box


@pytest.mark.parametrize("skin", [0.0, 0.2])
@pytest.mark.parametrize("lanes", [4, 8, 16, 32])
def test_chunk_rows_do_not_change_results(lanes, skin):
    box, st, n_amp = mixed_system(seed=41)
    p = mdpd_params(box, time=5)
    alone, pairs = _run([(p, st, n_amp)], lanes, lanes, skin)
    for side in (31, 48, 63, 79, 100):  # fillers of 30k to 1M rows: 2 to 32 rows per warp
        fill, fbox = _at_rest(side)
        got, gp = _run([(p, st, n_amp), (warren_params(fbox), fill, 0)], lanes, lanes, skin)
        n = len(fill["pos"])
        assert gp == pairs, n
        for k in ("pos", "vel", "acc"):
            assert np.array_equal(got[k], alone[k]), (n, k)


@pytest.mark.parametrize("n", [31, 33, 127, 129, 700])
def test_small_systems_against_the_oracle(n):
    # remainders of quads, groups, chunks and row blocks
    box = np.array([5.0, 5.5, 6.0])
    st = configs.liquid(box, n / box.prod(), seed=n)
    assert len(st["pos"]) == n
    p = warren_params(box, time=3)
    acc = oracle_forces(p, st)[3]
    for lanes in (4, 8, 16, 32):
        e = Engine()
        e.set_params(p)
        e.upload(st)
        e.set_tuning(1, 0.0, lanes=lanes)
        e.density()
        e.force()
        assert rel_force_err(e.download()["acc"], acc)[0] < FORCE_TOL, lanes
        e.close()
