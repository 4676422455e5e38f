"""The list builds test a cell's particles in pairs, up to 32 at a time, against 32
candidates: exact pair counts for cells of one to 100 particles (odd counts, batches that
just fit or just do not), with equal x coordinates (the ownership of such a pair goes by
row), against a count over all pairs."""
import numpy as np
import pytest

from helpers import warren_params
from implicit_dpd_gb300 import configs
from implicit_dpd_gb300.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skin", [0.0, 0.2])
@pytest.mark.parametrize("m", [1, 2, 3, 31, 32, 33, 64, 65, 100])
def test_cells_of_any_number_of_particles(m, skin):
    box = np.array([6.0, 7.0, 8.0])
    rng = np.random.default_rng(m)
    crowd = 3.7 + 0.5 * rng.random((m, 3))
    crowd[:, 0] = rng.choice([3.75, 3.9, 4.1], m)  # ties
    rest = rng.random((150, 3)) * box
    rest[:40, 0] = 3.9
    pos = np.concatenate([crowd, rest])
    n = len(pos)
    st = configs.liquid(box, n / box.prod(), seed=m)
    st["pos"], st["vel"] = pos, np.zeros((n, 3))
    dx = pos[:, None] - pos[None]
    r2 = ((dx - box * np.rint(dx / box)) ** 2).sum(axis=2)
    r2 = r2[np.triu_indices(n, 1)]
    assert np.abs(r2 - 1.0).min() > 1e-9  # none that a step of 1e-7 could move across
    p = warren_params(box)
    p.dt = 1.0e-7
    e = Engine()
    e.set_params(p)
    e.upload(st)
    e.set_tuning(1, skin)
    e.step(1)
    got = e.pair_count()
    e.close()
    assert got == 2 * int((r2 < 1.0).sum())
