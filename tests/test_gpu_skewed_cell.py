"""Pass 1 of a particle whose pairs fall to one lane of its warp: 600 particles on
one spot, every 32nd row of their cell, the rows between them out of their reach.
The weights of more than 512 pairs of weight near 1 exceed 32 bits in the
2^-23 fixed point."""
import numpy as np
import pytest

from helpers import FORCE_TOL, mdpd_params
from implicit_dpd_gb300.engine import Engine

pytestmark = pytest.mark.gpu


def test_density_of_pairs_on_one_lane():
    box = np.full(3, 5.99)  # five cells of 1.198 per side
    side = box[0] / 5
    rng = np.random.default_rng(12)
    spots = 0.02 + 1.16 * np.array([[0, 0, 0], [1, 1, 0], [0, 1, 1], [1, 0, 1.0]])
    n = 600 * 32
    r = np.arange(n)
    spot = np.where(r % 32 == 0, 0, 1 + (r // 32 + r) % 3)
    pos = 2 * side + spots[spot] + rng.random((n, 3)) * np.where(spot == 0, 1e-3, 1e-2)[:, None]
    assert np.all((pos / side).astype(int) == 2)
    none = np.full(n, 0xFFFFFFFF, np.uint32)
    st = {"pos": pos, "vel": np.zeros((n, 3)), "acc": np.zeros((n, 3)),
          "id": np.arange(n, dtype=np.uint32), "prop": (r % 3).astype(np.uint32),
          "amp_id": none, "unit": none.copy()}
    st["prop"][spot == 0] = 1
    e = Engine()
    e.set_params(mdpd_params(box, time=5))
    e.upload(st)
    e.set_tuning(1, 0.0)
    e.density()
    got = e.download_aux()["dens"]
    e.close()
    rows = np.concatenate([np.flatnonzero(spot == 0), rng.integers(0, n, 300)])
    for i in rows:
        d = np.linalg.norm(pos - pos[i], axis=1)
        w = np.where((d < 1.0) & (d > 0.0), (1.0 - d) ** 2, 0.0)
        want = np.bincount(st["prop"], w, 3)
        assert np.abs(got[i] - want).max() < FORCE_TOL * want.max(), (i, got[i], want)
