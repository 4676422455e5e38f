"""Densities of particles so close that their FP32 coordinates coincide while
their FP64 positions differ: the weight of such a pair is near 1. Coincident
FP64 positions contribute nothing (nbdf_calculator.hpp:29-31)."""
import numpy as np
import pytest

from helpers import FORCE_TOL, mdpd_params, warren_params
from implicit_dpd_gb300 import configs
from implicit_dpd_gb300.abi import WALK_DENSITY
from implicit_dpd_gb300.engine import WALK_DTYPES, Engine

pytestmark = pytest.mark.gpu

BOX = np.array([6.0, 6.5, 7.0])


def _system():
    rng = np.random.default_rng(8)
    st = configs.liquid(BOX, 3.0, seed=8)
    n = len(st["pos"])
    st["prop"] = rng.integers(0, 3, n).astype(np.uint32)
    for k, gap in enumerate([1e-6, 1e-7, 1e-8, 1e-9, 1e-11, 1e-13, 0.0]):
        for q in range(10):
            a, b = 20 * (10 * k + q) % n, (20 * (10 * k + q) + 1) % n
            st["pos"][b] = st["pos"][a] + gap * np.eye(3)[q % 3]
    return np.mod(st["pos"], BOX), st


def _want(pos, st, rd):
    out = np.zeros((len(pos), 3))
    norm = 15.0 / (2.0 * np.pi * rd ** 3) if rd else 1.0
    for i in range(len(pos)):
        d = pos - pos[i]
        d -= BOX * np.round(d / BOX)
        r = np.sqrt((d ** 2).sum(1))
        cut = rd or 1.0
        w = np.where((r < cut) & (r > 0.0), norm * (1.0 - r / cut) ** 2, 0.0)
        out[i] = np.bincount(st["prop"], w, 3)
    return out


@pytest.mark.parametrize("form", ["mdpd", "warren"])
@pytest.mark.parametrize("reach", [1, 2])
def test_density_of_nearly_coincident_particles(form, reach):
    pos, st = _system()
    st["pos"] = pos
    p = mdpd_params(BOX, time=5) if form == "mdpd" else warren_params(BOX)
    want = _want(pos, st, 0.0 if form == "mdpd" else p.warren_rd)
    e = Engine()
    e.set_params(p)
    e.upload(st)
    e.set_tuning(reach, 0.0)
    e.density()
    got = e.download_aux()["dens"]
    assert np.abs(got - want).max() < FORCE_TOL * want.max()
    # the same as one walk of all particles and their images around the box
    e.set_tuning(1, 0.0)
    shift = np.stack(np.meshgrid(*[[-1, 0, 1]] * 3), -1).reshape(-1, 3) * BOX
    img = (pos[None] + shift[:, None]).reshape(-1, 3)
    keep = np.all((img > -1.0) & (img < BOX + 1.0), axis=1)
    epi = np.zeros(len(pos), WALK_DTYPES[WALK_DENSITY][0])
    epi["prop"], epi["pos"] = st["prop"], pos
    epj = np.zeros(int(keep.sum()), WALK_DTYPES[WALK_DENSITY][1])
    epj["prop"], epj["pos"] = np.tile(st["prop"], len(shift))[keep], img[keep]
    e.dispatch_walks(WALK_DENSITY, [epi], [epj])
    got = e.retrieve_walks(WALK_DENSITY)[0]["dens"]
    assert np.abs(got - want).max() < FORCE_TOL * want.max()
    e.close()
