"""Boxes and tunings whose search cells exceed the 32-bit cell numbers are refused,
and a refused tuning leaves the handle as it was."""
import numpy as np
import pytest

from helpers import mdpd_params
from implicit_dpd_gb300.abi import SOLVENT
from implicit_dpd_gb300.engine import Engine, EngineError

pytestmark = pytest.mark.gpu


def _rows(box, n=200):
    rng = np.random.default_rng(4)
    none = np.full(n, 0xFFFFFFFF, np.uint32)
    # neighbours at the origin's corner, some across the box's edges
    return {"pos": np.mod(rng.normal(size=(n, 3)), box), "vel": rng.normal(size=(n, 3)),
            "acc": np.zeros((n, 3)), "id": np.arange(n, dtype=np.uint32),
            "prop": np.full(n, SOLVENT, np.uint32), "amp_id": none, "unit": none.copy()}


@pytest.mark.parametrize("side", [1291.0, 1626.0, 2000.0, 4000.0, 1e7, 3e38])
def test_a_box_of_too_many_cells_is_refused(side):
    """Also where the product of the cells wraps to a small or negative number."""
    box = np.full(3, side)
    e = Engine()
    e.set_params(mdpd_params(box))
    e.upload(_rows(np.full(3, 9.0)))
    with pytest.raises(EngineError, match="too many cells"):
        e.step(1)
    with pytest.raises(EngineError, match="too many cells"):
        e.density()
    e.set_params(mdpd_params(np.full(3, 9.0)))
    e.upload(_rows(np.full(3, 9.0)))
    e.step(2)
    e.close()


def test_a_refused_tuning_changes_nothing():
    box = np.array([2600.0, 2600.0, 60.0])  # 4.1e8 cells, 3.2e9 at reach 2
    out = []
    for refused in (False, True):
        e = Engine()
        e.set_params(mdpd_params(box))
        e.upload(_rows(box))
        e.step(2)
        if refused:
            with pytest.raises(EngineError, match="too many cells"):
                e.set_tuning(2, 0.0, lanes=8)
            assert e.tuning()["reach"] == 1 and e.tuning()["lanes"] == 16
        e.step(3)
        out.append(e.download())
        e.close()
    for k in ("pos", "vel", "acc"):
        assert np.array_equal(out[0][k], out[1][k]), k
