"""The cells that the centre-of-mass pass visits around a particle
(csrc/cell_reach.hpp) are cells of its stencil for every coordinate."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_cells_within_reach_stay_in_the_stencil(tmp_path):
    exe = tmp_path / "cell_reach_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "implicit_dpd_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "cell_reach_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("reach", [1, 2])
def test_density_over_a_row_outside_the_box_ends_in_an_error(reach):
    """idpd_density after rows that idpd_set_dynamics refuses: the error, and the
    right result with the next rows."""
    from helpers import mdpd_params, mixed_system
    from implicit_dpd_gb300.engine import Engine, EngineError

    box, st, n_amp = mixed_system(seed=33)
    rows = [np.ascontiguousarray(st[k], np.float64) for k in ("pos", "vel", "acc")]
    e = Engine()
    e.set_params(mdpd_params(box, time=5))
    e.upload(st)
    e.build_topology(n_amp, [0])
    e.set_tuning(reach, 0.0)
    e.density()
    want = e.download_aux(nei_cm=True)
    for k, v in enumerate([-1e30, 1e30, 1e14, -7e9, 50.0, np.nan, np.inf]):
        bad = rows[0].copy()
        bad[13 + 60 * k, k % 3] = v
        e.set_dynamics(bad, rows[1], rows[2])
        with pytest.raises(EngineError):
            e.density()
    e.set_dynamics(*rows)
    e.density()
    got = e.download_aux(nei_cm=True)
    for k in want:
        assert np.array_equal(got[k], want[k], equal_nan=True), k
    e.close()
