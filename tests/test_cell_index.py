"""The cell of a coordinate (cell_index, csrc/fp64_int.cuh) is an index of the
grid for every double: coordinates outside the box take the nearest cell, NaN
cell 0, as the plain product truncated and clamped gives them."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_cell_index_stays_in_the_grid_for_every_double(tmp_path):
    exe = tmp_path / "cell_index_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "implicit_dpd_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "cell_index_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
def test_rows_outside_the_box_take_the_nearest_cell():
    """idpd_cell_order_noalloc on rows outside [0, box): the cells of the
    coordinates clamped to the grid, in ascending row order."""
    import ctypes as C
    from implicit_dpd_gb300.engine import load

    torch = pytest.importorskip("torch")
    box = np.array([5.0, 6.25, 7.9])
    nc = box.astype(int)
    rng = np.random.default_rng(5)
    n = 700
    pos = (rng.random((n, 3)) * 3.0 - 1.0) * box
    bad = [-1e30, -1e300, 1e30, np.inf, -np.inf, np.nan, -np.nan, -0.0, -2.0 ** 31, 2.0 ** 31]
    for k, v in enumerate(bad):
        pos[7 * k, k % 3] = v
    q = pos * (nc / box)
    cell = np.where(q > 0.0, np.minimum(q, nc - 1.0), 0.0).astype(np.int64)  # NaN: 0
    want = (cell[:, 2] * nc[1] + cell[:, 1]) * nc[0] + cell[:, 0]
    pos_d = torch.from_numpy(pos).cuda()
    cell_d = torch.empty(n, dtype=torch.int32, device="cuda")
    perm_d = torch.empty(n, dtype=torch.int32, device="cuda")
    rc = load().idpd_cell_order_noalloc(
        C.c_void_p(pos_d.data_ptr()), n, box, C.c_void_p(cell_d.data_ptr()),
        C.c_void_p(perm_d.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    assert np.array_equal(cell_d.cpu().numpy(), want)
    assert np.array_equal(perm_d.cpu().numpy(), np.argsort(want, kind="stable"))


@pytest.mark.gpu
@pytest.mark.parametrize("skin", [0.0, 0.2])
def test_step_over_a_row_outside_the_box_ends_in_an_error(skin):
    """A bad row in step_host is binned before the error word is read: the call
    ends in the error, and the next one with good rows is right."""
    from helpers import FORCE_TOL, mdpd_params, mixed_system, rel_force_err
    from implicit_dpd_gb300.engine import Engine, EngineError

    box, st, n_amp = mixed_system(seed=31)
    good = [np.ascontiguousarray(st[k], np.float64) for k in ("pos", "vel", "acc")]

    def engine(time):
        e = Engine()
        e.set_params(mdpd_params(box, time=time))
        e.upload(st)
        e.build_topology(n_amp, [0, 3])
        e.set_tuning(1, skin)
        return e

    a = engine(5)
    a.step_host(*[x.copy() for x in good])
    bad = [-1e30, 1e300, -0.7, np.nan, -np.inf]
    for k, v in enumerate(bad):
        rows = [x.copy() for x in good]
        rows[0][11 + 50 * k, k % 3] = v
        with pytest.raises(EngineError):
            a.step_host(*rows)
    got = [x.copy() for x in good]
    a.step_host(*got)
    b = engine(5 + 1 + len(bad))
    want = [x.copy() for x in good]
    b.step_host(*want)
    assert np.array_equal(got[0], want[0])
    if skin == 0.0:
        assert np.array_equal(got[2], want[2]) and np.array_equal(got[1], want[1])
    assert rel_force_err(got[2], want[2])[0] < FORCE_TOL
    a.close()
    b.close()
