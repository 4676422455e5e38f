"""Host arrays that kernels read or write over the host link lie, whole, in one
page-locked allocation or registration (csrc/host_range.hpp); others go through
the copies, which refuse arrays that are page-locked in parts."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_only_whole_allocations_are_linked(tmp_path):
    exe = tmp_path / "host_range_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I",
                    os.path.join(ROOT, "implicit_dpd_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "host_range_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def _registered(st, ranges):
    """Three arrays with st's rows in page-aligned memory, each from the end of a page
    on over at least one whole page, with ranges(size) of it page-locked."""
    import mmap

    import torch

    rt = torch.cuda.cudart()
    torch.zeros(1, device="cuda")
    n, page = len(st["pos"]), mmap.PAGESIZE
    off = page - 4096
    size = -(-(off + 24 * n) // page) * page
    assert size >= 3 * page
    arrays, held = [], []
    for k in ("pos", "vel", "acc"):
        m = mmap.mmap(-1, size)
        a = np.frombuffer(m, np.float64, 3 * n, offset=off).reshape(n, 3)
        a[...] = st[k]
        for lo, hi in ranges(size, page):
            assert int(rt.cudaHostRegister(a.ctypes.data - off + lo, hi - lo, 0)) == 0
            held.append((m, a.ctypes.data - off + lo))
        arrays.append(a)
    return arrays, held


def _unregister(held):
    import torch

    for _, p in held:
        torch.cuda.cudart().cudaHostUnregister(p)


def _engine():
    from helpers import mdpd_params, mixed_system
    from implicit_dpd_gb300.engine import Engine

    box, st, n_amp = mixed_system(seed=82)
    e = Engine()
    e.set_params(mdpd_params(box, time=4))
    e.upload(st)
    e.build_topology(n_amp, [0])
    e.set_tuning(1, 0.2)
    e.step(1)
    return e, st


@pytest.mark.gpu
def test_registered_arrays_are_linked():
    out = []
    for registered in (True, False):
        e, st = _engine()
        held = []
        rows = [np.array(st[k], np.float64) for k in ("pos", "vel", "acc")]
        if registered:
            rows, held = _registered(st, lambda size, page: [(0, size)])
        try:
            for _ in range(3):
                e.step_host(*rows)
            out.append([x.copy() for x in rows])
            for x in rows:
                x[...] = -1.0
            e.download_dynamics(*rows)
            for x, y in zip(rows, out[-1]):
                assert np.array_equal(x, y)
            e.close()
        finally:
            _unregister(held)
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.gpu
def test_arrays_registered_at_both_ends_only_are_refused():
    """As by the copies: kernels never read the pages between the registrations."""
    from implicit_dpd_gb300.engine import EngineError

    e, st = _engine()
    rows, held = _registered(st, lambda size, page: [(0, page), (size - page, size)])
    try:
        with pytest.raises(EngineError):
            e.set_dynamics(*rows)
        with pytest.raises(EngineError):
            e.download_dynamics(*rows)
        good = [np.array(st[k], np.float64) for k in ("pos", "vel", "acc")]
        e.step_host(*good)  # the handle works on
        e.close()
    finally:
        _unregister(held)
