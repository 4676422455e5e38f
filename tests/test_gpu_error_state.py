"""A call that the runtime refuses ends in its error and leaves none behind: the
next calls, the engine's and other libraries', work."""
import mmap

import numpy as np
import pytest

from helpers import mdpd_params, mixed_system
from implicit_dpd_gb300.engine import Engine, EngineError

pytestmark = pytest.mark.gpu


def test_a_refused_copy_does_not_fail_the_next_call():
    import torch

    box, st, n_amp = mixed_system(seed=82)
    n, page = len(st["pos"]), mmap.PAGESIZE
    e = Engine()
    e.set_params(mdpd_params(box, time=4))
    e.upload(st)
    e.build_topology(n_amp, [0])
    e.step(1)
    torch.zeros(1, device="cuda")
    # rows that are page-locked up to a page within them: the runtime refuses the copy
    size = -(-24 * n // page) * page
    assert size > page
    m = mmap.mmap(-1, size)
    part = np.frombuffer(m, np.float64, 3 * n).reshape(n, 3)
    part[...] = st["pos"]
    rt = torch.cuda.cudart()
    assert int(rt.cudaHostRegister(part.ctypes.data, page, 0)) == 0
    good = [np.array(st[k], np.float64) for k in ("pos", "vel", "acc")]
    try:
        with pytest.raises(EngineError):
            e.set_dynamics(part, good[1], good[2])
        torch.full((5,), 1.0, device="cuda")
        e.step_host(*good)
        with pytest.raises(EngineError):
            e.download_dynamics(part, good[1], good[2])
        e.step(2)
    finally:
        rt.cudaHostUnregister(part.ctypes.data)
    e.close()


def test_an_error_left_by_another_library_is_not_the_exchange_calls():
    import torch

    box, st, n_amp = mixed_system(seed=83)
    e = Engine()
    e.set_params(mdpd_params(box, time=4))
    e.upload(st)
    e.build_topology(n_amp, [0])
    e.density()
    e.force()
    want = e.download_aux(press=True, nei_cm=True, dsr=True), e.download()
    rt = torch.cuda.cudart()

    def refused():  # memory that is not registered: the runtime keeps the error
        assert int(rt.cudaHostUnregister(st["pos"].ctypes.data)) != 0

    refused()
    aux = e.download_aux(press=True, nei_cm=True, dsr=True)
    for k, v in want[0].items():
        assert np.array_equal(aux[k], v, equal_nan=True), k
    refused()
    got = e.download()
    for k in ("pos", "vel", "acc"):
        assert np.array_equal(got[k], want[1][k]), k
    refused()
    e.set_dynamics(got["pos"], got["vel"], got["acc"])
    e.sync()
    e.close()
    try:  # the error goes to its own library
        torch.full((1,), 1.0, device="cuda")
    except RuntimeError:
        pass
