"""Page-locked host arrays are read and written over the host link by the kernels, any
other host arrays by copies: the same rows, bit for bit, in both directions and through
steps on host arrays, with and without kept lists; a page-locked array at an odd address
takes the copies."""
import numpy as np
import pytest

from helpers import mdpd_params, mixed_system, warren_params
from implicit_dpd_gb300 import configs
from implicit_dpd_gb300.engine import Engine

pytestmark = pytest.mark.gpu

KEYS = ("pos", "vel", "acc")


def _arrays(kind, src):
    """Three arrays of one kind with src's values, and what keeps them alive."""
    import torch

    n = len(src["pos"])
    keep = [torch.empty(24 * n + 16, dtype=torch.uint8, pin_memory=kind != "pageable")
            for _ in KEYS]
    out = [np.frombuffer(t.numpy(), np.float64, 3 * n, offset=4 if kind == "odd" else 0)
           .reshape(n, 3) for t in keep]
    for a, k in zip(out, KEYS):
        a[...] = src[k]
    return out, keep


def _run(kind, system, skin, sort_period):
    box, st, n_amp, p = system
    e = Engine(sort_period=sort_period)
    e.set_params(p)
    e.upload(st)
    if n_amp:
        e.build_topology(n_amp)
    e.set_tuning(1, skin)
    e.step(3)
    src = e.download()
    src["pos"] = np.clip(src["pos"] + 0.01, 0.0, np.nextafter(box, 0.0))
    a, keep = _arrays(kind, src)
    e.set_dynamics(*a)
    b, keep_b = _arrays(kind, src)
    for x in b:
        x[...] = -1.0
    e.download_dynamics(*b)
    for x, k in zip(b, KEYS):
        assert np.array_equal(x, src[k]), k
    for _ in range(3):
        e.step_host(*a)
    out = [x.copy() for x in a]
    e.close()
    return out


@pytest.mark.parametrize("skin", [0.0, 0.25])
@pytest.mark.parametrize("which", ["mixed", 43, 256, 1])
def test_host_arrays_of_any_kind(which, skin):
    if which == "mixed":
        box, st, n_amp = mixed_system(seed=81)
        system = (box, st, n_amp, mdpd_params(box))
    else:  # remainders of the blocks of numbers
        box = np.array([5.0, 5.5, 6.0])
        system = (box, configs.liquid(box, which / box.prod(), seed=2), 0, warren_params(box))
    want = _run("pageable", system, skin, 2)
    for kind in ("pinned", "odd"):
        for x, y, k in zip(_run(kind, system, skin, 2), want, KEYS):
            assert np.array_equal(x, y), (kind, k)
