"""The bench's launch count: runs of steps by the engine's rule, and the kernels of
each form of the step."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


@pytest.mark.parametrize("calls,t0,since,runs,reorders", [
    # a first call: the shortest run at once, a longer one behind as many steps
    ([20], 1, 0, [2, 2, 2, 2, 8, 4], 0),
    ([5, 20], 6, 5, [2, 2, 2, 2, 8, 4], 0),
    ([4, 4], 5, 4, [4], 0),  # the first call had use for the run of four
    ([20, 20], 21, 20, [8, 8, 4], 0),
    ([20, 1], 21, 20, [1], 0),
    ([20, 3], 21, 20, [2, 1], 0),
    # a step that removes the drift (counter 100), and a reorder after 100 steps
    ([20, 20], 95, 30, [4, 1, 1, 8, 4, 2], 0),
    ([20, 20], 41, 95, [4, 1, 8, 4, 2, 1], 1),
])
def test_runs_of_a_call(calls, t0, since, runs, reorders):
    assert bench.step_runs(calls, t0, since) == (runs, reorders)


def test_runs_after_a_long_call():
    assert bench.step_runs([5, 20], 6, 5, step_ms=1.7) == ([8, 8, 4], 0)
    assert bench.step_runs([5], 6, 5, step_ms=1.7) == ([2, 2, 1], 0)
    assert bench.step_runs([2, 20], 3, 2, step_ms=1.7) == ([2, 2, 2, 2, 8, 4], 0)


def test_launches_of_a_call():
    # 984k beads, kept lists: 20 steps, 7 rebuilds, runs of 8, 8 and 4 with 17 fused pairs
    assert bench.timed_launches([40, 20], True, 984040, 92000, 7, 2571, 70) == 20 * 9 + 7 * 6 - 17
    # the same up to 400,000 rows: the rebuild's kernels in every step
    assert bench.timed_launches([40, 20], True, 300000, 92000, 7, 2571, 70) == 20 * 14 - 17
    assert bench.timed_launches([40, 20], True, 8000, 600, 7, 2571, 70) == 20 * 13 - 17
    # without kept lists, and with a drift removal and a reorder
    assert bench.timed_launches([40, 20], False, 8000, 600, 0, 2571, 70) == 20 * 11 - 17
    assert (bench.timed_launches([20, 20], False, 8000, 60000, 0, 95, 95)
            == 20 * 12 + 4 + 3 - sum(r - 1 for r in bench.step_runs([20, 20], 95, 95)[0]))
    # one launch per step, the drift removal's kernels in each
    assert bench.timed_launches([40, 20], True, 984040, 92000, 7, 2571, 70, plain=True) == 20 * 18
