"""What a batch reports of its graph calls, and graphs over growing buffers.
Bar: info.launches counts the kernel launches captured -- a step of the queue is
one, a grid that steps by itself one for many steps -- and calls shorter than
one before, longer, and shorter again end where the sequential schedule does."""
import random

import numpy as np
import pytest

import stencil3d_gb300 as S
from tests.test_batch_split_gpu import SPECS, _run

pytestmark = pytest.mark.gpu


def _launches(specs, steps, schedule, **kw):
    with S.Batch([S.Grid(*g) for g, _, _ in specs], [p for _, p, _ in specs], **kw) as b:
        for i in range(len(specs)):
            for f in (S.FIELD_U, S.FIELD_V, S.FIELD_S):
                b.context(i).fill(f, S.FILL_CONST, 0, 0.0)
        b.iterate(steps, schedule)
        one = b.info().launches
        b.iterate(steps, schedule)
        b.synchronize()
        assert b.info().launches == 2 * one
        return one


def test_graph_calls_count_their_launches():
    steps = 200
    # one grid that fits shared memory, alone: a launch for all steps
    assert _launches(SPECS[3:4], steps, "graph") == 1
    # the same in the queue, which a named unit length asks for
    assert _launches(SPECS[3:4], steps, "graph", ichunk=64) == steps
    assert _launches(SPECS[3:4], steps, "persistent") == steps
    # large grids leave the queue: neither its launches alone nor one a grid and step
    assert _launches(SPECS, steps, "graph") not in (steps, len(SPECS) * steps)


def test_a_longer_call_after_a_short_one():
    """The amplitudes' and the queue's buffers grow, the graphs over them are made again."""
    calls = [(5, "graph"), (31, "graph"), (5, "graph"), (300, "graph"), (31, "graph"), (5, "graph")]
    got, info = _run(calls)
    assert info.graphs == 3
    want, _ = _run([(n, "sequential") for n, _ in calls])
    for (ua, va), (ub, vb) in zip(got, want):
        np.testing.assert_array_equal(ua, ub)
        np.testing.assert_array_equal(va, vb)


def test_a_short_call_stays_in_the_queue():
    """16 grids of 64 to 200 points: a few of them alone beside the queue were
    slower at 12 steps (2684 against 2410 us), all alone faster at 60."""
    rng = random.Random(2)
    specs = [(tuple(rng.randint(64, 200) for _ in range(3)) + (4, 4, 4), 0, None) for _ in range(16)]
    specs = [(g, rng.choice([7, 13, 25]), s) for g, _, s in specs]
    assert _launches(specs, 12, "graph") == 12
    assert _launches(specs, 60, "graph") < 60
