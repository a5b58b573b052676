"""Pinned drop-in wave calls of more steps than the pipeline of levels takes: a
large grid streams while that is the faster route, a small one and a long call
run phase by phase, and a call that asks for the streamed route gets it at any
length.  Bar: the route, and bit for bit the host arrays of the DIRECT path."""
import numpy as np
import pytest

import stencil3d_gb300 as S
from tests.helpers import wave_inputs
from tests.test_stream_gpu import STREAMED, _call

pytestmark = pytest.mark.gpu

AUTO, DIRECT = S.api.HOST_AUTO, S.api.HOST_DIRECT


@pytest.mark.parametrize("grid,points,steps,asked,taken", [
    ((512, 512, 512, 4, 4, 4), 7, 33, AUTO, STREAMED),
    ((64, 1024, 1024, 4, 4, 4), 25, 33, AUTO, DIRECT),  # too few chunks to hide the transfers
    ((64, 64, 64, 4, 4, 4), 7, 100, AUTO, DIRECT),
    ((120, 276, 603, 4, 4, 4), 7, 33, AUTO, DIRECT),  # rows that are not whole 16-byte words
    ((64, 64, 64, 4, 4, 4), 7, 41, STREAMED, STREAMED),
    ((130, 150, 200, 4, 4, 4), 13, 33, STREAMED, STREAMED),
    ((130, 150, 200, 4, 4, 4), 13, 120, AUTO, DIRECT),
], ids=lambda x: "x".join(map(str, x[:3])) if isinstance(x, tuple) else str(x))
def test_long_calls_take_the_faster_route(grid, points, steps, asked, taken):
    v, s, u = wave_inputs(grid, 7)
    v1, u1, p1 = _call(grid, points, "wave", steps, v, s, u, asked)
    assert p1 == taken
    v2, u2, p2 = _call(grid, points, "wave", steps, v, s, u, DIRECT)
    assert p2 == DIRECT
    np.testing.assert_array_equal(v1, v2)
    np.testing.assert_array_equal(u1, u2)
