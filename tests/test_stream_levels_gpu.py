"""The streamed drop-in wave call as a pipeline of levels over rows of tiles
(grids beyond shared-memory bricks, 4 to 32 steps).  Bar: two calls in a row
leave bit for bit the host arrays of the DIRECT path on the one-step kernel,
halos included -- 7, 13 and 25 points, the fewest and most levels, odd counts
(the buffers leave swapped), rows that are not whole 16-byte words and arrays
off a 16-byte boundary (the scalar copies), planes and rows that end inside an
item or a slab, halos of 1, 2, 4 and 16, both tile shapes, a source at an edge.
Each case asserts the kernel, its levels and its tile."""
import numpy as np
import pytest

import stencil3d_gb300 as S
from oracle import oracle as O
from tests.helpers import wave_inputs

pytestmark = pytest.mark.gpu

STREAMED, DIRECT = S.api.HOST_STREAMED, S.api.HOST_DIRECT

CASES = [
    # grid, points, steps, source, rows of a tile, elements past a 16-byte boundary
    ((70, 187, 423, 4, 4, 16), 13, 7, (69, 186, 422), 16, 0),
    ((50, 200, 508, 4, 4, 4), 25, 31, (0, 0, 0), 16, 0),
    ((37, 330, 192, 4, 4, 4), 25, 32, (18, 329, 191), 32, 0),
    ((90, 150, 300, 1, 1, 1), 7, 4, (45, 75, 150), 16, 0),
    ((66, 170, 384, 2, 2, 2), 13, 5, None, 16, 0),
    ((64, 256, 512, 4, 4, 4), 7, 20, None, 16, 1),
    ((5, 700, 520, 4, 4, 4), 25, 6, (4, 31, 8), 32, 1),
    ((33, 321, 190, 4, 5, 6), 7, 9, (32, 320, 64), 16, 3),
]


def _run(grid, points, steps, src, shift, inputs, **kw):
    g = S.Grid(*grid)
    held, arrays = [], []
    for a in inputs:
        p = S.PinnedArray((a.size + 4,), np.float32)
        held.append(p)
        arrays.append(p.array[shift:shift + a.size].reshape(a.shape))
        arrays[-1][...] = a
    try:
        with S.Stencil(g, points, "wave", "f32", dt=5e-4, src=src, **kw) as st:
            for _ in range(2):
                st.iterate_host(*arrays, steps)
            info = st.info()
        return arrays[0].copy(), arrays[2].copy(), info
    finally:
        del arrays
        for p in held:
            p.free()


@pytest.mark.parametrize("grid,points,steps,src,rows,shift", CASES,
                         ids=["%d-%s-%d" % (c[1], "x".join(map(str, c[0])), c[2]) for c in CASES])
def test_levels_equal_the_phases(grid, points, steps, src, rows, shift):
    v, _, u = wave_inputs(grid, 11 + points)
    s = O.fill_uniform(grid, 5, 2, -1.0, 1.0, np.float32)
    v1, u1, info = _run(grid, points, steps, src, shift, (v, s, u))
    assert (info.host_path, info.stream_levels, info.stream_tile_j) == (STREAMED, steps, rows)
    v2, u2, info = _run(grid, points, steps, src, shift, (v, s, u), host_path=DIRECT, tile_j=16, stages=4)
    assert info.host_path == DIRECT and info.stream_levels == 0
    np.testing.assert_array_equal(v1, v2)
    np.testing.assert_array_equal(u1, u2)


@pytest.mark.parametrize("steps,levels", [(3, 0), (32, 32), (33, 0)])
def test_levels_are_four_to_thirty_two(steps, levels):
    grid = (40, 200, 520, 4, 4, 4)
    v, s, u = wave_inputs(grid, 3)
    _, _, info = _run(grid, 7, steps, None, 0, (v, s, u), host_path=STREAMED)
    assert info.host_path == STREAMED and info.stream_levels == levels


@pytest.mark.parametrize("grid,points,steps,levels", [
    ((1000, 128, 128, 4, 4, 4), 25, 8, 0), ((1000, 128, 128, 4, 4, 4), 25, 16, 16),
    ((300, 100, 100, 4, 4, 4), 7, 5, 0), ((279, 367, 25, 4, 4, 4), 25, 4, 0), ((160, 160, 160, 4, 4, 4), 13, 6, 0),
    ((160, 160, 160, 4, 4, 4), 13, 7, 7), ((40, 300, 300, 4, 4, 4), 7, 4, 4)])
def test_few_steps_of_long_grids_run_over_chunks(grid, points, steps, levels):
    """Few steps, planes small beside the length: the chunks of planes are the
    faster form (a row of tiles spans all planes)."""
    v, s, u = wave_inputs(grid, 3)
    v1, u1, info = _run(grid, points, steps, None, 0, (v, s, u))
    assert info.host_path == STREAMED and info.stream_levels == levels
    v2, u2, _ = _run(grid, points, steps, None, 0, (v, s, u), host_path=DIRECT, tile_j=16, stages=4)
    np.testing.assert_array_equal(v1, v2)
    np.testing.assert_array_equal(u1, u2)
