"""Several FP32 wave steps in one launch (st3d_kernels_wave.cu).  Bar: bit for
bit the steps taken one call at a time (one launch each), for all columns at
work at once and several turns of them, both tile shapes, ragged rows and
columns, odd and split step counts, a
nonzero fixed halo and a source on a tile's edge; and the oracle's fused
flavour on one of them.  Each case asserts that the launch it means was taken."""
import numpy as np
import pytest

import stencil3d_gb300 as S
from oracle import oracle as O
from tests.helpers import wave_inputs

pytestmark = pytest.mark.gpu

CASES = [
    # grid, points, steps of the two calls
    ((256, 250, 250, 4, 4, 4), 7, (20, 3)),     # all columns at once, several levels
    ((150, 187, 423, 4, 4, 4), 13, (12, 11)),   # the same with ragged rows
    ((171, 169, 265, 4, 4, 4), 25, (40, 7)),    # 32 x 64 tiles
    ((64, 700, 1050, 4, 4, 4), 7, (9, 4)),      # turns, levels a row of tiles behind
    ((64, 700, 1050, 4, 4, 4), 25, (12, 5)),
    ((300, 16, 6000, 4, 4, 4), 7, (8, 8)),      # one row of tiles
    ((300, 3000, 60, 4, 4, 4), 13, (8, 8)),     # one tile along k
    ((48, 2000, 1500, 4, 4, 4), 13, (8, 9)),    # many turns
]


def _device(g, points, calls, v, s, u, src, lump):
    with S.Stencil(g, points, "wave", "f32", dt=5e-4, src=src) as st:
        st.upload(v, s, u)
        for n in calls:
            if lump:
                st.iterate(n)
            else:
                for _ in range(n):
                    st.iterate(1)
        vo, uo = g.empty(), g.empty()
        st.download(vo, uo)
        st.synchronize()
        return vo, uo, st.info()


@pytest.mark.parametrize("grid,points,calls", CASES,
                         ids=["%d-%s" % (c[1], "x".join(map(str, c[0][:3]))) for c in CASES])
def test_launches_of_many_steps_equal_single_steps(grid, points, calls):
    v, s, u = wave_inputs(grid, 31 + points)
    s = O.fill_uniform(grid, 5, 2, -1.0, 1.0, np.float32)
    g = S.Grid(*grid)
    src = (grid[0] // 2, min(grid[1] - 1, 15), grid[2] - 1)
    va, ua, many = _device(g, points, calls, v, s, u, src, True)
    vb, ub, one = _device(g, points, calls, v, s, u, src, False)
    assert one.launches == sum(calls)
    assert many.launches < one.launches, "the multi-step launch was not taken"
    assert many.step == one.step == sum(calls)
    np.testing.assert_array_equal(g.interior(ua), g.interior(ub))
    np.testing.assert_array_equal(g.interior(va), g.interior(vb))


def test_many_steps_match_the_oracle():
    grid = (20, 260, 1030, 4, 4, 4)
    v, s, u = wave_inputs(grid, 3)
    g = S.Grid(*grid)
    src = (10, 31, 128)
    va, ua, info = _device(g, 13, (6, 5), v, s, u, src, True)
    assert info.launches == 2
    c0, c1, c2 = O.wave_constants(13, 1500.0, 5e-4, 10.0)
    O.iterate_wave(u, v, s, grid, 13, 11, c0, c1, c2, src=src, amps=O.ricker_amps(0, 11, 5e-4), fma=True)
    np.testing.assert_array_equal(g.interior(ua), O.interior(u, grid))
    np.testing.assert_array_equal(g.interior(va), O.interior(v, grid))


def test_many_steps_beyond_one_launch():
    """More steps than one launch takes (its progress words and amplitudes)."""
    grid = (96, 180, 300, 4, 4, 4)
    v, s, u = wave_inputs(grid, 8)
    g = S.Grid(*grid)
    va, ua, many = _device(g, 7, (301,), v, s, u, (48, 90, 150), True)
    vb, ub, _ = _device(g, 7, (301,), v, s, u, (48, 90, 150), False)
    assert 2 <= many.launches < 10
    np.testing.assert_array_equal(ua, ub)
    np.testing.assert_array_equal(va, vb)
