"""Several FP32 wave steps of a small grid in one launch, the fields in shared
memory (st3d_kernels_brick.cu).  Bar: bit for bit the steps taken one call at a
time, for grids of one brick and many, bricks of the radius' width, ragged rows,
one plane, one row and one point, odd step counts, more steps than one launch
takes, a nonzero fixed halo and a source in the last column; and the oracle's
fused flavour on one of them."""
import numpy as np
import pytest

import stencil3d_gb300 as S
from oracle import oracle as O
from tests.helpers import wave_inputs

pytestmark = pytest.mark.gpu

CASES = [((64, 64, 64, 4, 4, 4), 7, (20, 3)), ((64, 64, 64, 4, 4, 4), 25, (5, 4)),
         ((20, 30, 45, 4, 4, 4), 25, (7, 6)), ((9, 9, 9, 4, 4, 4), 25, (5, 5)),
         ((5, 3, 7, 4, 4, 4), 13, (4, 3)), ((1, 40, 100, 4, 4, 4), 7, (6, 6)),
         ((50, 1, 33, 4, 4, 4), 13, (5, 4)), ((1, 1, 1, 4, 4, 4), 7, (3, 4)),
         ((70, 61, 90, 4, 4, 4), 13, (9, 8)), ((108, 109, 107, 4, 4, 4), 7, (3, 300)),
         ((20, 200, 200, 4, 4, 4), 7, (8, 3))]


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
def test_brick_launches_equal_single_steps(grid, points, calls):
    v, s, u = wave_inputs(grid, 31 + points)
    s = O.fill_uniform(grid, 5, 2, -1.0, 1.0, np.float32)
    g = S.Grid(*grid)
    src = (grid[0] // 2, grid[1] // 2, grid[2] - 1)
    va, ua, many = _device(g, points, calls, v, s, u, src, True)
    vb, ub, one = _device(g, points, calls, v, s, u, src, False)
    assert many.launches == sum((n + 255) // 256 for n in calls) and one.launches == sum(calls)
    assert many.step == one.step == sum(calls)
    np.testing.assert_array_equal(g.interior(ua), g.interior(ub))
    np.testing.assert_array_equal(g.interior(va), g.interior(vb))


def test_brick_steps_match_the_oracle():
    grid = (40, 33, 70, 4, 4, 4)
    v, s, u = wave_inputs(grid, 3)
    g = S.Grid(*grid)
    src = (20, 31, 68)
    va, ua, info = _device(g, 25, (6, 5), v, s, u, src, True)
    assert info.launches == 2
    c0, c1, c2 = O.wave_constants(25, 1500.0, 5e-4, 10.0)
    O.iterate_wave(u, v, s, grid, 25, 11, c0, c1, c2, src=src, amps=O.ricker_amps(0, 11, 5e-4), fma=True)
    np.testing.assert_array_equal(g.interior(ua), O.interior(u, grid))
    np.testing.assert_array_equal(g.interior(va), O.interior(v, grid))
