"""Mode R takes many steps in one launch (u and s stay fixed, the neighbour
sum of a point is formed once).  Bar: bit for bit the steps taken one call at a
time, and the oracle's fused flavour, at one step, a few, the launch's limit of
1024 and one past it, for every kernel that serves the mode and the streamed
drop-in call; infinities and NaN in s spread as they do step by step."""
import numpy as np
import pytest

import stencil3d_gb300 as S
from oracle import oracle as O
from tests.helpers import mode_r_inputs

pytestmark = pytest.mark.gpu

FORMS = [(7, "f32", "tma"), (13, "f32", "tma"), (25, "f32", "tma"), (25, "f32", "simple"),
         (7, "f64", "auto"), (25, "f64", "auto"), (2, "f32", "auto"), (2, "f64", "auto")]


@pytest.mark.parametrize("steps", [1, 3, 1024, 1025])
@pytest.mark.parametrize("points,dtype,kernel", FORMS)
def test_many_steps_equal_single_steps(points, dtype, kernel, steps):
    grid = (9, 18, 131, 4, 4, 4)
    v, s, u = mode_r_inputs(grid, 61, dtype)
    if steps == 3:
        s[6, 9, 20], s[7, 9, 40], u[8, 9, 60] = np.inf, np.nan, -np.inf
    g = S.Grid(*grid)
    got, one = np.zeros_like(v), np.zeros_like(v)
    with S.Stencil(g, points, "ref", dtype, kernel=kernel) as st:
        st.upload(v, s, u)
        st.iterate(steps)
        st.download(got)
        assert st.info().step == steps
        st.upload(v, s, u)
        for _ in range(steps):
            st.iterate(1)
        st.download(one)
    np.testing.assert_array_equal(O.interior(got, grid), O.interior(one, grid))
    if steps != 3:
        vf = v.copy()
        O.iterate_ref(vf, s, u, grid, points, steps, fma=True)
        np.testing.assert_array_equal(O.interior(got, grid), O.interior(vf, grid))


@pytest.mark.parametrize("steps", [20, 1024, 1025])
def test_streamed_call_takes_many_steps(steps):
    grid = (37, 20, 61, 4, 4, 4)
    v, s, u = mode_r_inputs(grid, 62, "f32")
    pins = [S.PinnedArray(a.shape, a.dtype) for a in (v, s, u)]
    try:
        for p, a in zip(pins, (v, s, u)):
            p.array[...] = a
        with S.Stencil(S.Grid(*grid), 13, "ref", "f32") as st:
            st.iterate_host(*(p.array for p in pins), steps)
            assert st.info().host_path == S.api.HOST_STREAMED
        got = pins[0].array.copy()
    finally:
        for p in pins:
            p.free()
    O.iterate_ref(v, s, u, grid, 13, steps, fma=True)
    np.testing.assert_array_equal(O.interior(got, grid), O.interior(v, grid))
