"""Host arrays may be written again as soon as st3d_upload returns, whatever the
stream still has to run before it.  Bar: the values the arrays held at the
call, pinned and pageable, rows of whole 16-byte words and not, with the
transfers queued behind a long run of steps."""
import numpy as np
import pytest

import stencil3d_gb300 as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _arrays(shape, dtype, pinned):
    if not pinned:
        return [np.empty(shape, dtype) for _ in range(3)], []
    held = [S.PinnedArray(shape, dtype) for _ in range(3)]
    return [p.array for p in held], held


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("grid", [(60, 250, 256, 4, 4, 4), (60, 250, 253, 4, 4, 4), (60, 128, 128, 2, 2, 1)])
def test_arrays_are_free_when_the_upload_returns(grid, dtype, pinned):
    np_t = np.float64 if dtype == "f64" else np.float32
    g = S.Grid(*grid)
    want = [O.fill_uniform(grid, 3, f, -1.0, 1.0, np_t) for f in range(3)]
    arrays, held = _arrays(g.shape, np_t, pinned)
    try:
        with S.Stencil(g, 7, "ref", dtype) as st:
            for a, w in zip(arrays, want):
                a[...] = w
            st.upload(*arrays)
            st.synchronize()
            for n in range(400):  # a launch each: the queue the next upload waits behind
                st.iterate(1)
            st.upload(*arrays)
            for a in arrays:
                a[...] = 9.0
            v, u = g.empty(np_t), g.empty(np_t)
            st.download(v, u)
    finally:
        del arrays
        for p in held:
            p.array = None
            p.free()
    np.testing.assert_array_equal(g.interior(v), O.interior(want[0], grid))
    np.testing.assert_array_equal(g.interior(u), O.interior(want[2], grid))
