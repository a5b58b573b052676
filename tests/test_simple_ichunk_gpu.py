"""The direct-load kernel's planes per block: st3d_get_info reports the length
that runs.  Bar: where none is named, a length that fills the GPU's blocks (64
planes of a 64^3 grid are 16 blocks), the same when named again, and a named
one as it was named; the bits do not depend on it."""
import numpy as np
import pytest

import stencil3d_gb300 as S
from tests.helpers import wave_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f32", "f64"])
@pytest.mark.parametrize("points", [7, 25])
def test_info_reports_the_length_that_runs(points, storage):
    grid = (64, 64, 64, 4, 4, 4)
    g = S.Grid(*grid)
    np_t = np.float64 if storage == "f64" else np.float32
    v, s, u = wave_inputs(grid, 5, np_t)
    runs = []
    for ichunk in (0, 64, None):
        named = runs[0][0] if ichunk is None else ichunk
        with S.Stencil(g, points, "wave", storage, kernel="simple", dt=5e-4, ichunk=named) as st:
            info = st.info()
            assert info.kernel == S.KERNEL_SIMPLE and (named == 0 or info.ichunk == named)
            vv, uu = v.copy(), u.copy()
            st.iterate_host(vv, s, uu, 3)
            runs.append((info.ichunk, vv, uu))
    assert 0 < runs[0][0] < 64
    for _, vv, uu in runs[1:]:
        np.testing.assert_array_equal(vv, runs[0][1])
        np.testing.assert_array_equal(uu, runs[0][2])
