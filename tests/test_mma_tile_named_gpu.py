"""The tensor-core kernel's tile by name: a context made anew from what
st3d_get_info reports of one runs the same kernel on the same tile.  Bar: tile,
and the bits of the default's run."""
import numpy as np
import pytest

import stencil3d_gb300 as S
from tests.test_f16_gpu import _inputs

pytestmark = pytest.mark.gpu


def _run(grid, storage, **kw):
    v, s, u = _inputs(grid, 3, False)
    g = S.Grid(*grid)
    with S.Stencil(g, 25, "wave", storage, dt=5e-4, **kw) as st:
        st.upload(v, s, u)
        st.iterate(5)
        a, b = g.empty(), g.empty()
        st.download(a, b)
        st.synchronize()
        return st.info(), g.interior(a).copy(), g.interior(b).copy()


@pytest.mark.parametrize("storage", ["f16", "bf16", "f16_hl"])
@pytest.mark.parametrize("grid,tile", [((20, 40, 70, 4, 4, 4), (32, 64)), ((64, 512, 152, 4, 4, 4), (16, 152))])
def test_a_context_made_from_its_info_is_the_same(grid, tile, storage):
    info, a, b = _run(grid, storage)
    assert (info.tile_j, info.tile_k) == tile
    for kernel in (info.kernel,) + ((0,) if tile[0] == 32 else ()):  # 0: automatic
        again, a2, b2 = _run(grid, storage, kernel=kernel, tile_j=info.tile_j, ichunk=info.ichunk)
        assert (again.kernel, again.tile_j, again.tile_k, again.ichunk) == \
            (S.KERNEL_MMA, info.tile_j, info.tile_k, info.ichunk)
        np.testing.assert_array_equal(a, a2)
        np.testing.assert_array_equal(b, b2)
    # either tile may be named on any grid
    for tj, tk in ((16, 152), (32, 64)):
        named, a2, _ = _run(grid, storage, kernel="mma", tile_j=tj)
        assert (named.tile_j, named.tile_k) == (tj, tk)
        np.testing.assert_array_equal(a, a2)
