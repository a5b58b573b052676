"""The two tiles of the tensor-core kernel (st3d_kernels_mma16.cu), 32 x 64 and
16 x 152.  Bar: the same bits -- a 16 x 8 block is summed by the same products
in the same order on either -- on ragged rows and columns, several units a CTA,
sources on a tile's edges, every storage and order.  Each case asserts that the
default took the tile it means."""
import numpy as np
import pytest

import stencil3d_gb300 as S
from tests.test_f16_gpu import _inputs

pytestmark = pytest.mark.gpu

CASES = [
    # grid, chunk (0 = default), source, the default's tile
    ((20, 40, 70, 4, 4, 4), 0, (10, 31, 63), (32, 64)),
    ((17, 33, 65, 4, 4, 4), 0, (0, 32, 64), (32, 64)),      # one row and column past a tile
    ((9, 31, 63, 4, 4, 4), 0, (8, 15, 7), (32, 64)),        # one short
    ((60, 70, 203, 4, 4, 4), 3, (30, 16, 202), (32, 64)),   # several units a CTA
    ((3, 97, 129, 4, 4, 4), 0, (1, 96, 128), (32, 64)),     # fewer planes than stages
    ((64, 512, 152, 4, 4, 4), 0, (32, 511, 151), (16, 152)),
]


@pytest.mark.parametrize("storage", ["f16", "bf16", "f16_hl"])
@pytest.mark.parametrize("points", [7, 13, 25])
@pytest.mark.parametrize("grid,chunk,src,tile", CASES, ids=["x".join(map(str, c[0][:3])) for c in CASES])
def test_tiles_agree(grid, chunk, src, tile, points, storage):
    v, s, u = _inputs(grid, 7 + points, False)
    g = S.Grid(*grid)
    out = []
    for kw in (dict(), dict(tile_j=16)):
        with S.Stencil(g, points, "wave", storage, kernel="mma", dt=5e-4, src=src, ichunk=chunk, **kw) as st:
            st.upload(v, s, u)
            st.iterate(9)
            a, b = g.empty(), g.empty()
            st.download(a, b)
            st.synchronize()
            info = st.info()
            out.append((g.interior(a).copy(), g.interior(b).copy(), (info.tile_j, info.tile_k)))
    assert out[0][2] == tile and out[1][2] == (16, 152)
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
