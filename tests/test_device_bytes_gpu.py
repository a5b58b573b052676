"""st3d_info.device_bytes with the multi-step wave launches' progress words (128
bytes a step and column of tiles: over 1 MB for these grids).  Bar: they are
counted, and no more is reported than making the contexts took from the
device's free memory."""
import pytest

import stencil3d_gb300 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [7, 25])
@pytest.mark.parametrize("grid", [(256, 256, 256), (40, 1400, 1024)])
def test_device_bytes_count_the_progress_words(grid, points):
    torch = pytest.importorskip("torch")
    g = S.Grid(*grid, 4, 4, 4)
    with S.Stencil(g, points, "wave", "f32", dt=5e-4):
        pass  # the library's own first allocations
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with S.Stencil(g, points, "wave", "f32", dt=5e-4) as st, \
            S.Stencil(g, points, "wave", "f32", dt=5e-4, tile_j=16, stages=4) as plain:
        taken = before - torch.cuda.mem_get_info()[0]
        held = st.info().device_bytes + plain.info().device_bytes
        assert st.info().device_bytes - plain.info().device_bytes > 1 << 20
    assert held <= taken
