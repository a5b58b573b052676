"""Requests that name the tensor-core kernel's tile, as the planner takes them."""
import pytest

import stencil3d_gb300 as S


def _plan(storage, **kw):
    return S.plan(S.Grid(64, 64, 64, 4, 4, 4), S.default_opts(25, "wave", storage, **kw))


@pytest.mark.parametrize("storage", ["f16", "bf16", "f16_hl"])
def test_both_tiles_can_be_named(storage):
    for kw in (dict(kernel="mma", tile_j=32), dict(tile_j=32), dict(kernel="mma", tile_j=32, stages=8)):
        info = _plan(storage, **kw)
        assert (info.kernel, info.tile_j, info.tile_k) == (S.KERNEL_MMA, 32, 64)
    info = _plan(storage, kernel="mma", tile_j=16)
    assert (info.kernel, info.tile_j, info.tile_k) == (S.KERNEL_MMA, 16, 152)


@pytest.mark.parametrize("storage,kw", [
    ("f16", dict(kernel="mma", tile_j=24)), ("f16", dict(kernel="tma", tile_j=32)), ("f16", dict(tile_j=64)),
    ("f16_hl", dict(kernel="mma", tile_j=32, stages=4)), ("f16_hl", dict(kernel="mma", tile_j=16, stages=8)),
    ("f16", dict(tile_j=32, stages=6)), ("f16_hilo", dict(tile_j=32))])
def test_other_heights_and_depths_are_refused(storage, kw):
    with pytest.raises(S.St3dError) as e:
        _plan(storage, **kw)
    assert e.value.status == S.api.ERR_UNSUPPORTED
