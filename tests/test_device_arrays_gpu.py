"""Device arrays in st3d_upload and st3d_download: the layout kernels read and
write them directly.  Bar: the values the host-array route moves, for rows
that are and are not whole 16-byte words, FP32 and FP64, k halos beside 4, one
thin grid, and arrays that start one element past a 16-byte boundary; points
outside the interior rows of the target stay untouched."""
import ctypes as C

import numpy as np
import pytest

import stencil3d_gb300 as S
from stencil3d_gb300 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu

GRIDS = [(5, 7, 64, 4, 4, 4), (3, 9, 61, 4, 4, 4), (6, 5, 70, 4, 4, 5), (2, 3, 1, 4, 4, 16),
         (4, 130, 257, 2, 3, 1), (1, 1, 1030, 4, 4, 2)]


def _device(a, shift):
    torch = pytest.importorskip("torch")
    t = torch.empty(a.size + 4, dtype=torch.from_numpy(a).dtype, device="cuda")
    t = t[shift:shift + a.size].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("grid", GRIDS)
def test_device_arrays_move_the_host_route_values(grid, shift, dtype):
    torch = pytest.importorskip("torch")
    np_t = np.float64 if dtype == "f64" else np.float32
    g = S.Grid(*grid)
    v, s, u = (O.fill_uniform(grid, 3, f, -1.0, 1.0, np_t) for f in range(3))
    dv, ds, du = (_device(a, shift) for a in (v, s, u))
    ov, ou = _device(np.full_like(v, -7.0), shift), _device(np.full_like(v, -7.0), shift)
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr())
    points = 7 if min(grid[3:]) < 2 else 13
    hv, hu = np.full_like(v, -7.0), np.full_like(u, -7.0)
    with S.Stencil(g, points, "ref", dtype) as a, S.Stencil(g, points, "ref", dtype) as b:
        a.upload(v, s, u)
        assert api.lib().st3d_upload(b.handle, p(dv), p(ds), p(du)) == 0
        for st in (a, b):
            st.iterate(2)
        a.download(hv, hu)
        assert api.lib().st3d_download(b.handle, p(ov), p(ou)) == 0
    np.testing.assert_array_equal(ov.cpu().numpy(), hv)
    np.testing.assert_array_equal(ou.cpu().numpy(), hu)


@pytest.mark.parametrize("storage", ["f16", "bf16", "f16_hl", "f16_hilo"])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("grid", [(5, 7, 64, 4, 4, 4), (3, 70, 61, 4, 4, 4), (6, 33, 262, 4, 4, 5),
                                  (2, 3, 1, 4, 4, 16)])
def test_device_arrays_in_16_bit_storage(grid, shift, storage):
    """Maxima, encoding and decoding straight from and to device arrays: the
    host-array route's words, at rows that are and are not whole fours and
    planes of several pieces."""
    torch = pytest.importorskip("torch")
    g = S.Grid(*grid)
    fields = []
    for f in range(3):
        a = np.zeros(O.shape(grid), np.float32)
        O.interior(a, grid)[...] = O.interior(O.fill_uniform(grid, 5, f, -3.0, 3.0), grid)
        fields.append(a)
    dev = [_device(a, shift) for a in fields]
    out = [_device(np.full_like(fields[0], -7.0), shift) for _ in range(2)]
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr())
    hv, hu = np.full_like(fields[0], -7.0), np.full_like(fields[0], -7.0)
    with S.Stencil(g, 7, "wave", storage, dt=1e-3) as a, S.Stencil(g, 7, "wave", storage, dt=1e-3) as b:
        a.upload(*fields)
        assert api.lib().st3d_upload(b.handle, *(p(t) for t in dev)) == 0
        for st in (a, b):
            st.iterate(2)
        a.download(hv, hu)
        assert api.lib().st3d_download(b.handle, p(out[0]), p(out[1])) == 0
        # a nonzero halo point is refused as it is on the host route
        bad = dev[2].clone()
        bad.view(-1)[0 if grid[3] <= 4 else -1] = 1.0
        torch.cuda.synchronize()
        assert api.lib().st3d_upload(b.handle, None, None, p(bad)) == S.api.ERR_UNSUPPORTED
    np.testing.assert_array_equal(out[0].cpu().numpy(), hv)
    np.testing.assert_array_equal(out[1].cpu().numpy(), hu)


@pytest.mark.parametrize("storage", ["f16", "bf16", "f16_hl"])
@pytest.mark.parametrize("grid", [(5, 9, 64, 4, 4, 4), (3, 40, 61, 5, 5, 5)])
def test_one_device_array_of_the_pair(grid, storage):
    """u or v alone: the other's values come from an earlier upload (then from
    the device state once a step was taken); a halo point of either is named."""
    torch = pytest.importorskip("torch")
    g = S.Grid(*grid)
    fields = []
    for f in range(5):
        a = np.zeros(O.shape(grid), np.float32)
        O.interior(a, grid)[...] = O.interior(O.fill_uniform(grid, 5, f, -3.0, 3.0), grid)
        fields.append(a)
    dev = [_device(a, 0) for a in fields]
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr())
    up, err = api.lib().st3d_upload, S.api.ERR_UNSUPPORTED
    got = []
    with S.Stencil(g, 7, "wave", storage, dt=1e-3) as a, S.Stencil(g, 7, "wave", storage, dt=1e-3) as b:
        for st, arr in ((a, [x.ctypes.data_as(C.c_void_p) for x in fields]), (b, [p(t) for t in dev])):
            assert up(st.handle, arr[0], arr[1], arr[2]) == 0
            assert up(st.handle, None, None, arr[3]) == 0
            assert up(st.handle, arr[4], None, None) == 0
            st.iterate(3)
            assert up(st.handle, None, None, arr[0]) == 0
            st.iterate(2)
            hv, hu = np.zeros_like(fields[0]), np.zeros_like(fields[0])
            st.download(hv, hu)
            st.synchronize()
            got.append((hv, hu))
        for which, name in ((0, "u or v"), (2, "u")):
            bad = dev[which].clone()
            bad.view(-1)[bad.numel() // 2] = 1.0  # a k halo point where zs is even, an inner one else
            i, j, k = np.unravel_index(bad.numel() // 2, fields[0].shape)
            inner = all(grid[3 + x] <= q < grid[3 + x] + grid[x] for x, q in enumerate((i, j, k)))
            if inner:
                bad.view(-1)[bad.numel() // 2 - k] = 1.0
            torch.cuda.synchronize()
            args = [None, None, None]
            args[which] = p(bad)
            assert up(b.handle, *args) == err
            assert ("; %s has" % name) in S.last_error()
    # a NaN is no halo value to refuse, on either route
    host = fields[2].copy()
    host.reshape(-1)[0] = np.nan
    nan = _device(host, 0)
    torch.cuda.synchronize()
    for u in (host.ctypes.data_as(C.c_void_p), p(nan)):
        with S.Stencil(g, 7, "wave", storage, dt=1e-3) as st:
            assert up(st.handle, p(dev[0]), p(dev[1]), u) == 0
    for x, y in zip(*got):
        np.testing.assert_array_equal(x, y)
