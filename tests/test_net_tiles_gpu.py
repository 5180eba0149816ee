"""Convolution and weight gradient at the edges of their bricks (8 x 16 voxels, the 16
along y or z): grids below, at and just past a brick, stacks of several bricks,
thin grids, and more bricks than a sum in TMEM takes."""
import ctypes as C

import numpy as np
import pytest

import net_oracle as N
from conftest import rel_l2

pytestmark = pytest.mark.gpu

# (nx, ny, nz); the last ones: 16 bricks of 128 voxels and more per CTA
SHAPES = [(1, 1, 1), (8, 16, 1), (9, 17, 2), (7, 3, 33), (8, 2, 16), (17, 31, 5), (3, 40, 7), (40, 33, 19)]


def _bits(a):
    import torch
    return torch.from_numpy(N.to_bits(a).view(np.int16).copy()).cuda()


def _ptr(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 64), (64, 64), (64, 32), (32, 16)])
@pytest.mark.parametrize("shape", SHAPES)
def test_conv_and_wgrad_match_oracle(shape, cin, cout):
    import torch
    from mizuho_edit_gb300 import capi
    L = capi.load()
    nx, ny, nz = shape
    rng = np.random.default_rng(nx * 100 + ny + cin + cout)
    x = N.bf16(rng.standard_normal((nz, ny, nx, cin)))
    w = N.bf16(rng.standard_normal((cout, 27, cin)) * 0.2)
    b = rng.standard_normal(cout).astype(np.float32)
    gy = N.bf16(rng.standard_normal((nz, ny, nx, cout)))
    dx, dw, dg, db = _bits(x), _bits(w), _bits(gy), torch.from_numpy(b).cuda()
    out = torch.full((nz * ny * nx * cout + 64,), 7.0, device="cuda")     # 64 more: nothing is written past the end
    capi.check(L.wpf_conv3d(cin, cout, nx, ny, nz, _ptr(dx), _ptr(dw), _ptr(db), 0, None, _ptr(out), None), "conv")
    got = out.cpu().numpy()
    # products of bf16 are exact in FP32; 27 cin of them summed in FP32: a few 1e-7 of the result
    assert rel_l2(got[:-64].reshape(nz, ny, nx, cout), N.conv3d(x, w, b)) < 1e-5
    assert (got[-64:] == 7.0).all()
    gw_ref, gb_ref = N.conv3d_wgrad(x, gy)
    for pad in (0, 1):                                                     # gw on a 16-byte boundary, and off one
        gw = torch.zeros(cout * 27 * cin + pad, device="cuda")
        gb = torch.zeros(cout, device="cuda")
        capi.check(L.wpf_conv3d_wgrad(cin, cout, nx, ny, nz, _ptr(dx), _ptr(dg), C.c_void_p(gw.data_ptr() + 4 * pad),
                                      _ptr(gb), None), "wgrad")
        assert rel_l2(gw.cpu().numpy()[pad:].reshape(cout, 27, cin), gw_ref) < 1e-5
        assert rel_l2(gb.cpu().numpy(), gb_ref) < 1e-5


@pytest.mark.parametrize("shift", [1, 4])
def test_operands_off_16_byte_boundaries(shift):
    """The weight gradient takes its operands on any boundary; the convolution, whose copies and
    stores are 16 bytes wide, refuses them."""
    import torch
    from mizuho_edit_gb300 import capi
    L = capi.load()
    nx, ny, nz, cin, cout = 9, 17, 3, 16, 32
    rng = np.random.default_rng(shift)
    x = N.bf16(rng.standard_normal((nz, ny, nx, cin)))
    gy = N.bf16(rng.standard_normal((nz, ny, nx, cout)))

    def off(a):
        b = _bits(a).reshape(-1)
        t = torch.zeros(b.numel() + 16, dtype=b.dtype, device="cuda")
        t[shift:shift + b.numel()] = b
        return t, C.c_void_p(t.data_ptr() + 2 * shift)

    (tx, px), (tg, pg) = off(x), off(gy)
    gw_ref, gb_ref = N.conv3d_wgrad(x, gy)
    ax, ag = _bits(x), _bits(gy)
    for qx, qg in ((px, pg), (px, _ptr(ag)), (_ptr(ax), pg)):
        gw = torch.zeros(cout * 27 * cin, device="cuda")
        gb = torch.zeros(cout, device="cuda")
        capi.check(L.wpf_conv3d_wgrad(cin, cout, nx, ny, nz, qx, qg, _ptr(gw), _ptr(gb), None), "wgrad")
        assert rel_l2(gw.cpu().numpy().reshape(cout, 27, cin), gw_ref) < 1e-5
        assert rel_l2(gb.cpu().numpy(), gb_ref) < 1e-5
    w = torch.zeros(cout * 27 * cin + 16, dtype=torch.int16, device="cuda")
    out = torch.zeros(nz * ny * nx * cout + 16, device="cuda")
    bad = C.c_void_p(w.data_ptr() + 2 * shift)
    assert L.wpf_conv3d(cin, cout, nx, ny, nz, px, _ptr(w), None, 0, None, _ptr(out), None) != 0
    assert L.wpf_conv3d(cin, cout, nx, ny, nz, _ptr(ax), bad, None, 0, None, _ptr(out), None) != 0
    assert L.wpf_conv3d(cin, cout, nx, ny, nz, _ptr(ax), _ptr(w), None, 0, None, C.c_void_p(out.data_ptr() + 4), None) != 0
