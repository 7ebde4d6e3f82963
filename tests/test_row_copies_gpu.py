"""The copies between rows of any pitch and address (fa_pad_rows, fa_pack_rows) against torch's, byte for byte."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
_I64x3 = ctypes.c_int64 * 3


def _random(shape, dtype):
    n = 1
    for s in shape:
        n *= s
    eb = torch.empty(0, dtype=dtype).element_size()
    return torch.randint(0, 256, (n * eb,), dtype=torch.uint8, device="cuda").view(dtype).view(shape)


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("dtype", [torch.uint8, torch.int16, torch.int32])
@pytest.mark.parametrize("N", [1, 3, 7, 8, 15, 16, 17, 49, 130, 777])
@pytest.mark.parametrize("layout", ["offset", "one_row", "heads_last"])
def test_pad_rows(dtype, N, layout, device_ok):
    from triton_flashattn_b200 import _cabi

    B, H, M = 2, 3, 37
    eb = torch.empty(0, dtype=dtype).element_size()
    if layout == "offset":
        src = _random((B, H, M, N + 5), dtype)[..., 3:N + 3]
    elif layout == "one_row":
        src = _random((B, 1, 1, N), dtype).expand(B, H, M, N)
    else:
        src = _random((B, M, H, N), dtype).transpose(1, 2)
    per = 32 // eb
    pad = (N + per - 1) // per * per
    buf = torch.full((B, H, M, pad), 0x55, dtype=dtype, device="cuda")
    st, ds = src.stride(), buf.stride()
    r = _cabi.load().fa_pad_rows(ctypes.c_void_p(buf.data_ptr()), _I64x3(*ds[:3]), ctypes.c_void_p(src.data_ptr()), _I64x3(*st[:3]),
                                 eb, B, H, M, N, 0, _stream())
    assert r == 0
    assert torch.equal(buf[..., :N], src)
    unit = 16 // eb
    filled = (N + unit - 1) // unit * unit
    assert not buf[..., N:filled].any() and (buf[..., filled:] == 0x55).all()


@pytest.mark.parametrize("dtype", [torch.int16, torch.int32])
@pytest.mark.parametrize("N", [1, 3, 7, 9, 49, 130, 777])
@pytest.mark.parametrize("rows", [1, 5, 1000])
def test_pack_rows(dtype, N, rows, device_ok):
    from triton_flashattn_b200 import _cabi

    src = _random((rows, N + 6), dtype)[:, 1:N + 1]
    out = torch.full((rows * N + 64,), 0x55, dtype=dtype, device="cuda")
    r = _cabi.load().fa_pack_rows(ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(src.data_ptr()), ctypes.c_int64(N + 6),
                                  src.element_size(), ctypes.c_int64(rows), N, 0, _stream())
    assert r == 0
    assert torch.equal(out[:rows * N].view(rows, N), src) and (out[rows * N:] == 0x55).all()
