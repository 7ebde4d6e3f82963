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


def test_an_earlier_error_is_not_taken_for_a_copys_own(device_ok):
    """A call on a device that does not exist leaves an error behind in the runtime; the copies after it report their own."""
    from triton_flashattn_b200 import _cabi

    lib = _cabi.load()
    src = _random((5, 9), torch.int16)
    padded = torch.zeros((5, 16), dtype=torch.int16, device="cuda")
    out = torch.zeros(5 * 9 + 3, dtype=torch.int16, device="cuda")

    def pad(device):
        return lib.fa_pad_rows(ctypes.c_void_p(padded.data_ptr()), _I64x3(80, 80, 16), ctypes.c_void_p(src.data_ptr()),
                               _I64x3(45, 45, 9), 2, 1, 1, 5, 9, device, _stream())

    def pack(device):
        return lib.fa_pack_rows(ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(padded.data_ptr()), ctypes.c_int64(16), 2,
                                ctypes.c_int64(5), 9, device, _stream())

    assert pad(-1) == 6 and pad(0) == 0
    assert pack(-1) == 6 and pack(0) == 0
    assert torch.equal(out[:45].view(5, 9), src)
