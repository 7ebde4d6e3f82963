"""CPU tests of the C-ABI boundary: the shared library loads, exports exactly what
include/fa_sm100.h declares, the ctypes mirror of fa_params has the C layout, and
argument validation answers with error codes before any CUDA call is made."""
import ctypes
import os
import re
import subprocess

import pytest

from triton_flashattn_b200 import _cabi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "fa_sm100.h")


def _declared_functions():
    text = open(HEADER).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(fa_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    lib = _cabi.load()
    declared = _declared_functions()
    assert len(declared) >= 10
    for name in declared:
        assert hasattr(lib, name), f"{name} is declared in fa_sm100.h but not exported"
    assert sorted(_cabi.EXPORTED_SYMBOLS) == sorted(n for n in declared if n in _cabi.EXPORTED_SYMBOLS)


def test_version_and_status_strings():
    lib = _cabi.load()
    assert lib.fa_version() == 2
    assert _cabi.status_string(0) == "ok"
    for code in range(1, 10):
        assert _cabi.status_string(code) not in ("ok", "unknown error code")
    assert _cabi.status_string(12345) == "unknown error code"


def test_struct_layout_matches_the_header(tmp_path):
    src = tmp_path / "sz.c"
    src.write_text(
        '#include "fa_sm100.h"\n#include <stdio.h>\n#include <stddef.h>\n'
        "int main(void){printf(\"%zu %zu %zu %zu %zu %zu %zu\\n\", sizeof(fa_params), offsetof(fa_params, sm_scale),"
        " offsetof(fa_params, q), offsetof(fa_params, delta), offsetof(fa_params, dbias_stride),"
        " offsetof(fa_params, ds16), offsetof(fa_params, ds16_stride));return 0;}\n")
    exe = tmp_path / "sz"
    subprocess.check_call(["gcc", "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe)])
    c = [int(x) for x in subprocess.check_output([str(exe)]).split()]
    P = _cabi.FaParams
    assert c == [ctypes.sizeof(P), P.sm_scale.offset, P.q.offset, P.delta.offset, P.dbias_stride.offset,
                 P.ds16.offset, P.ds16_stride.offset]


def _params(**kw):
    p = _cabi.FaParams()
    p.struct_size = ctypes.sizeof(_cabi.FaParams)
    p.B = p.H = 1
    p.M = p.N = 128
    p.D = 64
    p.dtype = _cabi.FA_BF16
    p.sm_scale = 0.125
    for k, v in kw.items():
        setattr(p, k, v)
    return p


@pytest.mark.parametrize("entry", ["fa_fwd", "fa_bwd", "fa_bwd_pre", "fa_bwd_dkdv", "fa_bwd_dq"])
def test_validation_error_codes_without_a_gpu(entry):
    fn = getattr(_cabi.load(), entry)
    assert fn(None, None) == 2  # FA_ERR_NULL
    assert fn(ctypes.byref(_params(struct_size=8)), None) == 1  # FA_ERR_ABI
    assert fn(ctypes.byref(_params(M=0)), None) == 3  # FA_ERR_SHAPE
    assert fn(ctypes.byref(_params(D=48)), None) == 3
    assert fn(ctypes.byref(_params(D=256)), None) == 2  # a legal head dim: next complaint is the null pointers
    assert fn(ctypes.byref(_params(dtype=7)), None) == 4  # FA_ERR_DTYPE
    assert fn(ctypes.byref(_params(bias_kind=9)), None) == 4
    assert fn(ctypes.byref(_params()), None) == 2  # pointers are null
    assert fn(ctypes.byref(_params(B=70000)), None) in (2, 9)


def test_selftest_entry_validates_arguments():
    lib = _cabi.load()
    assert lib.fa_selftest_umma(0, 1, None, None, None, 0, None) == 2
    assert lib.fa_last_device_status(0, None) == 2


def _small_params(**kw):
    """A backward over a few rows whose pointers are never followed: the answer comes before any CUDA call, or (device -1) from
    the first one."""
    p = _params(B=2, H=2, M=16, N=16, D=32, device=-1, bias_kind=1, write_dbias=1)
    for name in ("q", "k", "v", "o", "d_o", "dq", "dk", "dv", "bias", "dbias", "lse", "delta", "ds16"):
        setattr(p, name, 4096)
    for name in ("q", "k", "v", "o", "do", "dq", "dk", "dv", "bias", "dbias", "ds16"):
        setattr(p, name + "_stride", (ctypes.c_int64 * 3)(1024, 512, 32))
    for k, v in kw.items():
        setattr(p, k, v)
    return p


@pytest.mark.parametrize("entry", ["fa_fwd", "fa_small_fwd", "fa_bwd", "fa_small_bwd"])
@pytest.mark.parametrize("kind,offset", [(1, 1), (3, 2), (3, 1)])
def test_a_bias_off_its_natural_alignment_is_refused(entry, kind, offset):
    """The kernels for few rows and short sequences load a bias element by element: off its elements that would be a
    misaligned access on the device."""
    fn = getattr(_cabi.load(), entry)
    assert fn(ctypes.byref(_small_params(bias_kind=kind)), None) == 6  # FA_ERR_CUDA: nothing to complain about before
    assert fn(ctypes.byref(_small_params(bias_kind=kind, bias=4096 + offset)), None) == 5  # FA_ERR_ALIGN
    assert fn(ctypes.byref(_small_params(bias_kind=2, write_dbias=0, bias=4096 + 1)), None) == 6  # bytes lie anywhere
    if entry.endswith("bwd"):
        assert fn(ctypes.byref(_small_params(bias_kind=kind, dbias=4096 + offset)), None) == 5


def test_a_gradient_without_places_of_its_own_is_refused():
    lib = _cabi.load()
    for i in range(3):
        st = [1024, 512, 32]
        for bad in (0, -st[i]):
            st[i] = bad
            p = _small_params(dbias_stride=(ctypes.c_int64 * 3)(*st))
            assert lib.fa_small_bwd(ctypes.byref(p), None) == 5
        one = _small_params(dbias_stride=(ctypes.c_int64 * 3)(*st), **{"BHM"[i]: 1})
        assert lib.fa_small_bwd(ctypes.byref(one), None) == 6  # a stride over one element says nothing
    at, odd = ctypes.c_void_p(4096), ctypes.c_void_p(4097)
    assert lib.fa_pack_rows(at, odd, ctypes.c_int64(16), 2, ctypes.c_int64(4), 16, -1, None) == 5


@pytest.mark.parametrize("elem_bytes", [1, 2, 4])
def test_row_copies_refuse_rows_that_32_bits_cannot_count(elem_bytes):
    """Before any CUDA call: such a row would be taken for an empty or a negative one.  The longest row that fits gets as far as
    the device (-1, an error of its own)."""
    lib = _cabi.load()
    buf = ctypes.create_string_buffer(64)
    at = ctypes.c_void_p(ctypes.addressof(buf))
    st = (ctypes.c_int64 * 3)(0, 0, 0)
    longest = (2**31 - 17) // elem_bytes
    for n in (longest + 1, 2**31 // elem_bytes - 1, 2**31 - 1):
        assert lib.fa_pad_rows(at, st, at, st, elem_bytes, 1, 1, 1, n, -1, None) == 9  # FA_ERR_TOO_LARGE
        if elem_bytes > 1:
            assert lib.fa_pack_rows(at, at, ctypes.c_int64(n), elem_bytes, ctypes.c_int64(1), n, -1, None) == 9
    assert lib.fa_pad_rows(at, st, at, st, elem_bytes, 1, 1, 1, longest, -1, None) == 6  # FA_ERR_CUDA


def test_public_api_rejects_cpu_tensors_loudly():
    import torch
    from triton_flashattn_b200 import flash_attention_fn

    q = torch.randn(1, 16, 1, 16, dtype=torch.float16)
    with pytest.raises(ValueError, match="no CPU path"):
        flash_attention_fn(q, q, q)


@pytest.mark.parametrize("transform", ["vmap", "grad", "jvp", "captured"])
@pytest.mark.parametrize("packed", [False, True])
def test_func_transforms_are_refused(transform, packed):
    """There are no rules for torch.func transforms: any call under one raises, also one whose tensors are only
    captured by the transformed function, whatever their device."""
    import torch
    from triton_flashattn_b200 import flash_attention_fn, flash_attention_qkvpacked_fn

    x = torch.zeros(2, 4, 3, 1, 16) if packed else torch.zeros(2, 4, 1, 16)

    def f(t):
        return flash_attention_qkvpacked_fn(t) if packed else flash_attention_fn(t, t, t)

    with pytest.raises(RuntimeError, match="functorch transforms"):
        if transform == "vmap":
            torch.func.vmap(f)(x)
        elif transform == "grad":
            torch.func.grad(lambda t: f(t).sum())(x)
        elif transform == "jvp":
            torch.func.jvp(f, (x,), (x,))
        else:
            torch.func.vmap(lambda s: f(x) * s)(torch.ones(3))
    with pytest.raises((ValueError, TypeError)):  # outside the transform: the ordinary complaint
        f(x)


def test_launch_path_is_rebuilt_for_another_torch(tmp_path, monkeypatch):
    """The launch path is compiled against the installed torch: one built for another torch, or of unknown
    origin, is not up to date however new its file is."""
    import torch
    from triton_flashattn_b200 import build

    lib, stamp = tmp_path / "_fa_torch.so", tmp_path / "stamp"
    monkeypatch.setattr(build, "BINDING_PATH", str(lib))
    monkeypatch.setattr(build, "BINDING_STAMP", str(stamp))
    assert build._binding_stale()  # not there at all
    lib.write_bytes(b"")
    assert build._binding_stale()  # nothing says what it was built against
    stamp.write_text(build._binding_key())
    assert not build._binding_stale()
    monkeypatch.setattr(torch, "__version__", torch.__version__ + ".post1")
    assert build._binding_stale()
