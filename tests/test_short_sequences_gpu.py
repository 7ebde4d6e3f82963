"""The kernels for short sequences (M, N, D <= 64): edges of their 16-row tiles against the fp32 oracle, biases in layouts
the tile kernels do not take, and what the C entries refuse."""
import ctypes

import pytest
import torch

from tests._util import compare, make_inputs, run_ours
from tests.test_robustness_gpu import SENT16, SENT32, _guarded, _guards_intact

pytestmark = pytest.mark.gpu
BF, HF = torch.bfloat16, torch.float16


@pytest.mark.parametrize("M,N", [(1, 1), (16, 64), (17, 1), (17, 17), (33, 47), (48, 49), (49, 49), (64, 16), (64, 64), (64, 65),
                                 (65, 64)])
@pytest.mark.parametrize("D,dtype,kind,causal", [(16, HF, "float", False), (32, BF, "float", True), (64, HF, "float", True),
                                                 (32, HF, "bool", True), (64, BF, "bool", False), (16, BF, None, True),
                                                 (64, HF, None, False)])
def test_edges_against_oracle(M, N, D, dtype, kind, causal, device_ok):
    q, k, v, bias, do = make_inputs(3, M, N, 3, D, dtype, kind, 100 + M + N)
    ours = run_ours(q, k, v, bias, causal, None, do)
    compare(ours, q, k, v, bias, causal, None, do, dtype, label=f"{M}x{N}: ")


@pytest.mark.parametrize("S", [48, 49])
@pytest.mark.parametrize("layout", ["sliced", "heads_last", "expanded", "f32_sliced"])
def test_bias_in_any_layout(layout, S, device_ok):
    """A bias whose rows are not 16-byte aligned, in another order or expanded, gives what its copy into padded rows gives
    (48 columns: there pairs of elements are accessed at once), and that is right."""
    from triton_flashattn_b200 import flash_attention_fn

    B, H, D = 3, 4, 32
    q, k, v, bias, do = make_inputs(B, S, S, H, D, HF, "float", 77)
    if layout == "f32_sliced":
        bias = bias.float()
    if layout == "expanded":
        odd = bias = bias[:1].expand(B, H, S, S)
    else:
        shape = (B, S, H, S + 3) if layout == "heads_last" else (B, H, S, S + 3)
        odd = torch.zeros(shape, dtype=bias.dtype, device="cuda")[..., 1:S + 1]
        if layout == "heads_last":
            odd = odd.transpose(1, 2)
        odd.copy_(bias)
    padded = torch.zeros((B, H, S, 64), dtype=bias.dtype, device="cuda")[..., :S]
    padded.copy_(bias)

    def run(b):
        ins = [t.detach().clone().requires_grad_() for t in (q, k, v)]
        b = b.detach().requires_grad_()
        out = flash_attention_fn(*ins, b, True)
        return dict(zip(("dq", "dk", "dv", "dbias"), torch.autograd.grad(out, [*ins, b], do)), out=out.detach())

    want, got = run(padded), run(odd)
    for name in want:
        assert torch.equal(want[name], got[name]), name
    compare(want, q, k, v, bias.contiguous(), True, None, do, HF, label=f"{layout} {S}: ")


@pytest.mark.parametrize("M,N,D", [(49, 49, 32), (17, 64, 16), (64, 17, 64), (48, 48, 32), (1, 64, 64), (33, 1, 16)])
@pytest.mark.parametrize("dtype,causal", [(BF, False), (torch.float32, True)])
@pytest.mark.parametrize("layout", ["dense", "pitched", "odd", "heads_last"])
def test_stores_stay_inside_their_tensors(M, N, D, dtype, causal, layout, device_ok):
    """As for the tile kernels: every output lies in a sentinel-filled buffer; after fa_small_fwd and fa_small_bwd all of it has
    been written and nothing around it, the columns between the rows of a pitched gradient included.  "odd": an element
    beyond a pair, with an odd pitch, so that pairs cannot be accessed at once."""
    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    lib = _cabi.load()
    B, H = 2, 3
    q, k, v, bias, do = make_inputs(B, M, N, H, D, BF, "float", 80)
    bias = bias.to(dtype)
    o, lse, delta = (_guarded(s, t) for s, t in (((B, M, H, D), BF), ((B, H, M), torch.float32), ((B, H, M), torch.float32)))
    dq, dk, dv = (_guarded(t.shape, BF) for t in (q, k, v))
    cols = {"dense": N, "pitched": (N + 15) // 8 * 8 + 8, "odd": N + 4 + N % 2 + 1, "heads_last": N}[layout]
    shape = (B, M, H, cols) if layout == "heads_last" else (B, H, M, cols)
    first = 1 if layout == "odd" else 0
    whole, bias_whole = _guarded(shape, dtype), torch.zeros(shape, dtype=dtype, device="cuda")
    cut = [t[..., first:first + N] for t in (whole[0], bias_whole)]
    dbias, b = (t.transpose(1, 2) for t in cut) if layout == "heads_last" else cut
    b.copy_(bias)
    p = fa._params(q, k, v, o[0], lse[0], b, _cabi.FA_BIAS_SAME if dtype == BF else _cabi.FA_BIAS_F32, causal, D ** -0.5)
    for name, t in (("d_o", do), ("dq", dq[0]), ("dk", dk[0]), ("dv", dv[0]), ("dbias", dbias)):
        setattr(p, name, t.data_ptr())
        setattr(p, ("do" if name == "d_o" else name) + "_stride", fa._stride3(t))
    p.delta, p.write_dbias = delta[0].data_ptr(), 1
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _cabi.check(lib.fa_small_fwd(ctypes.byref(p), stream), "fa_small_fwd")
    _cabi.check(lib.fa_small_bwd(ctypes.byref(p), stream), "fa_small_bwd")
    torch.cuda.synchronize()
    for name, (_, raw, payload) in dict(o=o, lse=lse, delta=delta, dq=dq, dk=dk, dv=dv).items():
        assert _guards_intact(raw, payload), f"{name}: a store landed outside the tensor"
        assert not bool(torch.any(raw[payload] == (SENT16 if raw.dtype == torch.int16 else SENT32))), f"{name}: never written"
    assert _guards_intact(whole[1], whole[2]), "dbias: a store landed outside the buffer"
    sent = SENT16 if dtype == BF else SENT32
    words = whole[1][whole[2]].view(shape)
    assert bool(torch.all(words[..., :first] == sent)) and bool(torch.all(words[..., first + N:] == sent)), "dbias: between rows"
    assert not bool(torch.any(words[..., first:first + N] == sent)), "dbias: never written"
    ours = {"out": o[0], "dq": dq[0], "dk": dk[0], "dv": dv[0], "dbias": dbias}
    compare(ours, q, k, v, bias, causal, None, do, BF, label=f"{M}x{N} D{D} {layout}: ")


def test_masked_rows_and_nan(device_ok):
    """A row without a key gives zeros and zero gradients; a NaN score makes its row NaN."""
    q, k, v, bias, do = make_inputs(2, 40, 50, 2, 32, BF, "bool", 5)
    bias[0, 1, 7] = False
    ours = run_ours(q, k, v, bias, False, None, do)
    assert not ours["out"][0, 7, 1].any() and not ours["dq"][0, 7, 1].any()
    assert all(torch.isfinite(t).all() for t in ours.values())
    q[1, 3, 0, 0] = float("nan")
    ours = run_ours(q, k, v, None, False, None, do)
    assert torch.isnan(ours["out"][1, 3, 0]).all() and torch.isfinite(ours["out"][1, 4]).all()


def test_c_entries_refuse_what_the_tile_kernels_refuse(device_ok):
    from triton_flashattn_b200 import _cabi

    lib = _cabi.load()
    q, k, v, bias, _ = make_inputs(1, 49, 49, 2, 32, BF, "float", 3)
    o, lse = torch.empty_like(q), torch.empty(1, 2, 49, device="cuda")
    p = _cabi.FaParams()
    p.struct_size = ctypes.sizeof(_cabi.FaParams)
    p.B, p.H, p.M, p.N, p.D, p.dtype, p.bias_kind, p.sm_scale = 1, 2, 49, 49, 32, 1, 1, 0.2
    for name, t in (("q", q), ("k", k), ("v", v), ("o", o)):
        setattr(p, name, t.data_ptr())
        st = t.stride()
        setattr(p, name + "_stride", _cabi._I64x3(st[0], st[1], st[2]))
    p.lse, p.bias = lse.data_ptr(), bias.data_ptr()
    st = bias.stride()
    p.bias_stride = _cabi._I64x3(st[0], st[1], st[2])
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.fa_fwd(ctypes.byref(p), stream) == 5  # rows of 98 bytes
    assert lib.fa_small_fwd(ctypes.byref(p), stream) == 0
    p.M = 65
    assert lib.fa_small_takes(65, 49, 32) == 0 and lib.fa_small_fwd(ctypes.byref(p), stream) == 8
    torch.cuda.synchronize()


def test_a_converted_bias_is_kept_for_the_backward(device_ok):
    """A bias of another dtype is converted once: between forward and backward its fp32 copy stays, beside the result and the
    log-sum-exp, also where its rows (49 columns) are not 16-byte aligned."""
    from triton_flashattn_b200 import flash_attention_fn

    B, S, H, D = 16, 49, 4, 32
    q, k, v, bias, do = make_inputs(B, S, S, H, D, HF, "float", 78)
    bias = bias.to(BF)
    inputs = [t.requires_grad_() for t in (q, k, v)]
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    out = flash_attention_fn(*inputs, bias)
    held = torch.cuda.memory_allocated() - before
    assert held >= out.numel() * 2 + B * H * S * 4 + bias.numel() * 4
    want = torch.autograd.grad(flash_attention_fn(*inputs, bias.float()), inputs, do)
    for a, b in zip(torch.autograd.grad(out, inputs, do), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("S", [48, 49])
@pytest.mark.parametrize("kind", [None, "float", "bool", "f32"])
def test_the_reference_classes_take_the_same_kernels(S, kind, device_ok):
    """FlashAttentionFn and FlashAttentionQKVPackedFn give the bits of the functions, with as many launches, and ask for no scratch that these kernels do not use."""
    from triton_flashattn_b200 import _cabi, flash_attention as fa

    lib = _cabi.load()
    q, k, v, bias, do = make_inputs(3, S, S, 4, 32, HF, "float" if kind == "f32" else kind, 79)
    if kind == "f32":
        bias = bias.float()
    train = kind in ("float", "f32")

    def grads(fn, *tensors):
        ins = [t.detach().clone().requires_grad_() for t in tensors]
        b = bias.detach().clone().requires_grad_(train) if kind else None
        n = lib.fa_launch_count()
        out = fn(*ins, b, True)
        return [out.detach(), *torch.autograd.grad(out, ins + ([b] if train else []), do)], lib.fa_launch_count() - n

    want, n = grads(fa.flash_attention_fn, q, k, v)
    got, m = grads(lambda *a: fa.FlashAttentionFn.apply(*a), q, k, v)
    assert n == m == 2 and all(torch.equal(a, b) for a, b in zip(want, got))
    qkv = torch.stack([q, k, v], dim=2)
    got, m = grads(lambda *a: fa.FlashAttentionQKVPackedFn.apply(*a), qkv)
    packed = torch.stack(want[1:4], dim=2)
    assert m == 2 and torch.equal(got[0], want[0]) and torch.equal(got[1], packed)
    if train:
        assert torch.equal(got[2], want[4])
        if kind == "f32":
            b, bias_kind = fa._classify_bias(bias, q)
            p = fa._params(q, k, v, want[0], want[0], b, bias_kind, True, 0.1)
            assert lib.fa_bwd_workspace_bytes(ctypes.byref(p)) == S * ((S + 7) // 8 * 8) * 2


@pytest.mark.parametrize("B,H", [(1, 2), (3, 64)])
@pytest.mark.parametrize("M,N,D,kind,causal,dtype", [
    (65, 65, 64, "float", False, HF), (128, 128, 64, "float", True, BF), (129, 100, 32, "f32", True, HF), (256, 128, 64, "bool", False, BF),
    (1, 128, 64, None, False, BF), (20, 65, 64, "float", True, BF), (200, 1, 64, None, True, HF), (72, 72, 16, "float", False, HF),
    (255, 127, 32, "bool", True, HF), (128, 120, 64, "f32", False, BF), (130, 128, 64, None, True, BF)])
def test_one_launch_backward_equals_the_stages(M, N, D, kind, causal, dtype, B, H, device_ok):
    """One tile of keys: fa_bwd runs everything in one kernel, the three stage entries do it one by one; the same bits,
    delta among them."""
    assert one_launch_equals_the_stages(M, N, D, kind, causal, dtype, B, H) == (1, 3)  # up to two heads a CTA


@pytest.mark.parametrize("cap", [1, 3])
@pytest.mark.parametrize("M,N,D", [(256, 128, 64), (256, 65, 64), (131, 128, 32), (77, 65, 64)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("trained", [False, True])
def test_one_launch_backward_over_many_tiles(M, N, D, causal, trained, cap, device_ok, monkeypatch):
    """With an fp32 bias a CTA of the one-launch kernel walks any number of heads (here 7 or 20): rings, columns and rows
    asked for ahead of a tile go round many times."""
    monkeypatch.setenv("FA_MAX_CTAS", str(cap))
    launches = one_launch_equals_the_stages(M, N, D, "f32", causal, BF, 5, 4, trained)
    assert launches == (1, 3)


def one_launch_equals_the_stages(M, N, D, kind, causal, dtype, B, H, trained=True):
    from tests.test_robustness_gpu import _bwd_params
    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    lib = _cabi.load()
    g = torch.Generator(device="cuda").manual_seed(M * 1000 + N)
    q, k, v, do = (torch.randn(B, s, H, D, generator=g, device="cuda", dtype=torch.float32).to(dtype) for s in (M, N, N, M))
    bias = None
    if kind == "bool":
        bias = torch.rand(B, H, M, N, generator=g, device="cuda") < 0.9
    elif kind is not None:
        bias = torch.randn(B, H, M, N, generator=g, device="cuda", dtype=torch.float32).to(torch.float32 if kind == "f32" else dtype)
    o, lse = fa._flash_attn_fwd(q, k, v, bias, causal, D ** -0.5)

    def run(stages):
        outs = [torch.full_like(t, 7.0) for t in (q, k, v)]
        delta = torch.full_like(lse, 7.0)
        dbias = fa._new_dbias(bias, q, causal) if trained and kind in ("float", "f32") else None
        p, keep = _bwd_params(fa, q, k, v, o, lse, bias, causal, D ** -0.5, do, *outs, dbias, delta)
        ds16 = torch.empty(B, H, M, (N + 7) // 8 * 8, dtype=dtype, device="cuda")
        if kind == "f32":
            p.ds16, p.ds16_stride = ds16.data_ptr(), _cabi._I64x3(*ds16.stride()[:3])
        before = lib.fa_launch_count()
        for f in stages:
            assert f(ctypes.byref(p), None) == 0
        torch.cuda.synchronize()
        return outs + [delta] + ([dbias] if dbias is not None else []), lib.fa_launch_count() - before

    one, n_one = run([lib.fa_bwd])
    stages, n_stages = run([lib.fa_bwd_pre, lib.fa_bwd_dkdv, lib.fa_bwd_dq])
    ws = torch.empty(B * H * M * ((N + 7) // 8 * 8) * 2 if kind == "f32" else 16, dtype=torch.uint8, device="cuda")
    beside, n_beside = run([lambda p, stream: lib.fa_bwd_workspace(p, ws.data_ptr(), ws.numel(), stream)])  # dS is stored nowhere
    assert n_beside == n_one
    for a, b, c, name in zip(one, stages, beside, ("dq", "dk", "dv", "delta", "dbias")):
        assert torch.equal(a, b) and torch.equal(a, c), name
    return n_one, n_stages


def test_one_launch_backward_takes_and_refuses_what_the_stages_do(device_ok):
    """An fp32 gradient whose stride over a batch of one is zero is taken; a ds16 off its alignment is refused by fa_bwd and
    ignored beside a workspace; a dq, o or do off 16 bytes is refused."""
    from tests.test_robustness_gpu import _bwd_params
    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    lib = _cabi.load()
    q, k, v, bias, do = make_inputs(1, 100, 96, 2, 64, BF, "float", 70)
    bias = bias.float()
    o, lse = fa._flash_attn_fwd(q, k, v, bias, False, 0.1)
    outs = [torch.empty_like(t) for t in (q, k, v)]
    delta, dbias = torch.empty_like(lse), torch.full_like(bias, 7.0)
    ds16 = torch.empty(1, 2, 100, 96, dtype=BF, device="cuda")
    ws = torch.empty(2 * 100 * 96 * 2, dtype=torch.uint8, device="cuda")

    def params():
        p, keep = _bwd_params(fa, q, k, v, o, lse, bias, False, 0.1, do, *outs, dbias, delta)
        p.ds16, p.ds16_stride = ds16.data_ptr(), _cabi._I64x3(*ds16.stride()[:3])
        return p, keep

    p, keep = params()
    p.dbias_stride[0] = 0
    assert lib.fa_bwd(ctypes.byref(p), None) == 0
    torch.cuda.synchronize()
    got = dbias.clone()
    dbias.fill_(7.0)
    p, keep = params()
    for f in (lib.fa_bwd_pre, lib.fa_bwd_dkdv, lib.fa_bwd_dq):
        assert f(ctypes.byref(p), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(got, dbias)
    p.ds16 = ds16.data_ptr() + 2
    assert lib.fa_bwd(ctypes.byref(p), None) == 5  # FA_ERR_ALIGN
    assert lib.fa_bwd_workspace(ctypes.byref(p), ws.data_ptr(), ws.numel(), None) == 0
    torch.cuda.synchronize()
    for name in ("dq", "dk", "dv", "o", "d_o"):
        p, keep = params()
        setattr(p, name, getattr(p, name) + 2)
        assert lib.fa_bwd(ctypes.byref(p), None) == 5, name


@pytest.mark.parametrize("M,N,D", [(65, 65, 64), (128, 100, 32), (256, 128, 64), (129, 1, 16), (200, 127, 64)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B", [1, 60])
def test_one_launch_backward_leaves_ds_where_it_is_told_to(M, N, D, causal, B, device_ok):
    """fa_bwd with an fp32 bias leaves dS rounded to 16 bits in ds16, trained bias or not, and nothing behind the 16-byte
    unit in which a row ends; fa_bwd_workspace does not touch ds16."""
    ds16_is_left(M, N, D, causal, B)


def ds16_is_left(M, N, D, causal, B):
    from tests.test_robustness_gpu import _bwd_params
    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    lib, H = _cabi.load(), 3
    q, k, v, bias, do = make_inputs(B, M, N, H, D, HF, "float", 72)
    bias = bias.float()
    o, lse = fa._flash_attn_fwd(q, k, v, bias, causal, 0.2)
    pitch = (N + 7) // 8 * 8 + 8

    def run(entry, train):
        outs, delta = [torch.empty_like(t) for t in (q, k, v)], torch.empty_like(lse)
        dbias = fa._new_dbias(bias, q, causal) if train else None
        ds16 = torch.full((B, H, M, pitch), 7.0, dtype=HF, device="cuda")
        p, keep = _bwd_params(fa, q, k, v, o, lse, bias, causal, 0.2, do, *outs, dbias, delta)
        p.ds16, p.ds16_stride = ds16.data_ptr(), fa._stride3(ds16)
        assert entry(ctypes.byref(p)) == 0
        torch.cuda.synchronize()
        return outs, dbias, ds16

    ws = torch.empty(B * H * M * pitch * 2, dtype=torch.uint8, device="cuda")
    outs, dbias, ds16 = run(lambda p: lib.fa_bwd(p, None), True)
    visible = torch.ones(M, N, dtype=torch.bool, device="cuda")
    visible = visible.tril() if causal else visible  # above the diagonal it may hold anything
    assert torch.equal(ds16[..., :N][..., visible], dbias[..., :N].to(HF)[..., visible])
    assert (ds16[..., (N + 7) // 8 * 8:] == 7).all()
    outs2, _, untrained = run(lambda p: lib.fa_bwd(p, None), False)
    assert torch.equal(untrained, ds16) and all(torch.equal(a, b) for a, b in zip(outs, outs2))
    others = [lambda p: lib.fa_bwd_workspace(p, ws.data_ptr(), ws.numel(), None)]
    if lib.fa_small_takes(M, N, D):
        others.append(lambda p: lib.fa_small_bwd(p, None))
    for entry in others:
        outs2, _, untouched = run(entry, False)
        assert (untouched == 7).all() and all(torch.equal(a, b) for a, b in zip(outs, outs2))


@pytest.mark.parametrize("M,N,D", [(64, 64, 64), (49, 49, 32), (1, 17, 16), (40, 33, 64), (33, 1, 16)])
@pytest.mark.parametrize("causal", [False, True])
def test_short_backward_leaves_ds_where_it_is_told_to(M, N, D, causal, device_ok):
    """The same for the kernels for short sequences, whose own entry does not touch ds16 either."""
    ds16_is_left(M, N, D, causal, 2)
