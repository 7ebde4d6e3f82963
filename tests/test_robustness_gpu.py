"""GPU tests of what surrounds the arithmetic: the failure path of the bounded waits, stores
staying inside the tensors they belong to, and back-to-back calls without synchronisation.
Nothing here hangs, traps or faults a GPU: the one provoked failure is a wait with a short
limit on a barrier that nothing completes, after which the kernel returns normally."""
import ctypes

import pytest
import torch

from oracle import eager_oracle as oracle
from tests._util import accept, account, make_inputs, run_ours

pytestmark = pytest.mark.gpu

BF, HF = torch.bfloat16, torch.float16


def _bwd_params(fa, q, k, v, o, lse, bias, causal, scale, do, dq, dk, dv, dbias, delta):
    bias_t, kind = fa._classify_bias(bias, q)
    p = fa._params(q, k, v, o, lse, bias_t, kind, causal, scale)
    p.d_o, p.do_stride = do.data_ptr(), fa._stride3(do)
    p.dq, p.dq_stride = dq.data_ptr(), fa._stride3(dq)
    p.dk, p.dk_stride = dk.data_ptr(), fa._stride3(dk)
    p.dv, p.dv_stride = dv.data_ptr(), fa._stride3(dv)
    p.delta = delta.data_ptr() if delta is not None else None
    if dbias is not None:
        p.write_dbias = 1
        p.dbias, p.dbias_stride = dbias.data_ptr(), fa._stride3(dbias)
    return p, bias_t


def test_abandoned_wait_is_reported_and_service_resumes_after_reset():
    """A wait that runs out (1 ms limit, barrier nobody arms): the kernel returns, the status
    word names kernel and site, the host copy lets the next API call raise without a
    synchronisation, kernels launched meanwhile do no work, and a reset restores service."""
    from triton_flashattn_b200 import _cabi, flash_attention_fn

    lib = _cabi.load()
    words = _cabi.health_words(0)
    assert words[0] == 0
    q, k, v, _, _ = make_inputs(1, 128, 128, 1, 64, HF, None, 40)
    good = flash_attention_fn(q, k, v)
    torch.cuda.synchronize()
    try:
        _cabi.check(lib.fa_selftest_wait_timeout(0, 1000, None), "fa_selftest_wait_timeout")
        torch.cuda.synchronize()  # the kernel came back by itself
        st = _cabi.device_status(0)
        assert st[:6] == [1, 101, 0, 0, 7, 1000], st
        assert list(words[:6]) == st[:6]  # host copy, written by the kernel
        out32 = (ctypes.c_int32 * 8)()
        assert lib.fa_last_device_status(0, out32) == 7  # FA_ERR_DEVICE_WAIT
        # the public API refuses to hand out tensors nobody computed
        with pytest.raises(RuntimeError, match="abandoned a bounded wait"):
            flash_attention_fn(q, k, v)
        # through the C ABI a launch is still accepted, and documented to do no work
        from triton_flashattn_b200 import flash_attention as fa
        o = torch.full_like(q, 7.0)
        lse = torch.full((1, 1, 128), 7.0, device="cuda")
        p = fa._params(q, k, v, o, lse, None, _cabi.FA_BIAS_NONE, False, 0.125)
        assert lib.fa_fwd(ctypes.byref(p), None) == 0
        torch.cuda.synchronize()
        assert torch.all(o == 7.0) and torch.all(lse == 7.0)
    finally:
        _cabi.reset_device_status(0)
    assert _cabi.device_status(0)[0] == 0 and words[0] == 0
    again = flash_attention_fn(q, k, v)
    torch.cuda.synchronize()
    assert torch.equal(again, good)


SENT16 = 0x7B7B  # bit pattern written around every output (a large finite 16-bit float)
SENT32 = 0x7B7B7B7B


def _guarded(shape, dtype, pad_elems=4096):
    """A tensor of `shape` carved out of the middle of a sentinel-filled buffer; returns
    (view, whole buffer as int16/int32 words, slice of the payload)."""
    n = 1
    for s in shape:
        n *= s
    buf = torch.empty(n + 2 * pad_elems, dtype=dtype, device="cuda")
    raw = buf.view(torch.int16 if dtype.itemsize == 2 else torch.int32)
    raw.fill_(SENT16 if dtype.itemsize == 2 else SENT32)
    return buf[pad_elems:pad_elems + n].view(shape), raw, slice(pad_elems, pad_elems + n)


def _guards_intact(raw, payload):
    sent = SENT16 if raw.dtype == torch.int16 else SENT32
    return bool(torch.all(raw[:payload.start] == sent)) and bool(torch.all(raw[payload.stop:] == sent))


@pytest.mark.parametrize("M,N,D,causal,bias_kind", [(200, 136, 64, False, "float"), (300, 100, 128, True, "float"),
                                                    (129, 1, 64, False, "float"), (100, 300, 32, True, "bool"),
                                                    (384, 384, 128, True, "float"), (50, 70, 16, False, None)])
def test_stores_stay_inside_their_tensors(M, N, D, causal, bias_kind, device_ok):
    """o, lse, delta, dq, dk, dv and dbias are carved out of sentinel-filled buffers; after a
    forward and a backward through the C ABI the sentinels around them, and the pad columns of
    the dbias rows, are untouched and every payload element has been written."""
    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    lib = _cabi.load()
    B, H = 2, 2
    q, k, v, bias, do = make_inputs(B, M, N, H, D, BF, bias_kind, 50)
    scale = D ** -0.5
    o, o_raw, o_pl = _guarded((B, M, H, D), BF)
    lse, lse_raw, lse_pl = _guarded((B, H, M), torch.float32)
    delta, delta_raw, delta_pl = _guarded((B, H, M), torch.float32)
    dq, dq_raw, dq_pl = _guarded((B, M, H, D), BF)
    dk, dk_raw, dk_pl = _guarded((B, N, H, D), BF)
    dv, dv_raw, dv_pl = _guarded((B, N, H, D), BF)
    dbias = dbias_full = None
    if bias_kind == "float":
        n_pad = (N + 7) // 8 * 8 + 8  # always at least 8 pad columns per row
        dbias_full, db_raw, db_pl = _guarded((B, H, M, n_pad), BF)
        dbias = dbias_full[..., :N]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    p, keep = _bwd_params(fa, q, k, v, o, lse, bias, causal, scale, do, dq, dk, dv, dbias, delta)
    _cabi.check(lib.fa_fwd(ctypes.byref(p), stream), "fa_fwd")
    _cabi.check(lib.fa_bwd(ctypes.byref(p), stream), "fa_bwd")
    torch.cuda.synchronize()
    for name, raw, pl in (("o", o_raw, o_pl), ("lse", lse_raw, lse_pl), ("delta", delta_raw, delta_pl),
                          ("dq", dq_raw, dq_pl), ("dk", dk_raw, dk_pl), ("dv", dv_raw, dv_pl)):
        assert _guards_intact(raw, pl), f"{name}: a store landed outside the tensor"
        sent = SENT16 if raw.dtype == torch.int16 else SENT32
        assert not bool(torch.any(raw[pl] == sent)), f"{name}: an element was never written"
    if dbias is not None:
        assert _guards_intact(db_raw, db_pl), "dbias: a store landed outside the buffer"
        # A bulk tensor store is clipped at the tensor's extent N, but the hardware writes whole
        # 16-byte units: the bytes between element N and the next 16-byte boundary of a row may
        # be overwritten (with the zeros dS holds for keys >= N).  That is why a dbias row pitch
        # must be a multiple of 16 bytes.  Everything from that boundary on must be untouched.
        n16 = (N + 7) // 8 * 8
        tail = dbias_full[..., N:n16].contiguous().view(torch.int16)
        touched = int((tail != SENT16).sum().item())
        print(f"dbias N={N}: {touched} of {tail.numel()} elements between N and the 16-byte boundary were written",
              flush=True)
        # (+0 or -0: dS of a masked key is 0 * (dP - delta))
        assert bool(torch.all((tail == SENT16) | ((tail & 0x7FFF) == 0))), \
            "dbias: garbage between N and the 16-byte boundary"
        pads = dbias_full[..., n16:].contiguous().view(torch.int16)
        assert bool(torch.all(pads == SENT16)), "dbias: a store landed in the pad columns of a row"
        assert not bool(torch.any(dbias.contiguous().view(torch.int16) == SENT16)), "dbias: unwritten element"


@pytest.mark.parametrize("static_scratch", [False, True])
def test_back_to_back_steps_without_sync(static_scratch, device_ok):
    """Two different problems of the same shape enqueued one after the other on one stream with
    no synchronisation in between, re-using the very same scratch and output addresses (every
    kernel may start while its predecessor still runs).  The second step's results must be
    bitwise what that problem gives when run alone."""
    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    lib = _cabi.load()
    entry = lib.fa_bwd_static_scratch if static_scratch else lib.fa_bwd
    B, M, N, H, D, causal = 2, 640, 512, 4, 128, True
    scale = D ** -0.5
    X = make_inputs(B, M, N, H, D, BF, "float", 60)
    Y = make_inputs(B, M, N, H, D, BF, "float", 61)
    o, lse = torch.empty_like(X[0]), torch.empty((B, H, M), device="cuda", dtype=torch.float32)
    delta = torch.empty_like(lse)
    dq, dk, dv = torch.empty_like(X[0]), torch.empty_like(X[1]), torch.empty_like(X[2])
    dbias = fa._empty_dbias(X[3], BF)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def enqueue(inp):
        q, k, v, bias, do = inp
        p, keep = _bwd_params(fa, q, k, v, o, lse, bias, causal, scale, do, dq, dk, dv, dbias,
                              None if static_scratch else delta)
        _cabi.check(lib.fa_fwd(ctypes.byref(p), stream), "fa_fwd")
        _cabi.check(entry(ctypes.byref(p), stream), "backward")

    def snapshot():
        torch.cuda.synchronize()
        return [t.clone() for t in (o, lse, dq, dk, dv, dbias)]

    enqueue(Y)
    alone = snapshot()
    enqueue(X)
    enqueue(Y)  # no synchronisation between the two steps
    after = snapshot()
    for name, a, b in zip(("o", "lse", "dq", "dk", "dv", "dbias"), alone, after):
        assert torch.equal(a, b), f"{name} of the second step differs from the same step run alone"


@pytest.mark.parametrize("expanded", [False, True])
@pytest.mark.parametrize("D,M,N,causal,bias_kind", [(64, 300, 200, True, None), (128, 260, 390, False, "bool"),
                                                    (128, 200, 77, True, "float"), (64, 130, 260, False, "float"),
                                                    (256, 200, 136, True, None), (256, 130, 200, False, "bool")])
def test_backward_through_slabs_of_any_size(D, M, N, causal, bias_kind, expanded, device_ok):
    """fa_bwd_workspace with room for 1, 2, 4 and all of 6 problems in two batch elements (so with parts that cross
    from one to the other and a last part that is smaller), the bias another one per batch element or one for both:
    dq, dk, dv are those of fa_bwd bit for bit - the recomputing dQ kernel forms dS in the same order - and right.
    Nothing is written behind the workspace."""
    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    lib = _cabi.load()
    B, H, scale = 2, 3, D ** -0.5
    q, k, v, bias, do = make_inputs(B, M, N, H, D, BF, bias_kind, 60)
    if expanded and bias is None:
        pytest.skip("no bias to expand")
    if expanded:
        bias = bias[:1].expand(B, H, M, N)
    o, lse = fa._flash_attn_fwd(q, k, v, bias, causal, scale)
    delta = torch.empty_like(lse)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    one = M * ((N + 7) // 8 * 8) * 2
    results = []
    for room in (0, 1, 2, 4, 6):
        dq, dk, dv = (torch.full_like(t, 7.0) for t in (q, k, v))
        p, keep = _bwd_params(fa, q, k, v, o, lse, bias, causal, scale, do, dq, dk, dv, None, delta)
        assert lib.fa_bwd_workspace_bytes(ctypes.byref(p)) == 6 * one
        if room == 0 and D == 256:  # without slabs this head dim needs the ds16 tensor
            ds16 = torch.empty(B, H, M, (N + 7) // 8 * 8, dtype=BF, device="cuda")[..., :N]
            p.ds16, p.ds16_stride = ds16.data_ptr(), fa._stride3(ds16)
        ws, raw, payload = _guarded((room * one // 2 if room else 8,), BF)
        rc = lib.fa_bwd_workspace(ctypes.byref(p), ws.data_ptr(), room * one, stream)
        _cabi.check(rc, "fa_bwd_workspace")
        torch.cuda.synchronize()
        assert _guards_intact(raw, payload), room
        results.append((dq, dk, dv))
    for room, grads in zip((1, 2, 4, 6), results[1:]):
        for name, a, b in zip(("dq", "dk", "dv"), grads, results[0]):
            assert torch.equal(a, b), f"{name} with room for {room} problems"
    ref = oracle.attention_backward(q, k, v, bias, causal, scale, do, o_saved=o)
    for name, t in zip(("dq", "dk", "dv"), results[2]):
        accept(name, account(t, ref[name], BF), BF, label=f"D{D} M{M} N{N} {bias_kind}: ")


@pytest.mark.parametrize("which", ["q", "v", "bias", "qkv"])
def test_forward_mode_is_refused(which, device_ok):
    """No forward-mode rule exists: a dual tensor raises instead of losing its tangent."""
    import torch.autograd.forward_ad as fwad
    from triton_flashattn_b200 import flash_attention_fn, flash_attention_qkvpacked_fn

    x = {n: torch.randn(1, 64, 2, 64, dtype=torch.float16, device="cuda") for n in ("q", "k", "v")}
    x["bias"] = torch.randn(1, 2, 64, 64, dtype=torch.float16, device="cuda")
    qkv = torch.stack([x["q"], x["k"], x["v"]], dim=2)
    with fwad.dual_level(), pytest.raises(NotImplementedError, match="jvp"):
        if which == "qkv":
            flash_attention_qkvpacked_fn(fwad.make_dual(qkv, torch.ones_like(qkv)))
        else:
            x[which] = fwad.make_dual(x[which], torch.ones_like(x[which]))
            flash_attention_fn(x["q"], x["k"], x["v"], x["bias"])
    assert flash_attention_fn(x["q"], x["k"], x["v"]).shape == (1, 64, 2, 64)  # outside the level: as ever


@pytest.mark.parametrize("use", ["offload", "checkpoint"])
def test_nothing_bypasses_saved_tensor_hooks(use, device_ok):
    """A padding mask over 777 keys is copied into padded rows for the kernels; with hooks that take the saved
    tensors away, or under checkpointing, no such copy stays on the device between forward and backward."""
    from torch.utils.checkpoint import checkpoint
    from triton_flashattn_b200 import flash_attention_fn

    q, k, v, _, do = make_inputs(2, 1000, 777, 4, 64, BF, None, 61)
    lens = torch.tensor([[500], [700]], device="cuda")
    mask = (torch.arange(777, device="cuda")[None] < lens)[:, None, None].expand(2, 4, 1000, 777)
    inputs = [t.requires_grad_() for t in (q, k, v)]
    want = torch.autograd.grad(flash_attention_fn(*inputs, mask), inputs, do)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    if use == "offload":
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.cuda()):
            out = flash_attention_fn(*inputs, mask)
    else:
        out = checkpoint(lambda *a: flash_attention_fn(*a), *inputs, mask, use_reentrant=False)
    assert torch.cuda.memory_allocated() - before == out.numel() * 2
    got = torch.autograd.grad(out, inputs, do)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("packed", [False, True])
def test_no_upstream_gradient_counts_as_zeros(packed, device_ok):
    """A function behind the attention that returns None for its gradient: every input gets zeros, not None."""
    from triton_flashattn_b200 import flash_attention_fn, flash_attention_qkvpacked_fn

    class Stop(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            return x.clone()

        @staticmethod
        def backward(ctx, grad):
            return None

    q, k, v, bias, _ = make_inputs(2, 96, 96, 2, 64, BF, "float", 62)
    inputs = [torch.stack([q, k, v], dim=2), bias] if packed else [q, k, v, bias]
    for t in inputs:
        t.requires_grad_()
    Stop.apply((flash_attention_qkvpacked_fn if packed else flash_attention_fn)(*inputs)).sum().backward()
    for t in inputs:
        assert t.grad is not None and t.grad.shape == t.shape and not t.grad.any()


@pytest.mark.parametrize("kind", ["float", "0-d tensor", "tensor on the device", "text"])
def test_scale_is_whatever_float_takes(kind, device_ok):
    from triton_flashattn_b200 import flash_attention_fn

    q, k, v, _, _ = make_inputs(1, 40, 40, 2, 64, BF, None, 63)
    scale = {"float": 0.25, "0-d tensor": torch.tensor(0.25), "tensor on the device": torch.tensor(0.25, device="cuda"),
             "text": "0.25"}[kind]
    assert torch.equal(flash_attention_fn(q, k, v, None, False, scale), flash_attention_fn(q, k, v, None, False, 0.25))
    with pytest.raises(TypeError):
        flash_attention_fn(q, k, v, None, False, [0.25])
    with pytest.raises(ValueError):
        flash_attention_fn(q, k, v, None, False, "a quarter")


@pytest.mark.parametrize("M", [1, 16, 17])
def test_zero_strides_are_refused_by_every_kernel(M, device_ok):
    """A stride of zero over B, S or H of q, k, v (or do) is an alignment error, whichever kernel a call goes to.
    (All strides stay inside the tensors: a refusal that failed to come would read in bounds.)"""
    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    lib = _cabi.load()
    B, N, H, D = 2, 64, 2, 64
    q, k, v, bias, do = make_inputs(B, M, N, H, D, BF, "float", 64)
    o, lse = fa._flash_attn_fwd(q, k, v, bias, False, 0.1)
    dq, dk, dv = (torch.empty_like(t) for t in (q, k, v))
    dbias, delta = torch.zeros_like(bias), torch.empty_like(lse)
    for which in ("q", "k", "v", "do"):
        for i in range(3):
            p, keep = _bwd_params(fa, q, k, v, o, lse, bias, False, 0.1, do, dq, dk, dv, dbias, delta)
            st = list(getattr(p, which + "_stride"))
            st[i] = 0
            setattr(p, which + "_stride", _cabi._I64x3(*st))
            if which != "do":
                assert lib.fa_fwd(ctypes.byref(p), None) == 5, (which, i)  # FA_ERR_ALIGN
                assert lib.fa_small_fwd(ctypes.byref(p), None) == 5, (which, i)
            assert lib.fa_bwd_dkdv(ctypes.byref(p), None) == 5, (which, i)
            assert lib.fa_bwd_dq(ctypes.byref(p), None) == 5, (which, i)
            assert lib.fa_bwd(ctypes.byref(p), None) == 5 and lib.fa_small_bwd(ctypes.byref(p), None) == 5, (which, i)
    p, keep = _bwd_params(fa, q, k, v, o, lse, bias, False, 0.1, do, dq, dk, dv, dbias, delta)
    assert lib.fa_fwd(ctypes.byref(p), None) == 0 and lib.fa_bwd(ctypes.byref(p), None) == 0
    torch.cuda.synchronize()


@pytest.mark.parametrize("D,bias_kind,causal", [(128, "float", False), (128, "float", True), (64, "float", False),
                                                (128, "f32", False), (128, "bool", True), (256, "float", False)])
def test_full_size_forwards_repeat_bitwise(D, bias_kind, causal, device_ok):
    """Forty forwards of a problem that keeps every bias ring turning for several units give the same bits: a bias
    unit handed back before all its rows are read shows as a few wrong rows in about one pass in ten."""
    from triton_flashattn_b200 import flash_attention as fa

    B, S, H = 8, 2048, 16 if bias_kind != "f32" else 8
    g = torch.Generator(device="cuda").manual_seed(65)
    q, k, v = (torch.randn(B, S, H, D, generator=g, device="cuda", dtype=torch.float32).to(BF) for _ in range(3))
    if bias_kind == "bool":
        bias = torch.rand(B, H, S, S, generator=g, device="cuda") < 0.9
    else:
        bias = torch.randn(B, H, S, S, generator=g, device="cuda", dtype=torch.float32 if bias_kind == "f32" else BF)
    first, lse = fa._flash_attn_fwd(q, k, v, bias, causal, D ** -0.5)
    differing = 0
    for _ in range(40):
        out, lse2 = fa._flash_attn_fwd(q, k, v, bias, causal, D ** -0.5)
        differing += not (torch.equal(out, first) and torch.equal(lse, lse2))
    assert differing == 0, f"{differing} of 40 passes differ"


@pytest.mark.parametrize("D,bias_kind", [(256, "16bit"), (256, "none"), (256, "bool"), (128, "16bit"), (128, "none"), (64, "f32")])
def test_causal_units_of_every_length_repeat_bitwise(D, bias_kind, device_ok):
    """Units of one key block and longer ones in turn, several a CTA, a hundred passes: every wait ends and the bits stay.
    (An issuer that looked again at the barrier of a ring stage it had already handed back found it a completion further
    about once in some hundred launches and waited for good.)"""
    from triton_flashattn_b200 import flash_attention as fa

    B, S, H = 2, 1000, 40
    g = torch.Generator(device="cuda").manual_seed(66)
    q, k, v = (torch.randn(B, S, H, D, generator=g, device="cuda", dtype=torch.float32).to(BF) for _ in range(3))
    bias = None
    if bias_kind == "bool":
        bias = torch.rand(B, H, S, S, generator=g, device="cuda") < 0.9
    elif bias_kind != "none":
        bias = torch.randn(B, H, S, S, generator=g, device="cuda", dtype=torch.float32 if bias_kind == "f32" else BF)
    first, lse = fa._flash_attn_fwd(q, k, v, bias, True, D ** -0.5)
    differing = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(100):
        out, lse2 = fa._flash_attn_fwd(q, k, v, bias, True, D ** -0.5)
        differing += ((out != first).any() | (lse != lse2).any()).long()
    assert int(differing) == 0, f"{int(differing)} of 100 passes differ"


@pytest.mark.parametrize("D,bias_kind,M,N", [(64, "none", 900, 900), (64, "f32", 1030, 300), (128, "16bit", 1100, 700),
                                             (128, "bool", 520, 1304), (128, "none", 129, 129), (256, "16bit", 500, 500)])
def test_causal_forward_order_does_not_change_bits(D, bias_kind, M, N, device_ok, monkeypatch):
    """Pairs of a heavy and a light unit, or longest first: the number of CTAs decides, each row is the same work."""
    from oracle import eager_oracle as oracle
    from triton_flashattn_b200 import flash_attention as fa

    g = torch.Generator(device="cuda").manual_seed(67)
    q, k, v = (torch.randn(1, s, 5, D, generator=g, device="cuda", dtype=torch.float32).to(BF) for s in (M, N, N))
    bias = None
    if bias_kind == "bool":
        bias = torch.rand(1, 5, M, N, generator=g, device="cuda") < 0.9
    elif bias_kind != "none":
        bias = torch.randn(1, 5, M, N, generator=g, device="cuda", dtype=torch.float32 if bias_kind == "f32" else BF)
    first, lse = fa._flash_attn_fwd(q, k, v, bias, True, D ** -0.5)
    ref = oracle.attention_forward(q, k, v, bias, True, D ** -0.5)[0]
    seen = ref.abs().sum(-1, keepdim=True) > 0  # rows with no key at all are zeros here
    assert ((first.float() - ref.float()) * seen).abs().max() <= 2e-2 + 2 ** -7 * ref.abs().max()
    for cap in (1, 2, 3, 7, 11, 16, 19):
        monkeypatch.setenv("FA_MAX_CTAS", str(cap))
        out, lse2 = fa._flash_attn_fwd(q, k, v, bias, True, D ** -0.5)
        assert torch.equal(out, first) and torch.equal(lse, lse2), cap


@pytest.mark.parametrize("D,M,N", [(64, 130, 200), (128, 300, 300), (256, 100, 390), (32, 257, 65)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("dtype", [BF, HF])
def test_a_mask_is_a_bias_of_zeros_and_minus_infinity(D, M, N, causal, dtype, device_ok):
    """The forward scales a score before it masks it or adds a bias, so the two give the same bits; also with a row that sees
    no key, and with a scale that is no power of two (so that a scale folded into the exponent would round differently)."""
    from triton_flashattn_b200 import flash_attention as fa

    q, k, v, mask, _ = make_inputs(2, M, N, 3, D, dtype, "bool", 71)
    mask[1, 2, 5] = False
    zeros = torch.zeros(mask.shape, dtype=dtype, device="cuda")
    out, lse = fa._flash_attn_fwd(q, k, v, mask, causal, 0.11)
    want, want_lse = fa._flash_attn_fwd(q, k, v, zeros.masked_fill_(~mask, float("-inf")), causal, 0.11)
    assert torch.equal(out, want) and torch.equal(lse, want_lse)
    assert not out[1, 5, 2].any() and lse[1, 2, 5] == float("inf")


@pytest.mark.parametrize("D,M", [(16, 100), (32, 257), (64, 70), (64, 1), (128, 130), (256, 95)])
@pytest.mark.parametrize("kind", [None, "float", "bool"])
@pytest.mark.parametrize("layout", ["dense", "padded", "reversed batch"])
def test_forward_result_in_any_layout(layout, D, M, kind, device_ok):
    """The result leaves by bulk stores of 32 rows where its layout can be encoded, by plain ones where it cannot, and where a bias
    at head dims 128 and 256 leaves no shared memory for them: the same bits, and nothing beside it is touched.  M up to 16
    goes to the kernel for few rows."""
    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    B, H, N = 2, 3, 150
    g = torch.Generator(device="cuda").manual_seed(68)
    q, k, v = (torch.randn(B, s, H, D, generator=g, device="cuda", dtype=torch.float32).to(BF) for s in (M, N, N))
    bias = None
    if kind is not None:
        bias = torch.randn(B, H, M, N + 10, generator=g, device="cuda", dtype=torch.float32)  # rows of 160
        bias = (bias.to(BF) if kind == "float" else bias > -1)[..., :N]
    want, lse = fa._flash_attn_fwd(q, k, v, bias, False, D ** -0.5)
    pad = 0 if layout == "dense" else 8
    buf = torch.full((B, M + 3, H, D + pad), 7.0, dtype=BF, device="cuda")
    view = buf[:, :M, :, :D]
    lse2 = torch.empty_like(lse)
    b, bias_kind = fa._classify_bias(bias, q)
    p = fa._params(q, k, v, view, lse2, b, bias_kind, False, D ** -0.5)
    if layout == "reversed batch":
        p.o, p.o_stride[0] = view[1].data_ptr(), -view.stride(0)
    lib = _cabi.load()
    assert lib.fa_fwd(ctypes.byref(p), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    got = view.flip(0) if layout == "reversed batch" else view
    assert torch.equal(got, want) and torch.equal(lse, lse2)
    assert (buf[:, M:] == 7).all() and (buf[..., D:] == 7).all()


@pytest.mark.parametrize("M,N,D", [(40, 40, 32), (100, 90, 64), (10, 200, 64), (300, 300, 128), (130, 130, 256)])
def test_first_cuda_call_of_a_thread(M, N, D, device_ok):
    """A thread whose first CUDA call is one of this library's: no context is bound to it yet, which the encoding of tile
    maps wants.  (The autograd engine's thread is one in a program's first backward.)"""
    import threading

    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    lib = _cabi.load()
    q, k, v, bias, do = make_inputs(1, M, N, 2, D, BF, "float", 69)
    o, lse = fa._flash_attn_fwd(q, k, v, bias, False, 0.1)
    dq, dk, dv = (torch.empty_like(t) for t in (q, k, v))
    dbias, delta = fa._new_dbias(bias, q, False), torch.empty_like(lse)
    p, keep = _bwd_params(fa, q, k, v, o, lse, bias, False, 0.1, do, dq, dk, dv, dbias, delta)
    torch.cuda.synchronize()
    for f in (lib.fa_fwd, lib.fa_bwd, lib.fa_bwd_dkdv, lib.fa_bwd_dq):
        got = []
        t = threading.Thread(target=lambda: got.append(f(ctypes.byref(p), None)))
        t.start()
        t.join()
        assert got == [0]
    torch.cuda.synchronize()


def test_a_refused_layout_leaves_the_context_alone(device_ok):
    """A layout that the driver cannot encode (a batch stride of 2^41 bytes; nothing is launched) is refused, and the thread's
    current context stays the one that it was."""
    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    lib, cuda = _cabi.load(), ctypes.CDLL("libcuda.so.1")
    q, k, v, _, _ = make_inputs(2, 100, 100, 2, 64, BF, None, 73)
    o, lse = fa._flash_attn_fwd(q, k, v, None, False, 0.1)
    torch.cuda.synchronize()
    p = fa._params(q, k, v, o, lse, None, 0, False, 0.1)
    p.q_stride[0] = 1 << 40
    before, own, now = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    assert cuda.cuCtxGetCurrent(ctypes.byref(before)) == 0
    assert cuda.cuCtxCreate_v2(ctypes.byref(own), 0, p.device) == 0  # current from here on
    try:
        assert lib.fa_fwd(ctypes.byref(p), None) == 6  # FA_ERR_CUDA
        assert cuda.cuCtxGetCurrent(ctypes.byref(now)) == 0
    finally:
        assert cuda.cuCtxDestroy_v2(own) == 0 and cuda.cuCtxSetCurrent(before) == 0
    assert now.value == own.value


@pytest.mark.parametrize("bias_kind,D", [(0, 64), (2, 128), (0, 256), (3, 128)])
def test_scratch_for_ds_is_bounded(bias_kind, D, device_ok):
    """The scratch a backward asks for: at most 1.5 GiB, and nothing where that holds no problem or too few to fill
    the SMs; only where no other dQ kernel exists (head dim 256, fp32 bias) more, but never more than all of dS."""
    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    lib = _cabi.load()
    t, lse = torch.empty(1, 1, 1, D, dtype=BF, device="cuda"), torch.empty(1, device="cuda")
    p = fa._params(t, t, t, t, lse, t, bias_kind, True, 0.1)
    seen = set()
    for B, H, M, N in ((1, 1, 1, 1), (2, 16, 1000, 777), (4, 32, 4096, 4096), (1, 8, 16384, 16384), (1, 8, 20480, 20480),
                       (1, 8, 27000, 27000), (1, 3, 32768, 32768), (1, 1, 131072, 131072), (8, 1, 17, 1 << 20)):
        p.B, p.H, p.M, p.N = B, H, M, N
        one, got = M * ((N + 7) // 8 * 8) * 2, lib.fa_bwd_workspace_bytes(ctypes.byref(p))
        assert got % one == 0 and got <= one * B * H, (B, H, M, N)
        if D == 256 or bias_kind == 3:
            assert got >= one, (B, H, M, N)
        else:
            assert got <= 3 << 29, (B, H, M, N)
            if one > 3 << 29:
                assert got == 0, (B, H, M, N)
        seen.add(got // one)
    assert len(seen) > 2


def test_a_long_plain_backward_needs_no_quadratic_memory(device_ok):
    from triton_flashattn_b200 import flash_attention_fn

    S = 32768
    q, k, v = (torch.randn(1, S, 1, 64, device="cuda", dtype=BF, requires_grad=True) for _ in range(3))
    out = flash_attention_fn(q, k, v, None, True)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    out.backward(torch.ones_like(out))
    torch.cuda.synchronize()
    assert torch.cuda.max_memory_allocated() - before < 64 << 20  # gradients, do and delta; dS would be 2 GiB


def test_scratch_size_is_cheap_to_ask_for(device_ok):
    """Every backward asks for the scratch size on the host; with tens of thousands of small problems too."""
    import time

    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    lib = _cabi.load()
    t, lse = torch.empty(1, 1, 1, 64, dtype=BF, device="cuda"), torch.empty(1, device="cuda")
    p = fa._params(t, t, t, t, lse, None, 0, True, 0.1)
    for p.B, p.H, p.M, p.N in ((4096, 15, 160, 160), (8192, 7, 180, 180), (1, 65535, 120, 120), (4, 32, 4096, 4096)):
        best = 1.0
        for _ in range(20):
            start = time.perf_counter()
            lib.fa_bwd_workspace_bytes(ctypes.byref(p))
            best = min(best, time.perf_counter() - start)
        assert best < 40e-6, f"B{p.B} H{p.H} M{p.M}: {best * 1e6:.0f} us"


# Caps on the grid at which a causal dK/dV of six problems goes longest first in three or four rows of tiles, in two, and in
# one (a quarter of the tiles a CTA, or more, is the most it takes; one CTA always goes by pairs).
@pytest.mark.parametrize("M,N,caps", [(1024, 1024, (15, 17, 30)), (300, 700, (9, 11, 25)), (700, 300, (6, 7, 10)), (640, 640, (8, 13, 20))])
@pytest.mark.parametrize("D,bias_kind", [(64, None), (64, "float"), (64, "bool"), (64, "f32"), (128, None), (128, "float"),
                                         (128, "bool"), (128, "f32")])
def test_causal_gradients_do_not_depend_on_the_schedule(M, N, caps, D, bias_kind, device_ok, monkeypatch):
    """Few causal key blocks per CTA go longest first, many in pairs of a long and a short one: the same bits, also with key
    blocks that no query sees (M < N) and with several rows of tiles, every second one from the other end."""
    q, k, v, bias, do = make_inputs(2, M, N, 3, D, BF, "float" if bias_kind == "f32" else bias_kind, 71)
    if bias_kind == "f32":
        bias = bias.float()
    monkeypatch.setenv("FA_MAX_CTAS", "1")
    want = run_ours(q, k, v, bias, True, None, do)
    for ctas in (*caps, 7, 148):
        monkeypatch.setenv("FA_MAX_CTAS", str(ctas))
        got = run_ours(q, k, v, bias, True, None, do)
        for name in want:
            assert torch.equal(want[name], got[name]), (name, ctas)


@pytest.mark.parametrize("D,M,N,bias_kind,ctas", [(64, 300, 700, None, 5), (128, 1024, 1024, None, 5), (128, 700, 300, "bool", 2),
                                                  (64, 1024, 1024, "bool", 5)])
def test_longest_first_over_slabs(D, M, N, bias_kind, ctas, device_ok, monkeypatch):
    """The same with dS in slabs, two of six problems at a time (parts that begin behind the first problem), each part
    longest first in three or four rows of tiles: the bits of one CTA that goes by pairs."""
    from triton_flashattn_b200 import _cabi
    from triton_flashattn_b200 import flash_attention as fa

    lib = _cabi.load()
    q, k, v, bias, do = make_inputs(2, M, N, 3, D, BF, bias_kind, 72)
    o, lse = fa._flash_attn_fwd(q, k, v, bias, True, 0.1)
    delta = torch.empty_like(lse)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    one = M * ((N + 7) // 8 * 8) * 2
    ws = torch.empty(2 * one, dtype=torch.uint8, device="cuda")
    results = []
    for cap, room in ((1, 0), (ctas, 2), (1, 2)):
        monkeypatch.setenv("FA_MAX_CTAS", str(cap))
        grads = [torch.full_like(t, 7.0) for t in (q, k, v)]
        p, keep = _bwd_params(fa, q, k, v, o, lse, bias, True, 0.1, do, *grads, None, delta)
        _cabi.check(lib.fa_bwd_workspace(ctypes.byref(p), ws.data_ptr() if room else None, ctypes.c_uint64(room * one), stream), "bwd")
        results.append(grads)
    for grads in results[1:]:
        for name, a, b in zip(("dq", "dk", "dv"), grads, results[0]):
            assert torch.equal(a, b), name
