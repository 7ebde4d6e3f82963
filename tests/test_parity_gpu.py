"""GPU parity: the CUDA path (through the Python API and the C ABI) against the
fp32 oracle on identical seeded inputs.  Tolerances are the ones the target states:
max-abs <= 2e-2 for bf16 and <= 5e-3 for fp16 (tests/_util.py: TOL)."""
import pytest
import torch

from tests._util import TOL, accept, account, check_case, compare, make_inputs, run_ours
from oracle import eager_oracle as oracle

pytestmark = pytest.mark.gpu

BF, HF = torch.bfloat16, torch.float16


def test_umma_selftest(device_ok):
    """Descriptor encodings of every operand arrangement the kernels use."""
    from triton_flashattn_b200 import _cabi

    lib = _cabi.load()
    for dt, code in ((BF, 1), (HF, 0)):
        a = torch.randn(128, 128, device="cuda").to(dt)
        b = torch.randn(128, 128, device="cuda").to(dt)
        af, bf = a.double(), b.double()
        refs = {0: af @ bf.T, 1: af @ bf, 2: af.T @ bf, 3: af @ bf}
        for mode in range(5):
            c = torch.zeros(128, 128, device="cuda", dtype=torch.float32)
            _cabi.check(lib.fa_selftest_umma(mode, code, a.data_ptr(), b.data_ptr(), c.data_ptr(), 0, None),
                        "fa_selftest_umma")
            torch.cuda.synchronize()
            if mode == 4:
                got = c.view(dt)[:64].reshape(128, 128)
                assert torch.equal(got, a)
            else:
                assert (c.double() - refs[mode]).abs().max().item() < 1e-3


def test_config1_fp16_float_bias(device_ok):
    # B=2, M=N=128, H=4, D=64, fp16, trainable float bias, seed 0
    check_case(2, 128, 128, 4, 64, HF, "float", False, seed=0, sm_scale=1 / 8)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [BF, HF])
@pytest.mark.parametrize("bias_kind,causal", [(None, False), (None, True), ("float", False),
                                              ("float", True), ("bool", False), ("bool", True)])
def test_small_grid(D, dtype, bias_kind, causal, device_ok):
    check_case(2, 256, 256, 2, D, dtype, bias_kind, causal, seed=1)


@pytest.mark.parametrize("N", [129, 130, 131, 160, 163, 191, 194, 255, 287])
@pytest.mark.parametrize("kind,D,causal", [("bool", 128, False), ("bool", 128, True), ("f32", 128, False), ("f32", 64, True)])
def test_right_edge_of_a_bias_read_by_the_row_threads(N, kind, D, causal, device_ok):
    """A mask at head dim 128 and an fp32 bias come from global memory in words and 16-byte chunks; what stands behind column N
    in its row, a number here that would show, is not used."""
    from triton_flashattn_b200 import flash_attention_fn

    M, H = 290, 2
    q, k, v, bias, do = make_inputs(2, M, N, H, D, BF, "bool" if kind == "bool" else "float", 4)
    rows = torch.full((2, H, M, 320), 1 if kind == "bool" else float("nan"), dtype=torch.bool if kind == "bool" else torch.float32,
                      device="cuda")
    rows[..., :N] = bias
    bias = rows[..., :N]
    q, k, v = (t.requires_grad_() for t in (q, k, v))
    wrt = [q, k, v] + ([bias.requires_grad_()] if kind == "f32" else [])
    out = flash_attention_fn(q, k, v, bias, causal)
    grads = torch.autograd.grad(out, wrt, do)
    ours = dict(zip(("dq", "dk", "dv", "dbias"), grads), out=out.detach())
    compare(ours, q.detach(), k.detach(), v.detach(), bias.detach(), causal, None, do, BF, label=f"{kind} N{N}: ")


@pytest.mark.parametrize("M,N,D,causal", [(300, 200, 128, False), (256, 300, 64, True), (200, 130, 256, True), (100, 90, 64, True),
                                          (40, 50, 32, False), (4, 300, 128, False)])
@pytest.mark.parametrize("bias_kind", [None, "float", "bool"])
@pytest.mark.parametrize("sign", [0.0, -1.0])
def test_scale_of_zero_and_below(M, N, D, causal, bias_kind, sign, device_ok):
    """The maximum of raw scores is the maximum of the scaled ones only for a positive scale."""
    check_case(2, M, N, 3, D, BF, bias_kind, causal, seed=3, sm_scale=sign * D ** -0.5)


@pytest.mark.parametrize("M,N,causal", [(50, 70, False), (200, 136, False), (200, 200, True),
                                        (128, 384, False), (384, 128, False), (100, 300, True),
                                        (300, 100, True), (1, 1, False), (129, 1, False)])
@pytest.mark.parametrize("bias_kind", [None, "float", "bool"])
def test_ragged_lengths(M, N, causal, bias_kind, device_ok):
    check_case(1, M, N, 2, 64, HF, bias_kind, causal, seed=2)


@pytest.mark.parametrize("dtype", [BF, HF])
@pytest.mark.parametrize("M,N,causal", [(256, 256, False), (256, 256, True), (200, 136, False), (300, 100, True),
                                        (100, 300, True), (129, 1, False), (640, 512, True)])
@pytest.mark.parametrize("bias_kind,trainable", [(None, False), ("float", True), ("float", False), ("bool", False)])
def test_head_dim_256(dtype, M, N, causal, bias_kind, trainable, device_ok):
    """Head dimension 256 (flash_attention.py line 776 accepts it): one query tile per CTA in the
    forward, the transposed dV kernel and the streamed dK and dQ in the backward.

    delta = rowsum(o * do) is formed from the 16-bit output, and two correct 16-bit roundings of
    o differ by one unit in some of a row's elements; that difference, summed over D = 256
    products, enters dS = P (dP - delta) in full where P is near 1 (about 1.4x the D = 128
    figure).  So against the oracle fed its OWN rounded output the bf16 bound is taken 1.5x;
    against the oracle fed this library's saved output the plain rule must hold.  (The
    reference's own Triton kernels on the same inputs: dbias max-abs 5e-2 to 6e-2, 14 to 52
    elements over 2e-2; this library 2.5e-2 to 3.2e-2, 1 to 13 elements.)"""
    q, k, v, bias, do = make_inputs(2, M, N, 2, 256, dtype, bias_kind, 12)
    ours = run_ours(q, k, v, bias, causal, None, do, trainable)
    label = f"D256 M{M} N{N} {dtype} bias={bias_kind} trainable={trainable} causal={causal}: "
    compare(ours, q, k, v, bias, causal, None, do, dtype, 1.5 if dtype == BF else 1.0, label)
    ref_saved = oracle.attention_backward(q, k, v, bias, causal, None, do, o_saved=ours["out"])
    for n, t in ours.items():
        accept(n, account(t, ref_saved[n], dtype), dtype, label=label + "(saved output) ")


@pytest.mark.parametrize("causal", [False, True])
def test_head_dim_256_fp32_bias_and_packed_qkv(causal, device_ok):
    from triton_flashattn_b200 import flash_attention_fn, flash_attention_qkvpacked_fn

    B, S, H, D = 2, 200, 2, 256
    g = torch.Generator().manual_seed(13)
    qkv = torch.randn(B, S, 3, H, D, generator=g).to(BF).cuda()
    b32 = torch.randn(B, H, S, S, generator=g).cuda()
    do = torch.randn(B, S, H, D, generator=g).to(BF).cuda()
    qkv_g, bb = qkv.clone().requires_grad_(), b32.clone().requires_grad_()
    out = flash_attention_qkvpacked_fn(qkv_g, bb, causal)
    out.backward(do)
    q, k, v = (qkv[:, :, i] for i in range(3))
    ref = oracle.attention_backward(q, k, v, b32, causal, None, do)
    assert bb.grad.dtype == torch.float32 and qkv_g.grad.shape == qkv.shape
    ours = {"out": out.detach(), "dq": qkv_g.grad[:, :, 0], "dk": qkv_g.grad[:, :, 1], "dv": qkv_g.grad[:, :, 2],
            "dbias": bb.grad}
    for n, t in ours.items():
        accept(n, account(t, ref[n], BF), BF, label=f"D256 packed fp32 bias causal={causal} {n}: ")
    if causal:
        assert torch.all(bb.grad[0, 0].triu(1) == 0)
    # the unpacked entry on the same data gives the same bits
    qq, kk, vv = (t.clone().contiguous().requires_grad_() for t in (q, k, v))
    out2 = flash_attention_fn(qq, kk, vv, b32, causal)
    out2.backward(do)
    assert torch.equal(out2, out.detach()) and torch.equal(qq.grad, qkv_g.grad[:, :, 0])
    assert torch.equal(kk.grad, qkv_g.grad[:, :, 1]) and torch.equal(vv.grad, qkv_g.grad[:, :, 2])


@pytest.mark.parametrize("M,N", [(1, 1), (1, 17), (8, 63), (9, 16), (16, 1000), (3, 4099)])
@pytest.mark.parametrize("D,dtype", [(16, HF), (32, BF), (64, HF), (128, BF), (128, HF)])
@pytest.mark.parametrize("bias_kind,causal", [(None, False), (None, True), ("float", False), ("f32", False), ("bool", True)])
def test_few_query_rows(M, N, D, dtype, bias_kind, causal, device_ok):
    """M <= 16 runs a kernel of its own: one or two groups of 8 rows, 16-key tiles spread over the
    warps of 1 to 16 CTAs, warps and whole CTAs without a key among them.  B * H = 3 leaves room
    for the largest cluster."""
    q, k, v, bias, do = make_inputs(1, M, N, 3, D, dtype, "float" if bias_kind == "f32" else bias_kind, 15)
    if bias_kind == "f32":
        bias = bias.float()
    ours = run_ours(q, k, v, bias, causal, None, do)
    ours.pop("dbias", None)
    compare(ours, q, k, v, bias, causal, None, do, dtype, label=f"M{M} N{N} D{D} {bias_kind} causal={causal}: ",
            verbose=False)


@pytest.mark.parametrize("M", [1, 2, 4, 7, 8, 16])
@pytest.mark.parametrize("N,D", [(1, 128), (33, 64), (600, 128), (1023, 32), (1920, 64), (2049, 128), (4096, 128), (9000, 64), (20011, 128)])
def test_few_rows_result_does_not_depend_on_the_other_heads(M, N, D, device_ok):
    """How the keys of a head are split over warps and CTAs depends on how many heads the call has; the result
    does not: one head alone, a batch element alone and a shard of four heads have the bits of the whole call.
    (Key counts around two and four tiles a leaf and on both sides of the largest number of leaves.)"""
    from triton_flashattn_b200 import flash_attention as fa

    B, H = 8, 32
    g = torch.Generator(device="cuda").manual_seed(28)
    q, k, v = (torch.randn(B, S, H, D, generator=g, device="cuda").to(BF) for S in (M, N, N))
    out, lse = fa._flash_attn_fwd(q, k, v, None, False, D ** -0.5)
    for b, h in ((slice(0, 1), slice(0, 1)), (slice(3, 4), slice(0, 32)), (slice(2, 6), slice(8, 12)), (slice(0, 8), slice(5, 21))):
        o, l = fa._flash_attn_fwd(q[b, :, h], k[b, :, h], v[b, :, h], None, False, D ** -0.5)
        assert torch.equal(o, out[b, :, h]) and torch.equal(l, lse[b, h]), (b, h)
    ref = oracle.attention_backward(q[:1], k[:1], v[:1], None, False, None, torch.zeros_like(q[:1]))["out"] \
        if N <= 2049 else torch.nn.functional.scaled_dot_product_attention(
            *(t[:1].float().transpose(1, 2) for t in (q, k, v))).transpose(1, 2)
    assert (out[:1].float() - ref).abs().max().item() <= TOL[BF]


@pytest.mark.parametrize("S", [4, 100])
@pytest.mark.parametrize("layout", ["one element off", "padded head dim", "heads first"])
def test_packed_qkv_in_other_layouts(S, layout, device_ok):
    """Packed projections whose slices the kernels cannot read in place are copied: same results, gradients too."""
    from triton_flashattn_b200 import flash_attention_qkvpacked_fn

    x = torch.randn(2, S, 3, 2, 64, generator=torch.Generator().manual_seed(26)).to(BF).cuda()
    do = torch.randn(2, S, 2, 64, generator=torch.Generator().manual_seed(27)).to(BF).cuda()
    if layout == "one element off":
        y = torch.empty(x.numel() + 1, dtype=BF, device="cuda")[1:].view(x.shape)
        y.copy_(x)
    elif layout == "padded head dim":
        y = torch.nn.functional.pad(x, (0, 3))[..., :64]
    else:
        y = x.permute(0, 3, 1, 2, 4).contiguous().permute(0, 2, 3, 1, 4)
    res = []
    for t in (x, y):
        t = t.detach().requires_grad_()
        out = flash_attention_qkvpacked_fn(t, None, True)
        res.append((out, *torch.autograd.grad(out, t, do)))
    for a, b in zip(*res):
        assert torch.equal(a, b)


@pytest.mark.parametrize("M", [1, 4, 16, 17])
@pytest.mark.parametrize("bias_dtype", [torch.float64, HF, torch.float32])
@pytest.mark.parametrize("trainable,packed", [(True, False), (False, False), (True, True), (False, True)])
def test_few_rows_train_with_a_bias_of_another_dtype(M, bias_dtype, trainable, packed, device_ok):
    """The kernel for few rows reads a converted bias with any row pitch, the backward's do not.  (Packed: M keys.)"""
    from triton_flashattn_b200 import flash_attention_qkvpacked_fn

    N = M if packed else 77
    q, k, v, bias, do = make_inputs(2, M, N, 3, 64, BF, "float", 25)
    bias = bias.to(bias_dtype)
    if packed:
        qkv = torch.stack([q, k, v], dim=2).requires_grad_()
        b = bias.clone().requires_grad_(trainable)
        out = flash_attention_qkvpacked_fn(qkv, b)
        out.backward(do)
        ours = {"out": out.detach(), "dq": qkv.grad[:, :, 0], "dk": qkv.grad[:, :, 1], "dv": qkv.grad[:, :, 2]}
        if trainable:
            ours["dbias"] = b.grad
    else:
        ours = run_ours(q, k, v, bias, False, None, do, trainable)
    assert not trainable or ours["dbias"].dtype == bias_dtype
    compare(ours, q, k, v, bias, False, None, do, BF, label=f"M{M} {bias_dtype}: ", verbose=False)


@pytest.mark.parametrize("M", [1, 16, 17])
@pytest.mark.parametrize("where", ["q", "key", "bias", "inf bias"])
def test_nan_scores_reach_the_output(M, where, device_ok):
    """A NaN score (or an infinite one: inf - inf) makes its row NaN, by the kernel for few rows (M <= 16) as by
    the tile kernel, and no other row or head; the log-sum-exp of such a row is +inf."""
    from triton_flashattn_b200 import flash_attention as fa

    q, k, v, bias, _ = make_inputs(1, M, 300, 2, 128, BF, "float", 23)
    clean, lse = fa._flash_attn_fwd(q, k, v, bias, False, 0.1)
    rows = slice(0, M) if where == "key" else slice(0, 1)
    if where == "q":
        q[0, 0, 0, 3] = float("nan")
    elif where == "key":
        k[0, 200, 0, 3] = float("nan")
    else:
        bias[0, 0, 0, 5] = float("nan" if where == "bias" else "inf")
    out, lse_nan = fa._flash_attn_fwd(q, k, v, bias, False, 0.1)
    assert out[0, rows, 0].isnan().all() and lse_nan[0, 0, rows].isposinf().all()
    assert torch.equal(out[:, :, 1], clean[:, :, 1]) and torch.equal(lse_nan[:, 1], lse[:, 1])
    if where != "key":
        # the head's other rows: P may be rounded against another running maximum (2^-9 of each probability, twice)
        bound = 2.0 ** -8 * (v[0, :, 0].float().abs().max() + clean[0, 1:, 0].float().abs())
        assert bool(((out[0, 1:, 0].float() - clean[0, 1:, 0].float()).abs() <= bound).all())
        assert torch.allclose(lse_nan[0, 0, 1:], lse[0, 0, 1:], rtol=0, atol=1e-4)


@pytest.mark.parametrize("M", [1, 16, 17])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_masked_key_with_a_bad_score_takes_no_part(M, bad, device_ok):
    """Keys that the mask hides may hold anything (an unwritten cache slot): their scores are ignored.  (Their
    values may not: 0 * inf in the product with V.)"""
    from triton_flashattn_b200 import flash_attention_fn

    q, k, v, mask, _ = make_inputs(1, M, 300, 2, 128, BF, "bool", 24)
    mask[..., 200] = False
    k[0, 200, :, 3] = 0
    clean = flash_attention_fn(q, k, v, mask)
    k[0, 200, :, 3] = bad
    assert torch.equal(flash_attention_fn(q, k, v, mask), clean)


@pytest.mark.parametrize("D", [16, 32])
@pytest.mark.parametrize("bias_kind", [None, "float"])
def test_small_head_dims(D, bias_kind, device_ok):
    check_case(1, 192, 160, 2, D, HF, bias_kind, True, seed=3)


def test_longer_sequence_bf16(device_ok):
    check_case(1, 1024, 1024, 2, 128, BF, "float", False, seed=4, bias_scale=0.5)
    check_case(1, 1024, 1024, 2, 64, BF, None, True, seed=5)


@pytest.mark.parametrize("max_ctas", ["1", "3", "5"])
@pytest.mark.parametrize("D,bias_kind,causal", [(128, "float", False), (128, "float", True), (64, None, True),
                                                (128, "bool", True), (64, "float", False)])
def test_many_tiles_per_persistent_cta(max_ctas, D, bias_kind, causal, device_ok, monkeypatch):
    """The kernels are persistent (one CTA per SM walks several tiles, carrying ring stages and
    barrier phases across tile boundaries).  FA_MAX_CTAS caps the grid so that a small problem
    exercises many tile boundaries per CTA, including odd tile counts and ragged edges."""
    monkeypatch.setenv("FA_MAX_CTAS", max_ctas)
    check_case(2, 3 * 128 + 40, 5 * 128 - 9, 3, D, BF, bias_kind, causal, seed=21, bias_scale=0.5)


@pytest.mark.parametrize("max_ctas", ["1", "2"])
@pytest.mark.parametrize("M,N,causal,bias_kind,trainable", [
    (1, 129, False, None, False), (129, 128, True, "bool", False), (384, 192, False, "float", True),
    (130, 400, True, "float", True), (257, 65, False, "float", False), (300, 300, True, None, False)])
def test_head_dim_256_tile_edges(max_ctas, M, N, causal, bias_kind, trainable, device_ok, monkeypatch):
    """Head dimension 256 with several key tiles per CTA: one query block and several, a last key tile of one
    key, of 64 and of 65, key tiles that no query row sees (M < N, causal).  Bounds as in test_head_dim_256."""
    monkeypatch.setenv("FA_MAX_CTAS", max_ctas)
    q, k, v, bias, do = make_inputs(2, M, N, 2, 256, BF, bias_kind, 22)
    ours = run_ours(q, k, v, bias, causal, None, do, trainable)
    ref = oracle.attention_backward(q, k, v, bias, causal, None, do, o_saved=ours["out"])
    for n, t in ours.items():
        accept(n, account(t, ref[n], BF), BF, label=f"D256 M{M} N{N} bias={bias_kind} causal={causal} {n}: ")


def test_non_trainable_float_bias(device_ok):
    check_case(1, 256, 256, 2, 128, BF, "float", True, seed=6, trainable_bias=False)


def test_dq_both_variants_agree(device_ok, monkeypatch):
    """The streamed-dS dQ kernel and the recompute dQ kernel give the same dQ."""
    import ctypes
    from triton_flashattn_b200 import flash_attention as fa_mod, _cabi

    q, k, v, bias, do = make_inputs(1, 384, 320, 2, 128, BF, "float", 7)
    res = run_ours(q, k, v, bias, True, None, do)  # streamed-dS variant (trainable bias)
    res2 = run_ours(q, k, v, bias, True, None, do, trainable_bias=False)  # recompute variant
    assert (res["dq"].float() - res2["dq"].float()).abs().max().item() <= 2e-2
    assert (res["dk"].float() - res2["dk"].float()).abs().max().item() == 0.0


def test_packed_qkv_bool_causal(device_ok):
    from triton_flashattn_b200 import flash_attention_qkvpacked_fn

    B, S, H, D = 2, 384, 2, 128
    g = torch.Generator().manual_seed(8)
    qkv = torch.randn(B, S, 3, H, D, generator=g).to(BF).cuda().requires_grad_()
    mask = torch.rand(B, H, S, S, generator=g) < 0.9
    i = torch.arange(S)
    mask[:, :, i, i] = True
    mask = mask.cuda()
    do = torch.randn(B, S, H, D, generator=g).to(BF).cuda()
    out = flash_attention_qkvpacked_fn(qkv, mask, True, None)
    out.backward(do)
    q, k, v = qkv.detach()[:, :, 0], qkv.detach()[:, :, 1], qkv.detach()[:, :, 2]
    assert out.shape == (B, S, H, D) and qkv.grad.shape == qkv.shape
    ours = {"out": out.detach(), "dq": qkv.grad[:, :, 0], "dk": qkv.grad[:, :, 1], "dv": qkv.grad[:, :, 2]}
    compare(ours, q, k, v, mask, True, None, do, BF, label="packed bool causal: ")


def test_expanded_bias_and_fp32_bias(device_ok):
    from triton_flashattn_b200 import flash_attention_fn

    B, M, N, H, D = 2, 128, 256, 2, 64
    q, k, v, _, do = make_inputs(B, M, N, H, D, HF, None, 9)
    b0 = torch.randn(1, 1, M, N, generator=torch.Generator().manual_seed(98)).to(HF).cuda().requires_grad_()
    qq = q.clone().requires_grad_()
    out = flash_attention_fn(qq, k, v, b0.expand(B, H, M, N), False, None)
    out.backward(do)
    ref = oracle.attention_backward(q, k, v, b0.detach().expand(B, H, M, N), False, None, do)
    assert (out.float() - ref["out"]).abs().max().item() <= 5e-3
    assert b0.grad.shape == b0.shape
    assert (b0.grad.float() - ref["dbias"].sum((0, 1), keepdim=True)).abs().max().item() <= 2e-2


@pytest.mark.parametrize("dtype,D,M,N,causal", [(HF, 64, 128, 256, False), (BF, 128, 300, 200, True),
                                               (BF, 64, 200, 330, False), (HF, 32, 129, 70, True)])
def test_fp32_bias_is_streamed_in_fp32_and_its_gradient_is_fp32(dtype, D, M, N, causal, device_ok):
    """A float bias in another dtype than q (the reference adds it in fp32, flash_attention.py
    lines 52 and 292, and returns its gradient in the bias's dtype, line 799) is never rounded to
    16 bits: fp32 in, fp32 dS out.  The gradient therefore meets the absolute bound without the
    16-bit rounding allowance, and a bias with digits a 16-bit type cannot hold changes the output."""
    from triton_flashattn_b200 import flash_attention_fn

    B, H = 2, 2
    scale = 0.3 if D <= 32 else None  # (0.3 at D >= 64 makes scores of +-10: a test of bf16, not of this path)
    q, k, v, _, do = make_inputs(B, M, N, H, D, dtype, None, 9)
    g = torch.Generator().manual_seed(99)
    b32 = torch.randn(B, H, M, N, generator=g).cuda()
    qq, kk, vv, bb = (t.clone().requires_grad_() for t in (q, k, v, b32))
    out = flash_attention_fn(qq, kk, vv, bb, causal, scale)
    out.backward(do)
    ref = oracle.attention_backward(q, k, v, b32, causal, scale, do)
    assert bb.grad.dtype == torch.float32 and bb.grad.is_contiguous() and bb.grad.shape == b32.shape
    ours = {"out": out.detach(), "dq": qq.grad, "dk": kk.grad, "dv": vv.grad}
    for n, t in ours.items():
        accept(n, account(t, ref[n], dtype), dtype, label=f"fp32 bias {dtype} {n}: ")
    accept("dbias", account(bb.grad, ref["dbias"], dtype), dtype, label=f"fp32 bias {dtype} dbias: ")
    # Against the oracle fed this library's own saved 16-bit output (so that the one-unit
    # differences between two roundings of `o`, which move delta, drop out) the fp32 gradient
    # shows no trace of a 16-bit rounding of dS: a quarter of the absolute bound, no allowance.
    ref_saved = oracle.attention_backward(q, k, v, b32, causal, scale, do, o_saved=out.detach())
    err = (bb.grad - ref_saved["dbias"]).abs().max().item()
    print(f"fp32 dbias max-abs error vs oracle on the saved output {err:.2e}")
    assert err <= TOL[dtype] / 4, err
    if causal:
        assert torch.all(bb.grad[0, 0].triu(1) == 0)
    # the low bits of the fp32 bias matter: rounding it to 16 bits first gives another result
    out16 = flash_attention_fn(q, k, v, b32.to(dtype), causal, scale)
    assert not torch.equal(out16, out.detach())
    # a float64 bias takes the same path and gets a float64 gradient
    b64 = b32.double().requires_grad_()
    out64 = flash_attention_fn(q, k, v, b64, causal, scale)
    out64.backward(do)
    assert b64.grad.dtype == torch.float64 and torch.equal(out64, out.detach())
    assert torch.equal(b64.grad.float(), bb.grad)


def test_fully_masked_row_is_zero_not_nan(device_ok):
    q, k, v, _, do = make_inputs(1, 128, 128, 1, 64, HF, None, 10)
    mask = torch.ones(1, 1, 128, 128, dtype=torch.bool, device="cuda")
    mask[0, 0, 5, :] = False
    res = run_ours(q, k, v, mask, False, None, do)
    assert torch.all(res["out"][0, 5, 0] == 0)
    for t in res.values():
        assert torch.isfinite(t.float()).all()
    ref = oracle.attention_backward(q, k, v, mask, False, None, do)
    assert (res["out"].float() - ref["out"]).abs().max().item() <= 5e-3
    assert (res["dq"].float() - ref["dq"]).abs().max().item() <= 5e-3


def test_deterministic_bitwise(device_ok):
    q, k, v, bias, do = make_inputs(2, 384, 384, 2, 128, BF, "float", 11)
    a = run_ours(q, k, v, bias, True, None, do)
    b = run_ours(q, k, v, bias, True, None, do)
    for name in a:
        assert torch.equal(a[name], b[name]), name


def test_causal_dbias_upper_triangle_is_zero(device_ok):
    q, k, v, bias, do = make_inputs(1, 384, 384, 1, 64, HF, "float", 12)
    res = run_ours(q, k, v, bias, True, None, do)
    assert torch.all(res["dbias"][0, 0].triu(1) == 0)


def test_bad_arguments_raise():
    from triton_flashattn_b200 import flash_attention_fn

    q = torch.randn(1, 64, 2, 64, device="cuda", dtype=HF)
    with pytest.raises(ValueError):
        flash_attention_fn(q, q, q, torch.zeros(1, 1, 64, 64, device="cuda", dtype=HF))
    with pytest.raises(AssertionError):
        x = torch.randn(1, 64, 2, 48, device="cuda", dtype=HF)
        flash_attention_fn(x, x, x)
    with pytest.raises(TypeError):
        flash_attention_fn(q.float(), q.float(), q.float())


# ---- against the reference's own outputs (golden vectors made by its Triton kernels)
from tests import _golden  # noqa: E402


@pytest.mark.parametrize("name", _golden.names())
def test_against_reference_golden_vectors(name, device_ok):
    from triton_flashattn_b200 import flash_attention_fn, flash_attention_qkvpacked_fn

    g = _golden.load(name)
    bias = g.get("bias")
    if bias is not None:
        bias = bias.cuda()
    do = g["do"].cuda()
    tol = 5e-3  # both sides are fp16 results of the same algorithm
    if g["packed"]:
        x = g["qkv"].cuda().requires_grad_()
        out = flash_attention_qkvpacked_fn(x, bias, g["causal"], g["sm_scale"])
        out.backward(do)
        assert (out.float().cpu() - g["out"].float()).abs().max().item() <= tol
        assert (x.grad.float().cpu() - g["dqkv"].float()).abs().max().item() <= tol
        return
    q, k, v = (g[n].cuda().requires_grad_() for n in ("q", "k", "v"))
    trainable = "dbias" in g
    if trainable:
        bias = bias.requires_grad_()
    out = flash_attention_fn(q, k, v, bias, g["causal"], g["sm_scale"])
    out.backward(do)
    assert (out.float().cpu() - g["out"].float()).abs().max().item() <= tol
    for n, t in (("dq", q), ("dk", k), ("dv", v)):
        assert (t.grad.float().cpu() - g[n].float()).abs().max().item() <= tol, n
    if trainable:
        assert (bias.grad.float().cpu() - g["dbias"].float()).abs().max().item() <= tol


def _check_slices(ours, q, k, v, bias, do, causal, pairs, label):
    """Checks the (b, h) problems in `pairs` of a larger run against the oracle, one slice at
    a time, and returns the worst account per tensor."""
    worst = {}
    for b, h in pairs:
        sl = lambda t: t[b:b + 1, :, h:h + 1]
        bb = None if bias is None else bias[b:b + 1, h:h + 1]
        part = {n: sl(t) for n, t in ours.items() if n != "dbias"}
        if "dbias" in ours:
            part["dbias"] = ours["dbias"][b:b + 1, h:h + 1]
        acc = compare(part, sl(q), sl(k), sl(v), bb, causal, None, sl(do), BF, label=f"{label} (b={b},h={h}): ",
                      verbose=False)
        for n, a in acc.items():
            if n not in worst or a["raw"] > worst[n]["raw"]:
                worst[n] = a
    print(label + " worst over slices: " + " ".join(
        f"{n}={a['raw']:.2e}[over:{a['n_over']}]" for n, a in worst.items()), flush=True)
    return worst


# ---- the benchmark configurations at their full M, N, D (reduced batch/heads), checked
# ---- slice by slice against the fp32 oracle with the stated tolerances
@pytest.mark.parametrize("cfg", ["2", "3", "4", "5"])
def test_benchmark_config_shapes(cfg, device_ok):
    from triton_flashattn_b200 import flash_attention_qkvpacked_fn

    spec = {"2": (2, 4, 1024, 64, None, True), "3": (1, 4, 2048, 128, "float", False),
            "4": (1, 2, 4096, 128, "bool", True), "5": (1, 1, 8192, 128, "float", True)}[cfg]
    B, H, S, D, bias_kind, causal = spec
    q, k, v, bias, do = make_inputs(B, S, S, H, D, BF, bias_kind, int(cfg), bias_scale=0.5)
    if cfg == "4":
        qkv = torch.stack([q, k, v], dim=2).requires_grad_()
        out = flash_attention_qkvpacked_fn(qkv, bias, causal, None)
        out.backward(do)
        ours = {"out": out.detach(), "dq": qkv.grad[:, :, 0], "dk": qkv.grad[:, :, 1], "dv": qkv.grad[:, :, 2]}
    else:
        ours = run_ours(q, k, v, bias, causal, None, do)
    _check_slices(ours, q, k, v, bias, do, causal, [(b, h) for b in range(B) for h in range(H)],
                  f"config {cfg} shape")
    if cfg == "4":
        # the mask pattern is reproduced exactly: masked-out keys get exactly zero probability,
        # so dk/dv of a key that no query may see are exactly zero -- checked on a tiny extra case
        m = torch.ones(1, 1, 128, 128, dtype=torch.bool, device="cuda")
        m[..., 7] = False
        qq, kk, vv, _, dd = make_inputs(1, 128, 128, 1, 64, BF, None, 1)
        r = run_ours(qq, kk, vv, m, False, None, dd)
        assert torch.all(r["dk"][0, 7] == 0) and torch.all(r["dv"][0, 7] == 0)


def test_config3_full_size_sampled_slices(device_ok):
    """The headline configuration at its full size (B=8, H=16, M=N=2048, D=128, bf16, trainable
    bias): every persistent CTA walks 13-14 tiles.  Eight (b, h) problems spread over the
    batch, heads and the CTAs' tile lists are value-checked against the oracle."""
    B, H, S, D = 8, 16, 2048, 128
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *shape, scale=1.0: (scale * torch.randn(*shape, generator=g, device="cuda")).to(BF)
    q, k, v, do = rnd(B, S, H, D), rnd(B, S, H, D), rnd(B, S, H, D), rnd(B, S, H, D)
    bias = rnd(B, H, S, S, scale=0.5)
    ours = run_ours(q, k, v, bias, False, None, do)
    pairs = [(0, 0), (1, 5), (2, 10), (3, 15), (4, 3), (5, 8), (6, 13), (7, 15)]
    _check_slices(ours, q, k, v, bias, do, False, pairs, "config 3 full size")
