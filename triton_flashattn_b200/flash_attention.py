"""Flash attention with an optional trainable (B, H, M, N) bias for NVIDIA B200.

Drop-in for the public interface of the reference project's `flash_attention.py`
(cited below as FA:<line>): the same two functions, the same two
`torch.autograd.Function` classes, the same argument order, defaults, layouts and
return values.  The compute path is libfa_sm100.so (hand-written sm_100a CUDA
kernels behind a C ABI, see include/fa_sm100.h), reached through _fa_torch.so
(csrc/torch_binding.cpp: checks, allocation, autograd node); there is no other path.

    flash_attention_fn(q, k, v, bias=None, causal=False, sm_scale=None)          FA:848
    flash_attention_qkvpacked_fn(qkv, bias=None, causal=False, sm_scale=None)    FA:852

    q       : (B, M, H, D)      k, v : (B, N, H, D)      qkv : (B, S, 3, H, D)
    bias    : (B, H, M, N)      bool  -> scores where bias is False are ignored
                                float -> added to q.k^T * sm_scale before the softmax
    returns : (B, M, H, D) in q's dtype

If a float bias has requires_grad, backward also returns its gradient at the full
(B, H, M, N) shape (dS, written by the dK/dV kernel).
"""
from __future__ import annotations

import ctypes

import torch

from . import _cabi

_DTYPES = {torch.float16: _cabi.FA_F16, torch.bfloat16: _cabi.FA_BF16}


class _MissingLibrary:
    """Stands in for the launch path until it has been built: any use says how to build it."""

    def __init__(self, error: ImportError):
        self._error = error

    def __getattr__(self, name):
        raise ImportError(
            "triton_flashattn_b200/_fa_torch.so cannot be loaded: build it with `python -m "
            "triton_flashattn_b200.build` (needs nvcc with sm_100a support). There is no fallback path."
        ) from self._error


try:
    from . import _fa_torch as _native
except ImportError as e:
    _native = _MissingLibrary(e)
else:
    _native.set_health_registrar(lambda device: ctypes.addressof(_cabi.health_words(device)))


def _stride3(t: torch.Tensor):
    st = t.stride()
    return _cabi._I64x3(st[0], st[1], st[2])


def _classify_bias(bias, q):
    """Returns (kernel_bias_tensor_or_None, kind): the bias as the kernels read it (rows with a
    16-byte aligned pitch, copied only if they lack it; other float dtypes than q's as fp32)."""
    return _native.classify_bias(bias, q)


def _params(q, k, v, o, lse, bias_t, bias_kind, causal, sm_scale):
    B, M, H, D = q.shape
    N = k.shape[1]
    p = _cabi.FaParams()
    p.struct_size = ctypes.sizeof(_cabi.FaParams)
    p.device = q.device.index if q.device.index is not None else torch.cuda.current_device()
    p.B, p.H, p.M, p.N, p.D = B, H, M, N, D
    p.dtype = _DTYPES[q.dtype]
    p.bias_kind = bias_kind
    p.causal = 1 if causal else 0
    p.write_dbias = 0
    p.sm_scale = float(sm_scale)
    p.q, p.k, p.v, p.o = q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr()
    p.q_stride, p.k_stride, p.v_stride, p.o_stride = _stride3(q), _stride3(k), _stride3(v), _stride3(o)
    p.lse = lse.data_ptr()
    if bias_t is not None:
        p.bias = bias_t.data_ptr()
        p.bias_stride = _stride3(bias_t)
    return p


def _flash_attn_fwd(q, k, v, bias, causal, sm_scale):
    """Forward launch; returns (o, lse2).  Mirrors FA:649-685.
    lse2 is the log2-domain log-sum-exp, fp32, laid out (B, H, M)."""
    return _native.fwd(q, k, v, bias, causal, sm_scale)


def _flash_attn_bwd(do, q, k, v, o, bias, causal, sm_scale, lse, dq, dk, dv, dbias):
    """Backward launches; fills dq, dk, dv (and dbias) in place.
    Mirrors FA:688-763.  dbias, when given, must be a (B, H, M, N) tensor whose row pitch is a
    multiple of 16 bytes (see `_empty_dbias`): in q's dtype for a bias in q's dtype, fp32 (and
    zero-filled when causal) for any other float bias."""
    _native.bwd(do, q, k, v, o, bias, causal, sm_scale, lse, dq, dk, dv, dbias)


def _empty_dbias(bias: torch.Tensor, dtype: torch.dtype, zero: bool = False) -> torch.Tensor:
    """(B, H, M, N) gradient buffer with a 16-byte aligned row pitch: dense when N allows it,
    else a view of a padded buffer (the caller compacts it afterwards).  For a 16-bit bias no
    zero fill is needed: the dK/dV kernel writes every tile, including the causally skipped
    ones (the reference relies on zeros_like, FA:799).  `zero`: fp32 gradient of a causal
    problem, whose skipped tiles nobody writes."""
    return _pitched_empty(tuple(bias.shape), dtype, bias.device, zero)


def _pitched_empty(shape, dtype: torch.dtype, device, zero: bool = False) -> torch.Tensor:
    """(B, H, M, N) tensor whose row pitch is a multiple of 16 bytes (a view of a padded buffer
    when N needs it)."""
    B, H, M, N = shape
    per16 = 16 // dtype.itemsize
    n_pad = (N + per16 - 1) // per16 * per16
    make = torch.zeros if zero else torch.empty
    buf = make((B, H, M, n_pad), dtype=dtype, device=device)
    return buf[..., :N]


def _new_dbias(bias: torch.Tensor, q: torch.Tensor, causal: bool) -> torch.Tensor:
    """Gradient buffer for `bias` as the kernels write it: q's dtype when the bias has it, else
    fp32.  Zero-filled where the kernels skip the causally masked tiles without writing them
    (fp32 gradients; every gradient at head dim 256)."""
    if bias.dtype == q.dtype:
        return _empty_dbias(bias, q.dtype, zero=bool(causal) and q.shape[-1] == 256)
    return _empty_dbias(bias, torch.float32, zero=bool(causal))


def _finish_dbias(dbias, bias):
    """Gradient as the reference returns it (FA:799): dense, in the bias's own dtype."""
    if dbias is None:
        return None
    if dbias.dtype != bias.dtype:
        return dbias.to(bias.dtype)  # also compacts a padded buffer
    return dbias if dbias.is_contiguous() else dbias.contiguous()


def _grad_like(t: torch.Tensor) -> torch.Tensor:
    """empty_like (strides preserved, as FA:796-798) when the kernels can write through those
    strides, else a contiguous tensor."""
    g = torch.empty_like(t)
    s0, s1, s2, s3 = g.stride()
    ok = s3 == 1 and s0 > 0 and s1 > 0 and s2 > 0 and (s0 | s1 | s2) % 8 == 0 and g.data_ptr() % 16 == 0
    return g if ok else torch.empty(t.shape, dtype=t.dtype, device=t.device)


class FlashAttentionFn(torch.autograd.Function):
    """Separate q, k, v.  Mirrors FlashAttentionFn of the reference (FA:766-803).
    (`flash_attention_fn` builds the same node in C++; this class is the reference's public name.)"""

    @staticmethod
    def forward(ctx, q, k, v, bias=None, causal=False, sm_scale=None):
        D = q.shape[-1]
        sm_scale = (D ** -0.5) if sm_scale is None else sm_scale
        is_bias = bias is not None
        is_bias_trainable = bool(is_bias and bias.requires_grad)
        if is_bias_trainable and bias.dtype == torch.bool:
            raise TypeError("a bool mask cannot require grad")
        o, lse = _flash_attn_fwd(q, k, v, bias, causal, sm_scale)
        ctx.save_for_backward(q, k, v, o, lse, bias)
        ctx.sm_scale = sm_scale
        ctx.causal = causal
        ctx.is_bias = is_bias
        ctx.is_bias_trainable = is_bias_trainable
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, lse, bias = ctx.saved_tensors
        dq, dk, dv = _grad_like(q), _grad_like(k), _grad_like(v)
        dbias = _new_dbias(bias, q, ctx.causal) if ctx.is_bias_trainable else None
        _flash_attn_bwd(do, q, k, v, o, bias, ctx.causal, ctx.sm_scale, lse, dq, dk, dv, dbias)
        return dq, dk, dv, _finish_dbias(dbias, bias), None, None


class FlashAttentionQKVPackedFn(torch.autograd.Function):
    """Packed (B, S, 3, H, D) input; q, k, v are strided views and the three
    gradients are written into views of one dqkv tensor.  Mirrors FA:806-845."""

    @staticmethod
    def forward(ctx, qkv, bias=None, causal=False, sm_scale=None):
        if qkv.dim() != 5 or qkv.shape[2] != 3:
            raise ValueError("qkv must be (B, S, 3, H, D)")
        D = qkv.shape[-1]
        sm_scale = (D ** -0.5) if sm_scale is None else sm_scale
        is_bias = bias is not None
        is_bias_trainable = bool(is_bias and bias.requires_grad)
        if is_bias_trainable and bias.dtype == torch.bool:
            raise TypeError("a bool mask cannot require grad")
        o, lse = _flash_attn_fwd(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], bias, causal, sm_scale)
        ctx.save_for_backward(qkv, o, lse, bias)
        ctx.sm_scale = sm_scale
        ctx.causal = causal
        ctx.is_bias = is_bias
        ctx.is_bias_trainable = is_bias_trainable
        return o

    @staticmethod
    def backward(ctx, do):
        qkv, o, lse, bias = ctx.saved_tensors
        dqkv = torch.empty_like(qkv)
        if not dqkv.is_contiguous():
            dqkv = torch.empty(qkv.shape, dtype=qkv.dtype, device=qkv.device)
        dbias = _new_dbias(bias, qkv, ctx.causal) if ctx.is_bias_trainable else None
        _flash_attn_bwd(
            do, qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], o, bias, ctx.causal, ctx.sm_scale, lse,
            dqkv[:, :, 0], dqkv[:, :, 1], dqkv[:, :, 2], dbias,
        )
        return dqkv, _finish_dbias(dbias, bias), None, None


def flash_attention_fn(q, k, v, bias=None, causal=False, sm_scale=None):
    return _native.attention(q, k, v, bias, causal, sm_scale)


def flash_attention_qkvpacked_fn(qkv, bias=None, causal=False, sm_scale=None):
    return _native.attention_packed(qkv, bias, causal, sm_scale)
