"""Tensor-level entry points: torch tensors in, torch tensors out, C ABI in between.

PyTorch is plumbing here (device memory, current stream, device guard); every
computation is a kernel of libtrinix_b200.so. All functions require CUDA tensors and
raise otherwise — there is no CPU path and no fallback.
"""
from __future__ import annotations

import ctypes
import threading
from typing import Optional, Tuple

import torch

from . import _lib
from ._lib import I64x3

_DTYPE_CODE = {torch.float32: _lib.TRX_F32, torch.float16: _lib.TRX_F16,
               torch.bfloat16: _lib.TRX_BF16}

GLU_ACTS = {"swiglu": _lib.GLU_SWIGLU, "geglu": _lib.GLU_GEGLU_TANH, "reglu": _lib.GLU_REGLU}

# Number of kernels launched through this module (the benchmark reports it).
launch_count = 0


def _count(n: int = 1) -> None:
    global launch_count
    launch_count += n


def _code(t: torch.Tensor) -> int:
    try:
        return _DTYPE_CODE[t.dtype]
    except KeyError:
        raise TypeError(f"trinix_b200 supports float32/float16/bfloat16, got {t.dtype}") from None


def _need_cuda(*ts: Optional[torch.Tensor]) -> torch.device:
    dev = None
    for t in ts:
        if t is None:
            continue
        if not t.is_cuda:
            raise ValueError("trinix_b200 kernels require CUDA tensors (there is no CPU path)")
        if dev is None:
            dev = t.device
        elif t.device != dev:
            raise ValueError(f"tensors on different devices: {dev} and {t.device}")
    assert dev is not None
    return dev


_entries: dict = {}  # C entry points by name
# The current stream's handle without a torch.cuda.Stream object around it.
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None) or (
    lambda index: torch.cuda.current_stream(index).cuda_stream)


def _launch(name: str, dev: torch.device, *args) -> None:
    """Call one C entry point on dev's current stream (its last argument) and raise on a status.

    A call of this library is 3 to 100 us of device work, so what the host does around it counts:
    the entry point is looked up once, the device is only switched when another one is current,
    pointers go as plain integers, and the stream as its raw handle. 512 x 768 fp32 RMSNorm, call
    after call: 9.9 us, of which the launch itself is about 4; 22.3 us with a device guard, a stream
    object and a c_void_p per argument."""
    fn = _entries.get(name)
    if fn is None:
        fn = _entries[name] = getattr(_lib.load(), name)
    index, current = dev.index, torch.cuda.current_device()
    if index is None or index == current:
        rc = fn(*args, _raw_stream(current))
    else:
        with torch.cuda.device(index):
            rc = fn(*args, _raw_stream(index))
    if rc:
        _lib.check(name, rc)
    _count()


def _ptr(t: Optional[torch.Tensor]) -> int:
    return t.data_ptr() if t is not None else 0


def _dense(t: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """A parameter vector as the kernels read it; only its memory is used, so no detach."""
    return t if t is None or t.is_contiguous() else t.detach().contiguous()


def _rows(x: torch.Tensor) -> Tuple[torch.Tensor, int, int]:
    """x as rows of its last dim with a unit column stride: (tensor that holds them, number of rows,
    row stride). A view unless x has overlapping or strided rows, which are copied."""
    c = x.shape[-1]
    if c and x.is_contiguous():
        return x, x.numel() // c, c
    x2 = x.reshape(-1, c)
    # expanded tensors (a broadcast gradient, say) have rows that overlap: materialise them
    if x2.numel() and (x2.stride(-1) != 1 or (x2.shape[0] > 1 and x2.stride(0) < c)):
        x2 = x2.contiguous()
    return x2, x2.shape[0], x2.stride(0) if x2.shape[0] > 1 else c


# Types whose empty_like / new_empty are plain tensors; for any other subclass they are instances of it.
_PLAIN = (torch.Tensor, torch.nn.Parameter)


def _empty(x: torch.Tensor, shape, dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """An uninitialised plain tensor on x's device, of x's dtype unless another one is given."""
    if type(x) in _PLAIN:
        return x.new_empty(shape, dtype=dtype)
    return torch.empty(shape, dtype=dtype or x.dtype, device=x.device)


def _new(x: torch.Tensor, dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """The same of x's shape, with the strides of a contiguous tensor. Without the memory
    format empty_like keeps x's strides, arbitrary ones of size-1 dims among them, which the C
    entries that check their output's strides refuse. (1.0 us of host time; torch.empty with a
    dtype and a device 3.6.)"""
    if type(x) in _PLAIN:
        return torch.empty_like(x, dtype=dtype, memory_format=torch.contiguous_format)
    return _empty(x, x.shape, dtype)


def _check_weight(weight: torch.Tensor, x: torch.Tensor) -> None:
    if weight.numel() != x.shape[-1]:
        raise ValueError(f"weight has {weight.numel()} elements, rows have {x.shape[-1]}")


# ----------------------------------------------------------------------------- norms
def rmsnorm(x: torch.Tensor, weight: torch.Tensor, eps: float = 1e-6,
            return_rstd: bool = False):
    """RMSNorm over the last dim; output has x's dtype and shape."""
    dev = _need_cuda(x, weight)
    _check_weight(weight, x)
    x2, rows, stride = _rows(x)
    w, c, y = _dense(weight), x.shape[-1], _new(x)
    rstd = _row_stat(x, rows) if return_rstd else None
    _launch("trx_rmsnorm_fwd", dev, x2.data_ptr(), w.data_ptr(), y.data_ptr(), _ptr(rstd), rows, c,
            stride, c, float(eps), _code(x2), _code(w))
    return (y, rstd) if return_rstd else y


def _row_stat(x: torch.Tensor, rows: int) -> torch.Tensor:
    """fp32 output for one statistic per row of x."""
    return _empty(x, rows, dtype=torch.float32)


def _affine(x: torch.Tensor, weight: Optional[torch.Tensor], bias: Optional[torch.Tensor]):
    """(weight, bias, their dtype) of a LayerNorm as the kernels read them: one dtype for both."""
    dtype = weight.dtype if weight is not None else (bias.dtype if bias is not None else x.dtype)
    w = _dense(weight)
    b = _dense(bias if bias is None or bias.dtype == dtype else bias.detach().to(dtype))
    for t in (w, b):
        if t is not None and t.numel() != x.shape[-1]:
            raise ValueError("weight/bias size does not match the normalised dim")
    return w, b, dtype


def layernorm(x: torch.Tensor, weight: Optional[torch.Tensor], bias: Optional[torch.Tensor],
              eps: float = 1e-5, return_stats: bool = False):
    """LayerNorm over the last dim; weight/bias may be None. With return_stats, (y, mean, rstd)
    with the fp32 row statistics that layernorm_backward takes."""
    dev = _need_cuda(x, weight, bias)
    x2, rows, stride = _rows(x)
    w, b, wb_dtype = _affine(x, weight, bias)
    c, y = x.shape[-1], _new(x)
    mean, rstd = (_row_stat(x, rows), _row_stat(x, rows)) if return_stats else (None, None)
    _launch("trx_layernorm_fwd", dev, x2.data_ptr(), _ptr(w), _ptr(b), y.data_ptr(), _ptr(mean),
            _ptr(rstd), rows, c, stride, c, float(eps), _code(x2), _DTYPE_CODE[wb_dtype])
    return (y, mean, rstd) if return_stats else y


# ----------------------------------------------------------------------------- int8
def quantize_rowwise(x: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """Per-row symmetric int8: returns (codes int8 of x's shape, scales fp32 of shape[:-1])."""
    dev = _need_cuda(x)
    x2, rows, stride = _rows(x)
    c, codes = x.shape[-1], _new(x, torch.int8)
    scales = _empty(x, x.shape[:-1], dtype=torch.float32)
    _launch("trx_quant_rowwise_i8", dev, x2.data_ptr(), codes.data_ptr(), scales.data_ptr(), rows, c,
            stride, c, _code(x2))
    return codes, scales


def dequantize_rowwise(codes: torch.Tensor, scales: torch.Tensor,
                       dtype: torch.dtype = torch.bfloat16,
                       out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Inverse of quantize_rowwise: round_dtype(float(code) * scale[row])."""
    dev = _need_cuda(codes, scales)
    if codes.dtype != torch.int8 or scales.dtype != torch.float32:
        raise TypeError("codes must be int8 and scales float32")
    c2, rows, stride = _rows(codes)
    s = _dense(scales)
    if s.numel() != rows:
        raise ValueError("one scale per row expected")
    if out is None:
        out = _new(codes, dtype)
    elif out.dtype != dtype or out.numel() != c2.numel() or not out.is_contiguous():
        raise ValueError("out must be a contiguous tensor of the requested dtype and size")
    else:
        out = out.view(codes.shape)
    c = codes.shape[-1]
    _launch("trx_dequant_rowwise_i8", dev, c2.data_ptr(), s.data_ptr(), out.data_ptr(), rows, c,
            stride, c, _DTYPE_CODE[dtype])
    return out


def rmsnorm_quantize(x: torch.Tensor, weight: torch.Tensor,
                     eps: float = 1e-6) -> Tuple[torch.Tensor, torch.Tensor]:
    """Fused RMSNorm -> int8; equals quantize_rowwise(rmsnorm(x, weight, eps)) bit for bit."""
    dev = _need_cuda(x, weight)
    _check_weight(weight, x)
    x2, rows, stride = _rows(x)
    w, c, codes = _dense(weight), x.shape[-1], _new(x, torch.int8)
    scales = _empty(x, x.shape[:-1], dtype=torch.float32)
    _launch("trx_rmsnorm_quant_i8", dev, x2.data_ptr(), w.data_ptr(), codes.data_ptr(),
            scales.data_ptr(), rows, c, stride, c, float(eps), _code(x2), _code(w))
    return codes, scales


ROW_ACTIVATIONS = {"mish": 0, "quickgelu": 1, "squared_relu": 2}


def rmsnorm_activation(x: torch.Tensor, weight: torch.Tensor, eps: float = 1e-6,
                       activation: str = "mish") -> torch.Tensor:
    """activation(RMSNorm(x)) in one pass; activation in {"mish", "quickgelu", "squared_relu"}."""
    if activation not in ROW_ACTIVATIONS:
        raise ValueError(f"Unsupported activation '{activation}'. "
                         f"Supported: {sorted(ROW_ACTIVATIONS)}")
    dev = _need_cuda(x, weight)
    _check_weight(weight, x)
    x2, rows, stride = _rows(x)
    w, c, y = _dense(weight), x.shape[-1], _new(x)
    _launch("trx_rmsnorm_act_fwd", dev, x2.data_ptr(), w.data_ptr(), y.data_ptr(), rows, c, stride, c,
            float(eps), ROW_ACTIVATIONS[activation], _code(x2), _code(w))
    return y


def _check_residual(x: torch.Tensor, residual: torch.Tensor) -> None:
    if residual.shape != x.shape or residual.dtype != x.dtype:
        raise ValueError("residual must have the shape and dtype of x")


def residual_rmsnorm(x: torch.Tensor, residual: torch.Tensor, weight: torch.Tensor,
                     eps: float = 1e-6, return_sum: bool = False, return_rstd: bool = False):
    """RMSNorm(x + residual) with the sum kept in fp32 on chip; optionally also returns the
    summed residual stream rounded to x's dtype, and the fp32 rstd that rmsnorm_backward takes."""
    dev = _need_cuda(x, residual, weight)
    _check_residual(x, residual)
    _check_weight(weight, x)
    (x2, rows, stride), (r2, _, r_stride) = _rows(x), _rows(residual)
    w, c, y = _dense(weight), x.shape[-1], _new(x)
    s = _new(x) if return_sum else None
    rstd = _row_stat(x, rows) if return_rstd else None
    _launch("trx_residual_rmsnorm_fwd", dev, x2.data_ptr(), r2.data_ptr(), w.data_ptr(), y.data_ptr(),
            _ptr(s), _ptr(rstd), rows, c, stride, r_stride, c, c, float(eps), _code(x2), _code(w))
    out = (y,) + ((s,) if return_sum else ()) + ((rstd,) if return_rstd else ())
    return out if len(out) > 1 else y


def residual_layernorm(x: torch.Tensor, residual: torch.Tensor, weight: Optional[torch.Tensor],
                       bias: Optional[torch.Tensor], eps: float = 1e-5,
                       return_sum: bool = False, return_stats: bool = False):
    """LayerNorm(x + residual) with the sum kept in fp32 on chip; the normalised value is rounded
    to x's dtype before the affine part, as the reference's fused module does. Optionally also
    returns the summed residual stream rounded to x's dtype, and the fp32 mean and rstd that
    layernorm_backward takes."""
    dev = _need_cuda(x, residual, weight, bias)
    _check_residual(x, residual)
    w, b, wb_dtype = _affine(x, weight, bias)
    (x2, rows, stride), (r2, _, r_stride) = _rows(x), _rows(residual)
    c, y = x.shape[-1], _new(x)
    s = _new(x) if return_sum else None
    mean, rstd = (_row_stat(x, rows), _row_stat(x, rows)) if return_stats else (None, None)
    _launch("trx_residual_layernorm_fwd", dev, x2.data_ptr(), r2.data_ptr(), _ptr(w), _ptr(b),
            y.data_ptr(), _ptr(s), _ptr(mean), _ptr(rstd), rows, c, stride, r_stride, c, c, float(eps),
            _code(x2), _DTYPE_CODE[wb_dtype])
    out = (y,) + ((s,) if return_sum else ()) + ((mean, rstd) if return_stats else ())
    return out if len(out) > 1 else y


def residual_rmsnorm_quantize(x: torch.Tensor, residual: torch.Tensor, weight: torch.Tensor,
                              eps: float = 1e-6, return_sum: bool = False):
    """int8 codes and scales of RMSNorm(x + residual); equals
    quantize_rowwise(residual_rmsnorm(x, residual, weight, eps)) bit for bit."""
    dev = _need_cuda(x, residual, weight)
    _check_residual(x, residual)
    _check_weight(weight, x)
    (x2, rows, stride), (r2, _, r_stride) = _rows(x), _rows(residual)
    w, c, codes = _dense(weight), x.shape[-1], _new(x, torch.int8)
    scales = _empty(x, x.shape[:-1], dtype=torch.float32)
    s = _new(x) if return_sum else None
    _launch("trx_residual_rmsnorm_quant_i8", dev, x2.data_ptr(), r2.data_ptr(), w.data_ptr(),
            codes.data_ptr(), scales.data_ptr(), _ptr(s), rows, c, stride, r_stride, c, c, float(eps),
            _code(x2), _code(w))
    return (codes, scales, s) if return_sum else (codes, scales)


# ----------------------------------------------------------------------------- RoPE
def _bshd(t: torch.Tensor) -> torch.Tensor:
    if t.dim() != 4:
        raise ValueError(f"expected (batch, seq, heads, head_dim), got {tuple(t.shape)}")
    return t if t.stride(-1) == 1 or t.numel() == 0 else t.contiguous()


def _tma_view(t: torch.Tensor) -> torch.Tensor:
    """A (B, S, H, D) view the attention kernel's tensor maps accept: unit head-dim stride, a
    16-byte aligned base and batch / seq / head strides that are multiples of 8 elements (a
    stride of 0, an expanded dim, is fine and stays as it is). Any other legal view (a slice
    along D at an odd offset, a head stride of 100, ...) is materialised once."""
    t = _bshd(t)
    if t.numel() == 0:
        return t
    ok = t.data_ptr() % 16 == 0 and all(
        t.shape[i] == 1 or t.stride(i) % 8 == 0 for i in range(3))
    return t if ok else t.contiguous()


def rope(q: torch.Tensor, k: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor,
         inverse: bool = False) -> Tuple[torch.Tensor, torch.Tensor]:
    """Half-split rotary embedding of q (B,S,Hq,D) and k (B,S,Hk,D) in one launch.

    cos/sin are (S, D) (or anything that squeezes to it); only columns < D/2 are read.
    Tables must be float32 or have q's dtype.
    """
    dev = _need_cuda(q, k, cos, sin)
    if q.dtype != k.dtype:
        raise TypeError("q and k must share a dtype")
    q, k = _bshd(q), _bshd(k)
    B, S, Hq, D = q.shape
    if k.shape[0] != B or k.shape[1] != S or k.shape[3] != D:
        raise ValueError(f"k shape {tuple(k.shape)} does not match q {tuple(q.shape)}")
    cos2 = cos.reshape(-1, cos.shape[-1])
    sin2 = sin.reshape(-1, sin.shape[-1])
    if cos2.shape != sin2.shape or cos2.shape[0] < S or cos2.shape[1] < D // 2:
        raise ValueError("cos/sin tables must be (>= seq_len, >= head_dim/2) and alike")
    if cos2.dtype != sin2.dtype or cos2.dtype not in (torch.float32, q.dtype):
        cos2, sin2 = cos2.float(), sin2.float()
    cos2, sin2 = cos2.contiguous(), sin2.contiguous()
    qo, ko = _new(q), _new(k)
    _launch("trx_rope_fwd", dev, q.data_ptr(), k.data_ptr(), cos2.data_ptr(), sin2.data_ptr(),
            qo.data_ptr(), ko.data_ptr(), B, S, Hq, k.shape[2], D, I64x3(*q.stride()[:3]),
            I64x3(*k.stride()[:3]), I64x3(*qo.stride()[:3]), I64x3(*ko.stride()[:3]),
            cos2.stride(0), _code(cos2), _code(q), int(bool(inverse)))
    return qo, ko


# ----------------------------------------------------------------------------- GLU
def glu(x: torch.Tensor, act: str) -> torch.Tensor:
    """x (..., 2H) -> (..., H): x[..., :H] * act(x[..., H:]); act in swiglu/geglu/reglu."""
    dev = _need_cuda(x)
    two_h = x.shape[-1]
    if two_h % 2:
        raise ValueError("last dimension must be even")
    h = two_h // 2
    x2, rows, stride = _rows(x)
    y = _empty(x, (*x.shape[:-1], h))
    up = x2.data_ptr()
    _launch("trx_glu_fwd", dev, up, up + h * x2.element_size(), y.data_ptr(), rows, h, stride, stride, h,
            GLU_ACTS[act], _code(x2))
    return y


def glu_pair(up: torch.Tensor, gate: torch.Tensor, act: str) -> torch.Tensor:
    """Separate up / gate tensors of equal shape (..., H) -> up * act(gate)."""
    dev = _need_cuda(up, gate)
    if up.shape != gate.shape or up.dtype != gate.dtype:
        raise ValueError("up and gate must have the same shape and dtype")
    (u2, rows, u_stride), (g2, _, g_stride) = _rows(up), _rows(gate)
    h, y = up.shape[-1], _new(up)
    _launch("trx_glu_fwd", dev, u2.data_ptr(), g2.data_ptr(), y.data_ptr(), rows, h, u_stride, g_stride,
            h, GLU_ACTS[act], _code(u2))
    return y


# ----------------------------------------------------------------------------- backward
def glu_backward(dy: torch.Tensor, x: torch.Tensor, act: str) -> torch.Tensor:
    """Gradient of glu(x, act) with respect to x (..., 2H), given dy (..., H): the two halves
    dy * act(gate) and dy * up * act'(gate) written into one tensor of x's shape."""
    dev = _need_cuda(dy, x)
    h = x.shape[-1] // 2
    if x.shape[-1] % 2 or dy.shape != x.shape[:-1] + (h,) or dy.dtype != x.dtype:
        raise ValueError("dy must have x's leading shape, half its last dimension and its dtype")
    (x2, rows, stride), (dy2, _, dy_stride) = _rows(x), _rows(dy)
    dx = _new(x)
    off = h * x2.element_size()
    _launch("trx_glu_bwd", dev, dy2.data_ptr(), x2.data_ptr(), x2.data_ptr() + off, dx.data_ptr(),
            dx.data_ptr() + off, rows, h, dy_stride, stride, stride, 2 * h, 2 * h, GLU_ACTS[act],
            _code(x2))
    return dx


def _stat(t: torch.Tensor, rows: int) -> torch.Tensor:
    if t.dtype != torch.float32 or t.numel() != rows:
        raise ValueError("row statistics must be float32, one per row")
    return t.contiguous()


def _norm_bwd_workspace(x: torch.Tensor, rows: int, cols: int) -> torch.Tensor:
    return _empty(x, _lib.load().trx_norm_bwd_workspace_bytes(rows, cols), dtype=torch.uint8)


def rmsnorm_backward(dy: torch.Tensor, x: torch.Tensor, weight: torch.Tensor, eps: float = 1e-6,
                     need_dw: bool = True, residual: Optional[torch.Tensor] = None,
                     activation: Optional[str] = None, rstd: Optional[torch.Tensor] = None):
    """(dx, dw) of rmsnorm(x, weight, eps) given dy; dw is None when need_dw is False. The row
    statistics are recomputed from x unless the forward's `rstd` is given (not with an
    activation); dw is summed in fp32 in a fixed order. With `residual`, the
    gradient of residual_rmsnorm(x, residual, ...): dx is then also the residual's gradient. With
    `activation`, the gradient of rmsnorm_activation(x, weight, eps, activation)."""
    if activation is not None and activation not in ROW_ACTIVATIONS:
        raise ValueError(f"Unsupported activation '{activation}'. "
                         f"Supported: {sorted(ROW_ACTIVATIONS)}")
    if activation is not None and residual is not None:
        raise ValueError("residual and activation cannot be combined")
    if activation is not None and rstd is not None:
        raise ValueError("rstd and activation cannot be combined")
    dev = _need_cuda(dy, x, weight, residual, rstd)
    if dy.shape != x.shape or dy.dtype != x.dtype:
        raise ValueError("dy must have the shape and dtype of x")
    if residual is not None:
        _check_residual(x, residual)
    _check_weight(weight, x)
    (x2, rows, stride), (dy2, _, dy_stride) = _rows(x), _rows(dy)
    r2, _, r_stride = _rows(residual) if residual is not None else (None, 0, x.shape[-1])
    w, c, dx = _dense(weight), x.shape[-1], _new(x)
    dw = _new(w) if need_dw else None
    ws = _norm_bwd_workspace(x, rows, c)
    tail = (_code(x2), _code(w), ws.data_ptr(), ws.numel())
    if activation is not None:
        _launch("trx_rmsnorm_act_bwd", dev, dy2.data_ptr(), x2.data_ptr(), w.data_ptr(), dx.data_ptr(),
                _ptr(dw), rows, c, dy_stride, stride, c, float(eps), ROW_ACTIVATIONS[activation], *tail)
    elif rstd is not None:
        rstd = _stat(rstd, rows)
        _launch("trx_rmsnorm_bwd_saved", dev, dy2.data_ptr(), x2.data_ptr(), _ptr(r2), w.data_ptr(),
                rstd.data_ptr(), dx.data_ptr(), _ptr(dw), rows, c, dy_stride, stride, r_stride, c, *tail)
    elif residual is None:
        _launch("trx_rmsnorm_bwd", dev, dy2.data_ptr(), x2.data_ptr(), w.data_ptr(), dx.data_ptr(),
                _ptr(dw), rows, c, dy_stride, stride, c, float(eps), *tail)
    else:
        _launch("trx_residual_rmsnorm_bwd", dev, dy2.data_ptr(), x2.data_ptr(), r2.data_ptr(),
                w.data_ptr(), dx.data_ptr(), _ptr(dw), rows, c, dy_stride, stride, r_stride, c,
                float(eps), *tail)
    return dx, dw


def layernorm_backward(dy: torch.Tensor, x: torch.Tensor, weight: Optional[torch.Tensor],
                       eps: float = 1e-5, need_dw: bool = True, need_db: bool = True,
                       residual: Optional[torch.Tensor] = None,
                       mean: Optional[torch.Tensor] = None, rstd: Optional[torch.Tensor] = None):
    """(dx, dw, db) of layernorm(x, weight, bias, eps) given dy; weight may be None (then dw is
    None); db is returned in the weight's dtype (x's dtype without a weight). The row statistics
    are recomputed from x unless the forward's `mean` and `rstd` are given. With `residual`,
    the gradient of residual_layernorm(x, residual, ...): dx is then also the residual's."""
    dev = _need_cuda(dy, x, weight, residual, mean, rstd)
    if (mean is None) != (rstd is None):
        raise ValueError("mean and rstd come together")
    if dy.shape != x.shape or dy.dtype != x.dtype:
        raise ValueError("dy must have the shape and dtype of x")
    if residual is not None:
        _check_residual(x, residual)
    if weight is not None and weight.numel() != x.shape[-1]:
        raise ValueError("weight size does not match the normalised dim")
    (x2, rows, stride), (dy2, _, dy_stride) = _rows(x), _rows(dy)
    r2, _, r_stride = _rows(residual) if residual is not None else (None, 0, x.shape[-1])
    w, c, dx = _dense(weight), x.shape[-1], _new(x)
    p_dtype = w.dtype if w is not None else x.dtype
    dw = _empty(w, c) if need_dw and w is not None else None
    db = _empty(x, c, dtype=p_dtype) if need_db else None
    ws = _norm_bwd_workspace(x, rows, c)
    tail = (_code(x2), _DTYPE_CODE[p_dtype], ws.data_ptr(), ws.numel())
    if rstd is not None:
        mean, rstd = _stat(mean, rows), _stat(rstd, rows)
        _launch("trx_layernorm_bwd_saved", dev, dy2.data_ptr(), x2.data_ptr(), _ptr(r2), _ptr(w),
                mean.data_ptr(), rstd.data_ptr(), dx.data_ptr(), _ptr(dw), _ptr(db), rows, c, dy_stride,
                stride, r_stride, c, *tail)
    elif residual is None:
        _launch("trx_layernorm_bwd", dev, dy2.data_ptr(), x2.data_ptr(), _ptr(w), dx.data_ptr(), _ptr(dw),
                _ptr(db), rows, c, dy_stride, stride, c, float(eps), *tail)
    else:
        _launch("trx_residual_layernorm_bwd", dev, dy2.data_ptr(), x2.data_ptr(), r2.data_ptr(), _ptr(w),
                dx.data_ptr(), _ptr(dw), _ptr(db), rows, c, dy_stride, stride, r_stride, c, float(eps),
                *tail)
    return dx, dw, db


# ----------------------------------------------------------------------------- attention
_workspaces: dict = {}
_status_host: dict = {}  # device index -> pinned int32[1] mirror of the status word
_status_word: dict = {}  # device index -> the mirror as a ctypes integer: read on every call
_workspace_lock = threading.Lock()  # held by the thread that makes a device's three


def _dev_index(dev: torch.device) -> int:
    return dev.index if dev.index is not None else torch.cuda.current_device()


def _workspace(dev: torch.device) -> torch.Tensor:
    """The device's attention workspace: 256 zeroed bytes that every call on the device shares, with
    a pinned host word attached that a failing launch writes. Whichever thread comes first makes
    both; they are published when the set-up has run, so any thread and stream may use them (a first
    call under stream capture, which cannot be waited for, makes the set-up part of its graph)."""
    idx = _dev_index(dev)
    ws = _workspaces.get(idx)
    if ws is None:
        with _workspace_lock:
            ws = _workspaces.get(idx)
            if ws is None:
                ws = _make_workspace(idx)
    return ws


def _make_workspace(idx: int) -> torch.Tensor:
    n = int(_lib.load().trx_attn_workspace_bytes())
    host = torch.zeros(1, dtype=torch.int32).pin_memory()
    with torch.cuda.device(idx):
        ws = torch.zeros(n, dtype=torch.uint8, device=torch.device("cuda", idx))
        _lib.check("trx_attn_mirror", _lib.load().trx_attn_mirror(
            ws.data_ptr(), host.data_ptr(), _raw_stream(idx)))
        if not torch.cuda.is_current_stream_capturing():
            torch.cuda.current_stream(idx).synchronize()
    _status_host[idx] = host
    _status_word[idx] = ctypes.c_int32.from_address(host.data_ptr())
    _workspaces[idx] = ws  # last: a thread that finds it finds the words too
    return ws


def _clear_status(dev: torch.device) -> None:
    """Zero both copies of the status word. Launches queued before the device's copy is cleared still
    find the failure and write the host's copy, so that one is cleared when none of them is left."""
    _workspace(dev)[:4].zero_()
    torch.cuda.synchronize(dev)
    _status_host[_dev_index(dev)].zero_()


def _raise_if_failed(fn: str, dev: torch.device) -> None:
    """Host-side check of the status word's pinned mirror; no synchronisation while it is zero. A
    kernel that gave up on a bounded wait has written it, and so has every launch after it: they
    skipped their work and left their outputs unwritten. Both copies of the word are cleared, behind
    whatever is in flight, and the failure is raised: once, and the next call runs again (under
    stream capture, where nothing can be waited for, it is raised and stays). Outputs returned since
    the failing launch must be discarded."""
    word = _status_word[_dev_index(dev)].value
    if word:
        if not torch.cuda.is_current_stream_capturing():
            _clear_status(dev)
        raise _lib.TrinixB200Error(
            fn, _lib.TRX_ERR_DEVICE_STATUS,
            f"{_lib.load().trx_status_string(_lib.TRX_ERR_DEVICE_STATUS).decode()} "
            f"(status word {word:#x}); attention outputs produced since then are invalid")


def attention_status(device=None) -> int:
    """Status word of the attention workspace on `device` (synchronises). Non-zero means a
    bounded on-chip wait gave up in some earlier launch; the word is then cleared."""
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    ws = _workspace(dev)
    word = int(ws[:4].view(torch.int32).item())  # .item() waits for the stream
    if word:
        _clear_status(dev)
    else:
        _status_host[_dev_index(dev)].zero_()
    return word


def dropout_seed() -> int:
    """A fresh 62-bit seed for one dropout call, drawn from torch's CPU generator: reproducible
    under torch.manual_seed, and no device synchronisation (the reference draws its seed with
    `.item()` on a CUDA tensor, trinix/kernels/attention_kernel.py:526-532)."""
    return int(torch.randint(0, 2 ** 62, (1,), dtype=torch.int64).item())


def _dense_mask(mask: torch.Tensor, B: int, Hq: int, Sq: int, Sk: int, act_dtype):
    """The mask as the kernel reads it: fp32 or the activation dtype, unit key stride, and the
    (batch, head, query) element strides of its broadcast view (shape rules of
    TritonAttentionKernel._prepare_mask, trinix/kernels/attention_kernel.py:479-495)."""
    m = mask.detach()
    if m.dtype == torch.bool:
        m = torch.zeros(m.shape, dtype=torch.float32, device=m.device).masked_fill_(m, float("-inf"))
    elif m.dtype not in (torch.float32, act_dtype):
        m = m.to(torch.float32)
    if m.dim() == 2:
        m = m[None, None]
    elif m.dim() == 3:
        m = m[:, None]
    elif m.dim() != 4:
        raise ValueError(f"Unsupported mask shape: {tuple(mask.shape)}")
    if m.shape[-2:] != (Sq, Sk) or m.shape[0] not in (1, B) or m.shape[1] not in (1, Hq):
        raise ValueError(f"mask shape {tuple(mask.shape)} does not broadcast to "
                         f"({B}, {Hq}, {Sq}, {Sk})")
    if m.stride(-1) != 1 and Sk > 1:
        m = m.contiguous()
    sb = 0 if m.shape[0] == 1 else m.stride(0)
    sh = 0 if m.shape[1] == 1 else m.stride(1)
    sq = m.stride(2) if Sq > 1 else max(Sk, m.stride(2))
    if sq < Sk:  # an expanded query dim: materialise, the kernel wants real rows
        m = m.contiguous()
        sb = 0 if m.shape[0] == 1 else m.stride(0)
        sh = 0 if m.shape[1] == 1 else m.stride(1)
        sq = m.stride(2)
    return m, (sb, sh, sq)


def attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, causal: bool = False,
              scale: Optional[float] = None, window: Optional[Tuple[int, int]] = None,
              alibi_slopes: Optional[torch.Tensor] = None, return_lse: bool = False,
              attn_mask: Optional[torch.Tensor] = None, dropout_p: float = 0.0,
              seed: Optional[int] = None, offset: int = 0):
    """softmax(scale * q k^T + bias) v; q (B,Sq,Hq,D), k/v (B,Sk,Hk,D), Hq % Hk == 0.

    Query head h reads kv head h // (Hq // Hk). window = (left, right) keeps keys with
    -left <= j - i <= right. alibi_slopes (Hq,) adds -slope * |i - j|. attn_mask is a dense
    additive mask (Sq,Sk), (B,Sq,Sk), (B,1,Sq,Sk) or (B,Hq,Sq,Sk), float (added to the scaled
    scores) or bool (True = hidden), broadcast by stride, never expanded. dropout_p in [0, 1)
    drops normalised probabilities (realised in steps of 1/256) with a Philox stream keyed by
    `seed` (drawn from torch's CPU generator when None) and `offset`; see dropout_seed().
    """
    dev = _need_cuda(q, k, v, alibi_slopes, attn_mask)
    if not (q.dtype == k.dtype == v.dtype) or q.dtype not in (torch.bfloat16, torch.float16):
        raise TypeError("attention needs q, k, v of one dtype, bfloat16 or float16")
    if q.dim() == 4 and q.shape[-1] not in (64, 128) and 0 < q.shape[-1] < 128:
        # The kernel is built for head dims 64 and 128. Any smaller one runs as the next of the
        # two with zero columns appended: they add nothing to q.k and produce output columns that
        # are cut off again. Costs one padded copy of q, k, v; the scale keeps the true head dim.
        d_true = q.shape[-1]
        d_pad = 64 if d_true < 64 else 128
        if scale is None:
            scale = d_true ** -0.5
        pad = lambda t: torch.nn.functional.pad(t, (0, d_pad - d_true))
        res = attention(pad(q), pad(k), pad(v), causal=causal, scale=scale, window=window,
                        alibi_slopes=alibi_slopes, return_lse=return_lse, attn_mask=attn_mask,
                        dropout_p=dropout_p, seed=seed, offset=offset)
        if return_lse:
            return res[0][..., :d_true].contiguous(), res[1]
        return res[..., :d_true].contiguous()
    q, k, v = _tma_view(q), _tma_view(k), _tma_view(v)
    B, Sq, Hq, D = q.shape
    Bk, Sk, Hk, Dk = k.shape
    if (Bk, Dk) != (B, D) or v.shape != k.shape:
        raise ValueError(f"k {tuple(k.shape)} / v {tuple(v.shape)} do not match q {tuple(q.shape)}")
    if Hk == 0 or Hq % Hk:
        raise ValueError(f"query heads ({Hq}) must be a multiple of kv heads ({Hk})")
    if scale is None:
        scale = D ** -0.5
    wl, wr = (-1, -1)
    if window is not None:
        wl, wr = int(window[0]), int(window[1])
        if wl < 0 or wr < 0:
            raise ValueError("window sizes must be >= 0")
    slopes = None
    if alibi_slopes is not None:
        slopes = alibi_slopes.detach().reshape(-1).to(torch.float32).contiguous()
        if slopes.numel() != Hq:
            raise ValueError(f"alibi_slopes must have {Hq} entries")
    out = _new(q)
    lse = _empty(q, (B, Hq, Sq), dtype=torch.float32) if return_lse else None
    ws = _workspace(dev)
    # a failure recorded by an earlier launch surfaces here, before more work is queued
    _raise_if_failed("trx_attn_fwd", dev)
    head = (q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), _ptr(lse), _ptr(slopes))
    problem = (B, Sq, Sk, Hq, Hk, D, I64x3(*q.stride()[:3]), I64x3(*k.stride()[:3]),
               I64x3(*v.stride()[:3]), I64x3(*out.stride()[:3]), float(scale), int(bool(causal)), wl,
               wr, _code(q))
    work = (ws.data_ptr(), ws.numel())
    mask = (0, 0, I64x3(0, 0, Sk))
    if dropout_p and not 0.0 <= dropout_p < 1.0:
        raise ValueError(f"dropout_p must be in [0, 1), got {dropout_p}")
    if dropout_p and seed is None:
        seed = dropout_seed()
    if attn_mask is not None:
        m, strides = _dense_mask(attn_mask, B, Hq, Sq, Sk, q.dtype)  # m lives past the launch
        mask = (m.data_ptr(), _code(m), I64x3(*strides))
    if dropout_p:
        _launch("trx_attn_fwd_dropout", dev, *head, *mask, *problem, float(dropout_p),
                int(seed) & (2 ** 64 - 1), int(offset) & 0xFFFFFFFF, *work)
    elif attn_mask is not None:
        _launch("trx_attn_fwd_mask", dev, *head, *mask, *problem, *work)
    else:
        _launch("trx_attn_fwd", dev, *head, *problem, *work)
    return (out, lse) if return_lse else out
