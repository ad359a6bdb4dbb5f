"""Host-side mirror of the reference's operator interface for the dense hot path.

Function names and argument meaning follow yt::YTensor / yt::function in the reference
(matmul, linear, scaledDotProductAttention, softmax, rmsNorm, layerNorm, sum/mean/max, cast);
tensors are torch tensors that only serve as device memory with a shape and strides. Every
function calls the C ABI of libytensor_cuda.so; nothing here computes with torch.
"""
from __future__ import annotations

import builtins
import struct

import torch

from . import _lib
from ._lib import BF16, F16, F32, check, lib

_DT = {torch.float32: F32, torch.bfloat16: BF16, torch.float16: F16}


# What a call costs on the host is most of what a small operator costs (the kernels take 2 us): shapes and strides go to the
# library as packed bytes, results are allocated once, broadcasting is arithmetic on the strides instead of views, and the
# stream is asked for as a number. bias [1024] added to [7, 1024]: 33 us a call before, see the table of cases.
_PACK64 = [struct.Struct(f"{n}q").pack for n in range(65)]
_PACK32 = [struct.Struct(f"{n}i").pack for n in range(65)]


def _dt(t: torch.Tensor) -> int:
    try:
        return _DT[t.dtype]
    except KeyError:
        raise _lib.YtCudaInvalidArgument(_lib.UNSUPPORTED, f"unsupported dtype {t.dtype}")


def _stream() -> int:
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _require_cuda(*ts: torch.Tensor) -> None:
    for t in ts:
        if t is not None and not t.is_cuda:
            raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "device backend: tensor is not on a CUDA device")


def _broadcast(a: torch.Tensor, b: torch.Tensor):
    """Common shape of a and b, and the strides with which each of them is read in it (torch's expand)."""
    sa, sb, ta, tb = tuple(a.shape), tuple(b.shape), a.stride(), b.stride()
    if sa == sb:
        return sa, ta, tb
    na, nb = len(sa), len(sb)
    if nb <= na and sa[na - nb:] == sb:
        return sa, ta, (0,) * (na - nb) + tb
    n = na if na > nb else nb
    shape, xa, xb = [0] * n, [0] * n, [0] * n
    for i in range(1, n + 1):
        x = sa[na - i] if i <= na else 1
        y = sb[nb - i] if i <= nb else 1
        if x != y and x != 1 and y != 1:
            torch.broadcast_shapes(sa, sb)  # (raises, with the sizes)
        size = y if x == 1 else x
        shape[n - i] = size
        if i <= na and x == size:
            xa[n - i] = ta[na - i]
        if i <= nb and y == size:
            xb[n - i] = tb[nb - i]
    return tuple(shape), tuple(xa), tuple(xb)


def _batch_view(lead_shape, lead_stride):
    """(batch count, batch stride) if the leading dims collapse into one stride; None otherwise."""
    dims = [(n, s) for n, s in zip(lead_shape, lead_stride) if n != 1]
    if not dims:
        return 1, 0
    count, stride = dims[-1]
    for n, s in reversed(dims[:-1]):
        if s != stride * count and not (s == 0 and stride == 0):
            return None
        count *= n
    return count, stride


def matmul(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor | None = None, *, alpha: float = 1.0,
           beta: float = 0.0, out_dtype: torch.dtype | None = None) -> torch.Tensor:
    """C[..., m, n] = A[..., m, k] . B[..., k, n] with broadcast batch dims.

    Mirrors YTensor<T,dim>::matmul (reference src/ytensor_math.inl:284-316): the last dim of
    `a` must equal the second-to-last of `b` or std::invalid_argument (here ValueError) is raised.
    One batched launch replaces the reference's per-matrix loop (:1035-1049).
    """
    return _product(a, b, False, out, alpha, beta, out_dtype)


def _product(a: torch.Tensor, b: torch.Tensor, turned: bool, out=None, alpha: float = 1.0, beta: float = 0.0,
             out_dtype=None) -> torch.Tensor:
    """matmul; turned: b holds [..., n, k]."""
    _require_cuda(a, b, out)
    sa, sb, ta, tb = tuple(a.shape), tuple(b.shape), a.stride(), b.stride()
    if not sa or not sb:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "matmul: operands must have at least 1 dim")
    if len(sa) == 1:
        sa, ta = (1, *sa), (sa[0] * ta[0], *ta)
    if len(sb) == 1:
        sb, tb = (*sb, 1), (*tb, 1)
    m, k = sa[-2:]
    ra, ca = ta[-2:]
    if turned:
        n, kb = sb[-2:]
        cb, rb = tb[-2:]
    else:
        kb, n = sb[-2:]
        rb, cb = tb[-2:]
    if k != kb:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, f"matmul: inner dims differ ({k} vs {kb})")
    dt = a.dtype
    if dt != b.dtype:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "matmul: operand dtypes differ")
    la, lb = sa[:-2], sb[:-2]
    if la == lb or not lb:
        lead, xa, xb = la, ta[:-2], tb[:-2] if lb else (0,) * len(la)
    elif not la:
        lead, xa, xb = lb, (0,) * len(lb), tb[:-2]
    else:
        lead = torch.broadcast_shapes(la, lb)
        xa, xb = a.reshape(sa).expand(*lead, m, k).stride()[:-2], b.reshape(sb).expand(*lead, *sb[-2:]).stride()[:-2]
    if out is None:
        out = torch.empty(*lead, m, n, dtype=out_dtype or dt, device=a.device)
    elif tuple(out.shape) != (*lead, m, n):
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "matmul: out has the wrong shape")
    to = out.stride()
    av, bv, ov = (_batch_view(lead, x) for x in (xa, xb, to[:-2])) if lead else ((1, 0),) * 3
    if av is not None and bv is not None and ov is not None:
        check(lib().ytcuda_gemm(_dt(a), _dt(out), a.data_ptr(), b.data_ptr(), out.data_ptr(), m, n, k, alpha, beta, ra, ca,
                                rb, cb, to[-2], to[-1], builtins.max(av[0], bv[0], ov[0]), av[1], bv[1], ov[1], _stream()))
    else:
        # Leading dims that do not collapse into one stride: one call per outermost slice.
        ae, be = a.reshape(sa).expand(*lead, m, k), b.reshape(sb).expand(*lead, *sb[-2:])
        for idx in range(lead[0]):
            _product(ae[idx], be[idx], turned, out[idx], alpha, beta)
    return out


class Causal:
    """The predicate j <= i + offset, for the predicate forms of masked_matmul and scaledDotProductAttention
    (reference src/ytensor_math.inl:368-412, src/function/ops.inl:427-503): evaluated on the device, no mask tensor."""

    def __init__(self, offset: int = 0):
        self.offset = int(offset)

    def __call__(self, i: int, j: int) -> bool:
        return j <= i + self.offset


def masked_matmul(a: torch.Tensor, b: torch.Tensor, mask, masked_value: float = 0.0, *,
                  out_dtype: torch.dtype | None = None) -> torch.Tensor:
    """C[..., i, j] = (A . B)[..., i, j] where mask[i, j], masked_value elsewhere; mask is bool [m, n], a `Causal`
    predicate (evaluated on the device), or any callable (i, j) -> bool (materialised once into a bool mask).

    Mirrors YTensor<T,dim>::masked_matmul with a bool mask or a predicate (reference src/ytensor_math.inl:318-412): a
    mask of another shape is refused as the reference refuses it (std::invalid_argument, here ValueError). Output
    tiles in which the mask holds nowhere are not computed.
    """
    causal = mask if isinstance(mask, Causal) else None
    if causal is None and callable(mask) and not isinstance(mask, torch.Tensor):
        mm, nn = a.shape[-2], b.shape[-1]
        mask = torch.tensor([[bool(mask(i, j)) for j in range(nn)] for i in range(mm)], dtype=torch.bool,
                            device=a.device)
    _require_cuda(a, b, None if causal else mask)
    if a.dim() < 2 or b.dim() < 2:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "masked_matmul: operands must have at least 2 dims")
    if a.shape[-1] != b.shape[-2]:
        raise _lib.YtCudaInvalidArgument(
            _lib.INVALID_ARG, f"masked_matmul: inner dims differ ({a.shape[-1]} vs {b.shape[-2]})")
    m, k = a.shape[-2:]
    n = b.shape[-1]
    if causal is None:
        if mask.dtype != torch.bool or tuple(mask.shape) != (m, n):
            raise _lib.YtCudaInvalidArgument(
                _lib.INVALID_ARG, f"masked_matmul: mask must be bool [{m}, {n}], got {mask.dtype} {tuple(mask.shape)}")
        if mask.stride(1) != 1:
            mask = mask.contiguous()
    bshape = torch.broadcast_shapes(a.shape[:-2], b.shape[:-2])
    ae, be = a.expand(*bshape, m, k), b.expand(*bshape, k, n)
    out = torch.empty(*bshape, m, n, dtype=out_dtype or a.dtype, device=a.device)
    av, bv, ov = (_batch_view(t.shape[:-2], t.stride()[:-2]) for t in (ae, be, out))
    if av is None or bv is None or ov is None:
        for idx in range(bshape[0]):
            out[idx] = masked_matmul(ae[idx], be[idx], mask, masked_value, out_dtype=out_dtype)
        return out
    batch = builtins.max(av[0], bv[0], ov[0])
    if causal is not None:
        check(lib().ytcuda_gemm_masked_causal(_dt(ae), _dt(out), ae.data_ptr(), be.data_ptr(), out.data_ptr(), m, n, k,
                                              ae.stride(-2), ae.stride(-1), be.stride(-2), be.stride(-1),
                                              out.stride(-2), out.stride(-1), batch, av[1], bv[1], ov[1],
                                              causal.offset, float(masked_value), _stream()))
        return out
    check(lib().ytcuda_gemm_masked(_dt(ae), _dt(out), ae.data_ptr(), be.data_ptr(), out.data_ptr(), m, n, k,
                                   ae.stride(-2), ae.stride(-1), be.stride(-2), be.stride(-1), out.stride(-2),
                                   out.stride(-1), batch, av[1], bv[1], ov[1], mask.data_ptr(), mask.stride(0),
                                   float(masked_value), _stream()))
    return out


def linear(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None = None) -> torch.Tensor:
    """x . weight^T (+ bias), weight [out_features, in_features] (reference src/function/ops.inl:84-105)."""
    y = _product(x, weight, True) if weight.dim() >= 2 else matmul(x, weight.transpose(-1, -2))
    if bias is not None:
        add_(y, bias)
    return y


# ------------------------------------------------------------------ N-d helpers
def _i64(vals) -> bytes:
    return _PACK64[len(vals)](*vals)


def _i32(vals) -> bytes:
    return _PACK32[len(vals)](*vals)


def _axes(axes) -> list[int]:
    return [axes] if type(axes) is int else [int(axes)] if isinstance(axes, int) else [int(a) for a in axes]


def _nd(t: torch.Tensor):
    """(dims, shape, strides) as the library takes them; a scalar counts as one element."""
    n = t.dim()
    return (n, _i64(t.shape), _i64(t.stride())) if n else (1, _i64((1,)), _i64((1,)))


def _like(x: torch.Tensor, dtype: torch.dtype | None = None) -> torch.Tensor:
    return torch.empty_like(x, dtype=dtype, memory_format=torch.contiguous_format)


# ------------------------------------------------------------------ softmax / norms
def softmax(x: torch.Tensor, axes=-1, out: torch.Tensor | None = None) -> torch.Tensor:
    """Softmax jointly over `axes` (reference yt::function::softmax, src/function/activation.inl:336-375)."""
    _require_cuda(x, out)
    y = _like(x) if out is None else out
    ax = _axes(axes)
    nd, shape, xs = _nd(x)
    check(lib().ytcuda_softmax(_dt(x), _dt(y), x.data_ptr(), y.data_ptr(), shape, xs, _i64(y.stride() or (1,)),
                               nd, _i32(ax), len(ax), _stream()))
    return y


def softmax_(x: torch.Tensor, axes=-1) -> torch.Tensor:
    """In-place form (reference yt::function::softmax_, src/function/activation.inl:376-409)."""
    return softmax(x, axes, out=x)


def rmsNorm(x: torch.Tensor, weight: torch.Tensor | None, axes=-1, eps: float = 1e-5,
            out: torch.Tensor | None = None) -> torch.Tensor:
    """x / sqrt(mean(x^2) + eps) * weight (reference yt::function::rmsNorm, src/function/normalization.inl:234-277).
    `weight` has one dim per axis; a shape mismatch raises like the reference's _makeAffineView."""
    _require_cuda(x, weight, out)
    ax = _axes(axes)
    if weight is not None:
        want = [x.shape[a] for a in ax]
        if list(weight.shape) != want:
            raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "rmsNorm: weight shape must match affine axes")
        weight = weight.contiguous()
    y = _like(x) if out is None else out
    nd, shape, xs = _nd(x)
    check(lib().ytcuda_rmsnorm(_dt(x), _dt(y), _dt(weight) if weight is not None else F32, x.data_ptr(),
                               weight.data_ptr() if weight is not None else None, y.data_ptr(), shape, xs,
                               _i64(y.stride() or (1,)), nd, _i32(ax), len(ax), eps, _stream()))
    return y


def rmsNorm_(x, weight, axes=-1, eps: float = 1e-5):
    return rmsNorm(x, weight, axes, eps, out=x)


def layerNorm(x: torch.Tensor, gamma: torch.Tensor | None = None, bias: torch.Tensor | None = None, axes=-1,
              eps: float = 1e-5, out: torch.Tensor | None = None) -> torch.Tensor:
    """(x - mean) / sqrt(var + eps) [* gamma + bias] (reference yt::function::layerNorm,
    src/function/normalization.inl:159-230)."""
    _require_cuda(x, gamma, bias, out)
    ax = _axes(axes)
    if (gamma is None) != (bias is None):
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "layerNorm: gamma and bias come together")
    if gamma is not None:
        want = [x.shape[a] for a in ax]
        if list(gamma.shape) != want or list(bias.shape) != want:
            raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "layerNorm: gamma/bias shape must match affine axes")
        gamma, bias = gamma.contiguous(), bias.contiguous().to(gamma.dtype)
    y = _like(x) if out is None else out
    nd, shape, xs = _nd(x)
    check(lib().ytcuda_layernorm(_dt(x), _dt(y), _dt(gamma) if gamma is not None else F32, x.data_ptr(),
                                 gamma.data_ptr() if gamma is not None else None,
                                 bias.data_ptr() if bias is not None else None, y.data_ptr(), shape, xs,
                                 _i64(y.stride() or (1,)), nd, _i32(ax), len(ax), eps, _stream()))
    return y


def layerNorm_(x, gamma=None, bias=None, axes=-1, eps: float = 1e-5):
    return layerNorm(x, gamma, bias, axes, eps, out=x)


def _check_affine(y: torch.Tensor, gamma, bias, ax) -> None:
    if gamma is None or bias is None:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "gamma and bias come together")
    want = [y.shape[a] for a in ax]
    if list(gamma.shape) != want or list(bias.shape) != want:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "gamma/bias shape must match affine axes")


def _affine_(y: torch.Tensor, gamma, bias, axes) -> torch.Tensor:
    """y *= gamma; y += bias with gamma / bias holding one dim per axis (the reference's _applyScale_ / _applyBias_,
    src/function/normalization.inl:88-116, through _makeAffineView)."""
    if gamma is None and bias is None:
        return y
    ax = [a % y.dim() for a in axes]
    _check_affine(y, gamma, bias, ax)
    # the reference views the affine tensor's MEMORY with the axis sizes in ascending axis order, whatever order the
    # axes were listed in (src/ytensor_function.inl:137-158): a plain reshape of the contiguous tensor does the same
    view = [1] * y.dim()
    for a in ax:
        view[a] = y.shape[a]
    g = gamma.contiguous().reshape(view)
    b = bias.contiguous().reshape(view)
    _binary("mul", y, g.to(y.dtype), y)
    _binary("add", y, b.to(y.dtype), y)
    return y


def _channel_norm(x: torch.Tensor, y: torch.Tensor, shape, xt, yt, axes, eps: float, gamma, bias, channel: int,
                  wstrides) -> torch.Tensor:
    """layerNorm of x over `axes` into y, then gamma and bias of the channels (axis `channel`). x and y are read as
    shape / xt and shape / yt, which may group the channels; `wstrides` says how far a step of each of those dims moves in
    gamma. One launch where the strides allow it, else three."""
    if gamma is not None and bias is not None and gamma.is_cuda and bias.is_cuda:
        _check_affine(y, gamma, bias, [channel])
        _require_cuda(x, y)
        g, b = gamma.contiguous().to(y.dtype), bias.contiguous().to(y.dtype)
        rc = lib().ytcuda_layernorm_strided(_dt(x), _dt(y), _dt(y), x.data_ptr(), g.data_ptr(), b.data_ptr(), y.data_ptr(),
                                            _i64(shape), _i64(xt), _i64(yt), _i64(wstrides), len(shape), _i32(axes),
                                            len(axes), eps, _stream())
        if rc != _lib.UNSUPPORTED:
            check(rc)
            return y
    layerNorm(x.as_strided(shape, xt), None, None, axes, eps, out=y.as_strided(shape, yt))
    return _affine_(y, gamma, bias, [channel])


def normalize(x: torch.Tensor, axes=-1, p: float = 2.0, eps: float = 1e-12, gamma=None, bias=None,
              out: torch.Tensor | None = None) -> torch.Tensor:
    """x / (sum_axes |x|^p + eps)^(1/p) [* gamma + bias] (reference yt::function::normalize,
    src/function/normalization.inl:56-85, 278-372)."""
    _require_cuda(x, gamma, bias, out)
    if p <= 0:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "yt::function::normalize: p must be positive")
    ax = _axes(axes)
    y = _like(x) if out is None else out
    nd, shape, xs = _nd(x)
    check(lib().ytcuda_normalize(_dt(x), _dt(y), x.data_ptr(), y.data_ptr(), shape, xs, _i64(y.stride() or (1,)),
                                 nd, _i32(ax), len(ax), float(p), float(eps), _stream()))
    return _affine_(y, gamma, bias, ax)


def normalize_(x, axes=-1, p: float = 2.0, eps: float = 1e-12, gamma=None, bias=None):
    return normalize(x, axes, p, eps, gamma, bias, out=x)


def _channel_axis(x: torch.Tensor, channelAxis: int, who: str) -> int:
    c = channelAxis % x.dim()
    if x.dim() < 2:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, f"{who} requires dim >= 2")
    if c == 0:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, f"{who}: channelAxis must not be batch axis 0")
    return c


def instanceNorm(x: torch.Tensor, gamma=None, bias=None, channelAxis: int = 1, eps: float = 1e-5,
                 out: torch.Tensor | None = None) -> torch.Tensor:
    """Standardises every (sample, channel) over the remaining axes (reference yt::function::instanceNorm,
    src/function/normalization.inl:378-433); gamma / bias are per channel."""
    c = _channel_axis(x, channelAxis, "yt::function::instanceNorm_")
    axes = [a for a in range(x.dim()) if a not in (0, c)]
    if not axes:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "yt::function::instanceNorm: requires at least one spatial axis")
    y = _like(x) if out is None else out
    return _channel_norm(x, y, x.shape, x.stride(), y.stride(), axes, eps, gamma, bias, c, [int(a == c) for a in range(x.dim())])


def instanceNorm_(x, gamma=None, bias=None, channelAxis: int = 1, eps: float = 1e-5):
    return instanceNorm(x, gamma, bias, channelAxis, eps, out=x)


def batchNorm(x: torch.Tensor, gamma=None, bias=None, channelAxis: int = 1, eps: float = 1e-5,
              out: torch.Tensor | None = None) -> torch.Tensor:
    """Standardises every channel over all other axes, batch included (reference yt::function::batchNorm,
    src/function/normalization.inl:435-489: statistics of the tensor itself, no running averages)."""
    c = _channel_axis(x, channelAxis, "yt::function::batchNorm_")
    axes = [a for a in range(x.dim()) if a != c]
    y = _like(x) if out is None else out
    return _channel_norm(x, y, x.shape, x.stride(), y.stride(), axes, eps, gamma, bias, c, [int(a == c) for a in range(x.dim())])


def batchNorm_(x, gamma=None, bias=None, channelAxis: int = 1, eps: float = 1e-5):
    return batchNorm(x, gamma, bias, channelAxis, eps, out=x)


def groupNorm(x: torch.Tensor, groups: int, gamma=None, bias=None, channelAxis: int = 1, eps: float = 1e-5,
              out: torch.Tensor | None = None) -> torch.Tensor:
    """Standardises every (sample, group of channels) over the group's channels and the remaining axes (reference
    yt::function::groupNorm, src/function/normalization.inl:491-577). The reference permutes the channel axis to the
    front and copies; here the grouped tensor is a strided VIEW [n, groups, channels / groups, ...] of x and of the
    output, handed to the generic-axes kernel as it is."""
    c = _channel_axis(x, channelAxis, "yt::function::groupNorm_")
    if groups <= 0:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "yt::function::groupNorm: groups must be positive")
    ch = x.shape[c]
    if ch % groups:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG,
                                         "yt::function::groupNorm: channel count must be divisible by groups")
    if x.dim() + 1 > 8:
        raise _lib.YtCudaInvalidArgument(_lib.UNSUPPORTED, "groupNorm: at most 7 dims")
    y = _like(x) if out is None else out
    per = ch // groups  # the channel axis in two: [n, groups, per, the other axes in their order]

    def grouped(v, split):
        return [v[0], *split(v[c]), *(v[a] for a in range(1, len(v)) if a != c)]

    shape = grouped(x.shape, lambda _: (groups, per))
    xt, yt = (grouped(t.stride(), lambda st: (st * per, st)) for t in (x, y))
    ws = [0, per, 1] + [0] * (len(shape) - 3)
    return _channel_norm(x, y, shape, xt, yt, list(range(2, len(shape))), eps, gamma, bias, c, ws)


def groupNorm_(x, groups: int, gamma=None, bias=None, channelAxis: int = 1, eps: float = 1e-5):
    return groupNorm(x, groups, gamma, bias, channelAxis, eps, out=x)


def rmsnorm_add_softmax_cast(x: torch.Tensor, weight: torch.Tensor, residual: torch.Tensor,
                             out_dtype: torch.dtype = torch.bfloat16, eps: float = 1e-6) -> torch.Tensor:
    """cast(softmax(rmsNorm(x, w, -1, eps) + residual, -1)) in one pass. x [B, L, H] fp32 contiguous,
    residual [B, L, H] or [1, L, H]."""
    _require_cuda(x, weight, residual)
    if x.dim() != 3 or x.dtype != torch.float32 or not x.is_contiguous():
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "chain: x must be a contiguous fp32 [B, L, H] tensor")
    B, Lr, H = x.shape
    if tuple(residual.shape) not in ((B, Lr, H), (1, Lr, H)) or tuple(weight.shape) != (H,):
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "chain: residual / weight shape mismatch")
    residual, weight = residual.contiguous().float(), weight.contiguous().float()
    out = torch.empty(B, Lr, H, dtype=out_dtype, device=x.device)
    check(lib().ytcuda_rmsnorm_add_softmax_cast(_DT[out_dtype], x.data_ptr(), weight.data_ptr(), residual.data_ptr(),
                                                out.data_ptr(), B, Lr, H, int(residual.shape[0] == B), eps, _stream()))
    return out


# ------------------------------------------------------------------ reductions
def _reduce(op: int, x: torch.Tensor, axes, want_index: bool):
    _require_cuda(x)
    ax = _axes(axes)
    nd, shape, xs = _nd(x)
    ks = list(x.shape) or [1]
    for a in ax:
        ks[a % nd] = 1
    y = torch.empty(*ks, dtype=x.dtype, device=x.device)
    idx = torch.empty(*ks, dtype=torch.int32, device=x.device) if want_index else None
    check(lib().ytcuda_reduce(op, _dt(x), _dt(y), x.data_ptr(), y.data_ptr(), idx.data_ptr() if want_index else None,
                              shape, xs, nd, _i32(ax), len(ax), _stream()))
    return (y, idx) if want_index else y


def sum(x: torch.Tensor, axes) -> torch.Tensor:  # noqa: A001 - mirrors YTensor::sum
    """Keep-dim sum over an axis or axes (reference YTensor::sum, src/ytensor_math.inl:414-509)."""
    return _reduce(0, x, axes, False)


def mean(x: torch.Tensor, axes) -> torch.Tensor:
    """Keep-dim mean (reference YTensor::mean, src/ytensor_math.inl:531-574)."""
    return _reduce(1, x, axes, False)


def max(x: torch.Tensor, axes):  # noqa: A001 - mirrors YTensor::max
    """Keep-dim maximum and the int index of its first occurrence (reference YTensor::max,
    src/ytensor_math.inl:591-692)."""
    return _reduce(2, x, axes, True)


# ------------------------------------------------------------------ elementwise
_BIN = {"add": 0, "sub": 1, "mul": 2, "div": 3}


def _binary(op: str, a: torch.Tensor, b, out: torch.Tensor | None) -> torch.Tensor:
    if not isinstance(b, torch.Tensor):
        return _unary({"add": 3, "sub": 3, "mul": 2, "div": 2}[op], a, out,
                      {"add": float(b), "sub": -float(b), "mul": float(b), "div": 1.0 / float(b)}[op])
    _require_cuda(a, b, out)
    try:
        shape, xa, xb = _broadcast(a, b)
    except RuntimeError as e:  # std::runtime_error in the reference (src/kernel/broadcast.inl:133)
        raise _lib.YtCudaError(_lib.INVALID_ARG, f"broadcast mismatch: {e}")
    if out is None:
        out = _like(a) if shape == a.shape else torch.empty(shape, dtype=a.dtype, device=a.device)
    elif tuple(out.shape) != shape:
        raise _lib.YtCudaError(_lib.INVALID_ARG, "in-place operand cannot be broadcast to the result shape")
    nd, osh, ost = _nd(out)
    check(lib().ytcuda_binary(_BIN[op], _dt(a), _dt(b), _dt(out), a.data_ptr(), b.data_ptr(), out.data_ptr(), nd, osh,
                              _i64(xa or (1,)), _i64(xb or (1,)), ost, _stream()))
    return out


def add(a, b): return _binary("add", a, b, None)
def sub(a, b): return _binary("sub", a, b, None)
def mul(a, b): return _binary("mul", a, b, None)
def div(a, b): return _binary("div", a, b, None)
def add_(a, b): return _binary("add", a, b, a)
def sub_(a, b): return _binary("sub", a, b, a)
def mul_(a, b): return _binary("mul", a, b, a)
def div_(a, b): return _binary("div", a, b, a)


def _unary(op: int, x: torch.Tensor, out: torch.Tensor | None, param: float = 0.0,
           out_dtype: torch.dtype | None = None) -> torch.Tensor:
    _require_cuda(x, out)
    if out is None:
        out = _like(x, out_dtype)
    elif out is not x and out.shape != x.shape:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "unary: shape mismatch")
    nd, shape, xs = _nd(x)
    check(lib().ytcuda_unary(op, _dt(x), _dt(out), x.data_ptr(), out.data_ptr(), nd, shape, xs, _i64(out.stride() or (1,)),
                             param, _stream()))
    return out


def swish(x, order=0): return _unary(_act_op("swish", 1, order), x, None)


def swish_(x, order=0):
    """x * sigmoid(x) in place (reference yt::function::swish_, src/function/activation.inl:631-647); order 1: its
    first derivative."""
    return _unary(_act_op("swish", 1, order), x, x)

# The other activations of yt::function (reference src/function/activation.inl); `name_` works in place.
_ACTIVATIONS = {"relu": 4, "exp": 5, "sigmoid": 6, "leakyRelu": 7, "elu": 8, "selu": 9, "gelu": 10, "tanh": 11,
                "softplus": 12, "mish": 13, "hardSigmoid": 14, "hardSwish": 15}
_ACT_DEFAULT_PARAM = {"leakyRelu": 0.01, "elu": 1.0}


def _act_op(name: str, op: int, order: int) -> int:
    if order == 0:
        return op
    if order == 1:
        return 32 + op
    raise _lib.YtCudaInvalidArgument(_lib.UNSUPPORTED, f"{name}: order {order} is not on the device (0 and 1 are)")


def _make_activation(name: str, op: int):
    default = _ACT_DEFAULT_PARAM.get(name)
    if default is None:
        def f(x, order=0):
            return _unary(_act_op(name, op, order), x, None, 0.0)

        def f_(x, order=0):
            return _unary(_act_op(name, op, order), x, x, 0.0)
    else:
        def f(x, alpha=default, order=0):
            return _unary(_act_op(name, op, order), x, None, float(alpha))

        def f_(x, alpha=default, order=0):
            return _unary(_act_op(name, op, order), x, x, float(alpha))

    f.__name__, f_.__name__ = name, name + "_"
    f.__doc__ = f_.__doc__ = (f"yt::function::{name} (reference src/function/activation.inl): order 0 the function, "
                              "order 1 its first derivative.")
    return f, f_


for _n, _op in _ACTIVATIONS.items():
    globals()[_n], globals()[_n + "_"] = _make_activation(_n, _op)


def cast(x: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    """dtype conversion with the reference's rounding (YTensorBase::cast, include/ytensor_base.hpp:399-404)."""
    _require_cuda(x)
    return copy_(_like(x, dtype), x)


FP8_KINDS = {"float8_e5m2": _lib.F8_E5M2, "float8_e4m3": _lib.F8_E4M3, "float8_e8m0": _lib.F8_E8M0}


def cast_to_fp8(x: torch.Tensor, kind: str) -> torch.Tensor:
    """float / bfloat16 / float16 -> the reference's 8-bit storage types (yt::float8_e5m2, float8_e4m3, float8_e8m0,
    include/types/float_spec.hpp:534-536) as uint8 bit patterns, with FloatSpec::fromFloat32's rounding (:435-491).
    These are the reference's own formats (the largest exponent is infinity / NaN), not the OCP fn variants, so the
    result is a uint8 tensor rather than a torch float8 dtype."""
    _require_cuda(x)
    out = torch.empty(x.shape, dtype=torch.uint8, device=x.device)
    s_, d = (x.reshape(1), out.reshape(1)) if x.dim() == 0 else (x, out)
    check(lib().ytcuda_cast(_dt(x), FP8_KINDS[kind], s_.data_ptr(), d.data_ptr(), d.dim(), _i64(d.shape),
                            _i64(s_.stride()), _i64(d.stride()), _stream()))
    return out


def cast_from_fp8(bits: torch.Tensor, kind: str, dtype: torch.dtype = torch.float32) -> torch.Tensor:
    """uint8 bit patterns of one of the reference's 8-bit types -> float / bfloat16 / float16 (FloatSpec::toFloat32,
    include/types/float_spec.hpp:299-371, then the target type's own constructor)."""
    _require_cuda(bits)
    if bits.dtype != torch.uint8:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "cast_from_fp8: uint8 bit patterns expected")
    out = torch.empty(bits.shape, dtype=dtype, device=bits.device)
    s_, d = (bits.reshape(1), out.reshape(1)) if bits.dim() == 0 else (bits, out)
    check(lib().ytcuda_cast(FP8_KINDS[kind], _dt(out), s_.data_ptr(), d.data_ptr(), d.dim(), _i64(d.shape),
                            _i64(s_.stride()), _i64(d.stride()), _stream()))
    return out


def copy_(dst: torch.Tensor, src: torch.Tensor) -> torch.Tensor:
    """Strided copy with conversion (YTensorBase::copy_, src/ytensor_base.inl:257-430)."""
    _require_cuda(dst, src)
    if dst.shape != src.shape:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "copy_: shape mismatch")
    nd, shape, ds = _nd(dst)
    check(lib().ytcuda_cast(_dt(src), _dt(dst), src.data_ptr(), dst.data_ptr(), nd, shape, _i64(src.stride() or (1,)), ds,
                            _stream()))
    return dst


def topk_sample(logits: torch.Tensor, k: int = 20, uniform: torch.Tensor | None = None):
    """Top-k sampling as qwen3::Qwen3ForCausalLM::generate does it (example/qwen3/src/qwen3.cpp:465-486).

    logits fp32 [rows, vocab]. Returns (top_probs [rows, k], top_idx [rows, k] int32, sampled [rows] int32 or None):
    the k most probable tokens of softmax(logits) in descending order and, when `uniform` (fp32 [rows], numbers in
    [0, 1]) is given, the token whose running sum first reaches uniform * sum(top_probs)."""
    _require_cuda(logits, uniform)
    if logits.dim() != 2 or logits.dtype != torch.float32 or logits.stride(1) != 1:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "topk_sample: logits must be fp32 [rows, vocab], unit stride")
    rows, vocab = logits.shape
    probs = torch.empty(rows, k, dtype=torch.float32, device=logits.device)
    idx = torch.empty(rows, k, dtype=torch.int32, device=logits.device)
    sampled = None
    if uniform is not None:
        if uniform.dtype != torch.float32 or uniform.numel() != rows or not uniform.is_contiguous():
            raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "topk_sample: uniform must be fp32 [rows]")
        sampled = torch.empty(rows, dtype=torch.int32, device=logits.device)
    check(lib().ytcuda_topk_sample(logits.data_ptr(), logits.stride(0), rows, vocab, k,
                                   uniform.data_ptr() if uniform is not None else None, probs.data_ptr(),
                                   idx.data_ptr(), sampled.data_ptr() if sampled is not None else None, _stream()))
    return probs, idx, sampled


def swiglu(gate_up: torch.Tensor, out_dtype: torch.dtype | None = None) -> torch.Tensor:
    """swish(gate) * up for a fused [..., 2*I] projection (example/qwen3/src/qwen3.cpp:193-200)."""
    _require_cuda(gate_up)
    if gate_up.stride(-1) != 1 or gate_up.shape[-1] % 2:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "swiglu: last dim must be contiguous and even")
    inter = gate_up.shape[-1] // 2
    g2 = gate_up if gate_up.dim() == 2 else gate_up.reshape(-1, 2 * inter)
    out = torch.empty(*gate_up.shape[:-1], inter, dtype=out_dtype or gate_up.dtype, device=gate_up.device)
    check(lib().ytcuda_swiglu(_dt(g2), _dt(out), g2.data_ptr(), out.data_ptr(), g2.shape[0], inter, g2.stride(0), inter,
                              _stream()))
    return out


# ------------------------------------------------------------------ attention
def _heads_view(t: torch.Tensor, what: str):
    """[batch..., heads..., len, dim] -> (tensor, batch, heads, strides {batch, head, row}); the leading dims must
    collapse into one batch stride and one head stride, and the last dim must have unit stride."""
    if t.stride(-1) != 1 and t.shape[-1] != 1:
        t = copy_(torch.empty(t.shape, dtype=t.dtype, device=t.device), t)
    return t


def scaledDotProductAttention(query: torch.Tensor, key: torch.Tensor, value: torch.Tensor, scale: float = 0.0,
                              mask: torch.Tensor | None = None, bias: torch.Tensor | None = None, *,
                              causal: bool = False, causal_offset: int | None = None) -> torch.Tensor:
    """softmax(scale * Q K^T + bias, masked) V (reference yt::function::scaledDotProductAttention,
    src/function/ops.inl:368-425).

    Shapes as the reference's callers use them: query [b, kv_heads, groups, q_len, d] with key / value either the
    zero-stride repeat [b, kv_heads, groups, kv_len, d] or plain [b, kv_heads, kv_len, d]; 4-D query
    [b, heads, q_len, d] with [b, kv_heads, kv_len, d] keys (heads a multiple of kv_heads); 3-D and 2-D forms have no
    batch / head dims. `mask` is a bool [q_len, kv_len] tensor; `causal=True` is the predicate form c <= r + offset
    with offset = kv_len - q_len unless given. Mismatched shapes raise ValueError like std::invalid_argument."""
    _require_cuda(query, key, value, mask, bias)
    if query.shape[-1] != key.shape[-1]:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "Query and key head dim must match.")
    if key.shape[-2] != value.shape[-2]:
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "Key/value sequence length must match.")
    if not (query.dtype == key.dtype == value.dtype):
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "scaledDotProductAttention: dtypes differ")
    lq, d = query.shape[-2:]
    lk, dv = value.shape[-2:]
    out_shape = (*query.shape[:-1], dv)
    q, k, v = query, key, value
    if q.dim() == 5:
        b, kvh, g = q.shape[:3]
        if k.dim() == 5:
            k, v = k[:, :, 0], v[:, :, 0]
        q = q.reshape(b, kvh * g, lq, d)
    elif q.dim() == 4:
        b, h = q.shape[:2]
        kvh = k.shape[1]
        if h % kvh:
            raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "query heads must be a multiple of key/value heads")
        g = h // kvh
    else:
        lead = q.shape[:-2]
        n = 1
        for x in lead:
            n *= x
        q, k, v = q.reshape(1, n, lq, d), k.reshape(1, n, lk, d), v.reshape(1, n, lk, dv)
        b, kvh, g = 1, n, 1
    if tuple(k.shape) != (b, kvh, lk, d) or tuple(v.shape) != (b, kvh, lk, dv):
        raise _lib.YtCudaInvalidArgument(_lib.INVALID_ARG, "key/value batch or head dims do not match the query")
    q, k, v = _heads_view(q, "query"), _heads_view(k, "key"), _heads_view(v, "value")
    mask_kind, mptr, mrs, off = 0, None, 0, 0
    if mask is not None:
        if tuple(mask.shape) != (lq, lk):
            raise _lib.YtCudaInvalidArgument(
                _lib.INVALID_ARG, "Mask shape must match the last two dimensions of the score tensor.")
        # (a bool is a byte of 0 or 1: read as it lies)
        m8 = mask if mask.dtype == torch.uint8 else mask.view(torch.uint8) if mask.dtype == torch.bool else mask.to(torch.uint8)
        m8 = m8.contiguous()
        mask_kind, mptr, mrs = 2, m8.data_ptr(), m8.stride(0)
    elif causal:
        mask_kind, off = 1, (lk - lq) if causal_offset is None else int(causal_offset)
    bptr, brs, bcs = None, 0, 0
    if bias is not None:
        if tuple(bias.shape) != (lq, lk):
            raise _lib.YtCudaInvalidArgument(
                _lib.INVALID_ARG, "Bias shape must match the last two dimensions of the score tensor.")
        bias = bias.float()
        bptr, brs, bcs = bias.data_ptr(), bias.stride(0), bias.stride(1)
    out = torch.empty(*out_shape, dtype=query.dtype, device=query.device)  # ([b, heads, q_len, dv], whatever the leading dims)
    check(lib().ytcuda_flash_attn_fwd(_dt(q), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), b, kvh, g, lq,
                                      lk, d, dv, float(scale), _i64(q.stride()[:3]), _i64(k.stride()[:3]),
                                      _i64(v.stride()[:3]), _i64((kvh * g * lq * dv, lq * dv, dv)), mask_kind, off, mptr, mrs,
                                      bptr, brs, bcs, _stream()))
    return out
