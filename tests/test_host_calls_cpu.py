"""What the host layer hands to the library, with a stand-in for the library that computes on host memory from the raw
pointers, shapes and strides: broadcasts, products of every arrangement of leading dims, grouped norms."""
import ctypes as C
import itertools
import struct

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from ytensor_b200 import api  # noqa: E402


def raw(ptr, shape, strides):
    """The fp32 memory at `ptr`, element strides."""
    span = 1 + sum((n - 1) * s for n, s in zip(shape, strides)) if all(shape) else 0
    base = np.ctypeslib.as_array(C.cast(ptr, C.POINTER(C.c_float)), (max(span, 1),))
    return np.lib.stride_tricks.as_strided(base, shape, [4 * s for s in strides])


def words(b, n):
    assert len(b) == 8 * n
    return struct.unpack(f"{n}q", b)


class HostLibrary:
    def ytcuda_binary(self, op, da, db, do, a, b, o, nd, shape, sa, sb, so, st):
        s = words(shape, nd)
        x, y = raw(a, s, words(sa, nd)), raw(b, s, words(sb, nd))
        raw(o, s, words(so, nd))[...] = (x + y, x - y, x * y, x / y)[op]
        return 0

    def ytcuda_gemm(self, di, do, a, b, c, m, n, k, alpha, beta, rsa, csa, rsb, csb, rsc, csc, batch, bsa, bsb, bsc, st):
        x, y = raw(a, (batch, m, k), (bsa, rsa, csa)), raw(b, (batch, k, n), (bsb, rsb, csb))
        z = raw(c, (batch, m, n), (bsc, rsc, csc))
        z[...] = alpha * (x @ y) + (beta * z if beta else 0)
        return 0

    def ytcuda_layernorm_strided(self, dx, dy, dw, x, g, b, y, shape, xs, ys, ws, nd, axes, na, eps, st):
        s, ax = words(shape, nd), struct.unpack(f"{na}i", axes)
        v = raw(x, s, words(xs, nd))
        v = (v - v.mean(ax, keepdims=True)) / np.sqrt(v.var(ax, keepdims=True) + eps)
        raw(y, s, words(ys, nd))[...] = v * raw(g, s, words(ws, nd)) + raw(b, s, words(ws, nd))
        return 0


@pytest.fixture(autouse=True)
def host(monkeypatch):
    monkeypatch.setattr(api, "lib", HostLibrary)
    monkeypatch.setattr(api, "_require_cuda", lambda *t: None)
    monkeypatch.setattr(api, "_stream", lambda: 0)


SHAPES = [(), (1,), (3,), (4,), (3, 1), (1, 4), (3, 4), (2, 3, 4), (2, 1, 4), (1, 1, 1), (5, 1, 3, 1), (0, 4)]


@pytest.mark.parametrize("sa,sb", list(itertools.product(SHAPES, SHAPES)))
def test_broadcast(sa, sb):
    a, b = torch.randn(sa), torch.randn(sb)
    try:
        want = a + b
    except RuntimeError:
        with pytest.raises(Exception):
            api.add(a, b)
        return
    shape, xa, xb = api._broadcast(a, b)
    assert shape == tuple(want.shape)
    for got, t in ((xa, a), (xb, b)):  # (the stride of an axis of one element is never used)
        assert all(n == 1 or g == e for n, g, e in zip(shape, got, t.expand(shape).stride()))
    if want.numel():
        assert torch.equal(api.add(a, b), want)


@pytest.mark.parametrize("la,lb", [((), ()), ((4,), ()), ((), (4,)), ((4,), (4,)), ((4,), (1,)), ((2, 3), ()), ((2, 3), (3,)),
                                   ((2, 1), (1, 3)), ((1, 3), (2, 1)), ((2, 3), (2, 3)), ((2, 1, 3), (2, 5, 3))])
@pytest.mark.parametrize("order", ["plain", "turned", "stepped"])
def test_products(la, lb, order):
    def make(lead, r, c):
        if order == "turned":
            return torch.randn(*lead, c, r).transpose(-1, -2)
        return torch.randn(*lead, r, 2 * c)[..., ::2] if order == "stepped" else torch.randn(*lead, r, c)

    a, b = make(la, 3, 5), make(lb, 5, 4)
    close = dict(rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(api.matmul(a, b), a @ b, **close)
    torch.testing.assert_close(api.linear(a, b.transpose(-1, -2)), a @ b, **close)
    out = torch.randn_like(a @ b)
    want = 2 * (a @ b) + 3 * out
    torch.testing.assert_close(api.matmul(a, b, out, alpha=2.0, beta=3.0), want, **close)


def test_vectors_and_refusals():
    v, m = torch.randn(5), torch.randn(5, 4)
    torch.testing.assert_close(api.matmul(v, m), (v @ m)[None], rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(api.matmul(m.T, v), (m.T @ v)[:, None], rtol=1e-5, atol=1e-5)
    for a, b in ((torch.randn(3, 4), torch.randn(5, 4)), (torch.randn(()), m), (torch.randn(2, 3, 5), torch.randn(3, 5, 4)),
                 (v, m.double())):
        with pytest.raises(Exception):
            api.matmul(a, b)
    with pytest.raises(Exception):
        api.matmul(m.T, m, torch.empty(4, 5))


@pytest.mark.parametrize("axis", [1, 2, 3])
def test_channel_norms(axis, monkeypatch):
    monkeypatch.setattr(torch.Tensor, "is_cuda", True, raising=False)
    x = torch.randn(3, 4, 6, 8).permute(0, 2, 1, 3)[:, :, :, :]  # [3, 6, 4, 8], strides out of order
    c = x.shape[axis]
    g, b = torch.randn(c), torch.randn(c)
    moved = x.movedim(axis, 1)
    want = torch.nn.functional.group_norm(moved.contiguous(), 2, g, b).movedim(1, axis)
    torch.testing.assert_close(api.groupNorm(x, 2, g, b, axis), want, rtol=1e-4, atol=1e-4)
    want = torch.nn.functional.batch_norm(moved.contiguous(), None, None, g, b, True).movedim(1, axis)
    torch.testing.assert_close(api.batchNorm(x, g, b, axis), want, rtol=1e-4, atol=1e-4)
