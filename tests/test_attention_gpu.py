"""GPU parity tests of ytcuda_flash_attn_fwd against the CPU oracle and the golden vectors.
fp32 (one-warp-per-row kernel): 1e-5 normwise. bf16 / fp16 (tcgen05 kernel, fp32 accumulation, P rounded to
16 bits before P.V): 2e-2 normwise against the fp32 oracle run on the same 16-bit inputs."""
import numpy as np
import pytest

from _util import bits_to_torch, normwise, torch_to_bits

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

F32_TOL, H_TOL = 1e-5, 2e-2


@pytest.fixture(scope="module")
def L():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ytensor_b200 import _lib
    lib = _lib.lib()
    yield lib
    lib.ytcuda_attn_set_path(0)


@pytest.fixture(scope="module")
def api(L):
    from ytensor_b200 import api
    return api


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# ------------------------------------------------------------------ fp32, golden vectors
def test_doc_example(api, golden):
    q, k, v = dev(golden["doc_sdpa_q"]), dev(golden["doc_sdpa_k"]), dev(golden["doc_sdpa_v"])
    m = dev(golden["doc_sdpa_mask"]).bool()
    got = api.scaledDotProductAttention(q, k, v, 0.0, m).cpu().numpy()
    assert normwise(got, golden["doc_sdpa_out_flash_mask"]) < F32_TOL
    assert normwise(got, golden["doc_sdpa_out_math_mask"]) < F32_TOL
    # the documentation's predicate j <= i is the causal form with offset 0
    got = api.scaledDotProductAttention(q, k, v, 0.0, causal=True, causal_offset=0).cpu().numpy()
    assert normwise(got, golden["doc_sdpa_out_flash_pred"]) < F32_TOL


def test_fp32_golden(api, golden):
    q, k, v = dev(golden["att_q"]), dev(golden["att_k"]), dev(golden["att_v"])
    A = api.scaledDotProductAttention
    assert normwise(A(q, k, v, causal=True).cpu().numpy(), golden["att_causal"]) < F32_TOL
    assert normwise(A(q, k, v).cpu().numpy(), golden["att_full"]) < F32_TOL
    got = A(q, k, v, 0.0, dev(golden["att_mask"]).bool()).cpu().numpy()
    assert normwise(got, golden["att_masked"]) < F32_TOL
    assert np.all(got[:, :, :, 4, :] == 0.0)  # a row that sees no key is zero
    got = A(q, k, v, 0.2, None, dev(golden["att_bias"]), causal=True).cpu().numpy()
    assert normwise(got, golden["att_bias_causal"]) < F32_TOL
    assert normwise(A(dev(golden["att_q_short"]), k, v, causal=True).cpu().numpy(), golden["att_short_causal"]) < F32_TOL
    assert normwise(A(dev(golden["att_q_one"]), k, v, causal=True).cpu().numpy(), golden["att_decode"]) < F32_TOL
    # the zero-stride repeat form of the keys, as the decoder passes them
    k5 = k.unsqueeze(2).expand(-1, -1, 2, -1, -1)
    v5 = v.unsqueeze(2).expand(-1, -1, 2, -1, -1)
    assert normwise(A(q, k5, v5, causal=True).cpu().numpy(), golden["att_causal"]) < F32_TOL


def test_shape_errors(api):
    q = torch.zeros(1, 2, 2, 4, 8, device="cuda")
    with pytest.raises(ValueError):
        api.scaledDotProductAttention(q, torch.zeros(1, 2, 5, 16, device="cuda"), torch.zeros(1, 2, 5, 8, device="cuda"))
    with pytest.raises(ValueError):
        api.scaledDotProductAttention(q, torch.zeros(1, 2, 5, 8, device="cuda"), torch.zeros(1, 2, 6, 8, device="cuda"))
    with pytest.raises(ValueError):
        api.scaledDotProductAttention(q, torch.zeros(1, 2, 5, 8, device="cuda"), torch.zeros(1, 2, 5, 8, device="cuda"),
                                      0.0, torch.ones(3, 5, device="cuda").bool())


# ------------------------------------------------------------------ 16-bit, tensor-core kernel
def run_tc(L, api, port, q, k, v, dt=1, **kw):
    """q, k, v fp32 numpy; rounds to the 16-bit type, runs the device kernel (tcgen05 forced) and the oracle."""
    f2b, b2f = (port.f32_to_bf16, port.bf16_to_f32) if dt == 1 else (port.f32_to_f16, port.f16_to_f32)
    tdt = torch.bfloat16 if dt == 1 else torch.float16
    qb, kb, vb = f2b(q), f2b(k), f2b(v)
    okw = {}
    dkw = {}
    if kw.get("mask") is not None:
        okw["mask"] = kw["mask"]
        dkw["mask"] = dev(kw["mask"]).bool()
    if kw.get("causal"):
        okw["causal"] = True
        dkw["causal"] = True
    if kw.get("bias") is not None:
        okw["bias"] = kw["bias"]
        dkw["bias"] = dev(kw["bias"])
    want = port.sdpa(b2f(qb), b2f(kb), b2f(vb), scale=kw.get("scale", 0.0), **okw)
    L.ytcuda_attn_set_path(2)
    try:
        out = api.scaledDotProductAttention(bits_to_torch(qb, tdt), bits_to_torch(kb, tdt), bits_to_torch(vb, tdt),
                                            kw.get("scale", 0.0), dkw.get("mask"), dkw.get("bias"),
                                            causal=dkw.get("causal", False))
    finally:
        L.ytcuda_attn_set_path(0)
    assert L.ytcuda_device_status(None) == 0
    return b2f(torch_to_bits(out)), want


@pytest.mark.parametrize("b,kvh,g,lq,lk,d,causal", [
    (1, 1, 2, 128, 128, 128, False),
    (1, 1, 2, 128, 128, 128, True),
    (2, 2, 2, 256, 256, 128, True),
    (1, 1, 4, 384, 384, 128, True),
    (1, 2, 1, 512, 512, 128, True),     # no head pairs: two neighbouring row blocks share the K/V stream
    (1, 1, 1, 300, 300, 128, True),
    (1, 1, 2, 200, 333, 128, True),     # ragged lengths, causal window anchored at the end of the keys
    (1, 1, 2, 77, 500, 128, False),
    (1, 1, 3, 130, 130, 128, True),     # odd group count
    (1, 2, 2, 256, 256, 64, True),
    (1, 1, 2, 100, 640, 64, False),
    (1, 1, 2, 1, 300, 128, True),       # a decode step through the same kernel
])
def test_bf16_vs_oracle(L, api, port, b, kvh, g, lq, lk, d, causal):
    rng = np.random.default_rng(b + kvh * 3 + g * 5 + lq + lk * 7 + d)
    q = rng.standard_normal((b, kvh, g, lq, d)).astype(np.float32)
    k = rng.standard_normal((b, kvh, lk, d)).astype(np.float32)
    v = rng.standard_normal((b, kvh, lk, d)).astype(np.float32)
    got, want = run_tc(L, api, port, q, k, v, causal=causal)
    assert normwise(got, want) < H_TOL


def test_fp16_mask_bias_and_empty_rows(L, api, port):
    rng = np.random.default_rng(21)
    q = rng.standard_normal((1, 2, 2, 150, 128)).astype(np.float32)
    k = rng.standard_normal((1, 2, 260, 128)).astype(np.float32)
    v = rng.standard_normal((1, 2, 260, 128)).astype(np.float32)
    m = (rng.random((150, 260)) < 0.5).astype(np.uint8)
    m[7] = 0
    m[140] = 0
    bias = rng.standard_normal((150, 260)).astype(np.float32)
    got, want = run_tc(L, api, port, q, k, v, dt=2, mask=m)
    assert normwise(got, want) < H_TOL
    assert np.all(got[:, :, :, 7, :] == 0) and np.all(got[:, :, :, 140, :] == 0)
    got, want = run_tc(L, api, port, q, k, v, dt=2, causal=True, bias=bias, scale=0.05)
    assert normwise(got, want) < H_TOL


def test_large_logits_rescale_path(L, api, port):
    """Scores that grow along the keys force the running maximum to move by more than 2^8 many times."""
    rng = np.random.default_rng(5)
    lk = 640
    q = np.ones((1, 1, 2, 128, 128), np.float32)
    k = (np.linspace(0.0, 1.5, lk)[:, None] * np.ones((1, 128))).astype(np.float32)[None, None]
    k = k + 0.05 * rng.standard_normal(k.shape).astype(np.float32)
    v = rng.standard_normal((1, 1, lk, 128)).astype(np.float32)
    got, want = run_tc(L, api, port, q, k, v, scale=1.0)
    assert normwise(got, want) < H_TOL


def test_strided_views_of_fused_qkv(L, api, port):
    """q, k, v as slices of one fused projection output [b, l, (h + 2 kvh) * d], permuted to [b, h, l, d]."""
    rng = np.random.default_rng(9)
    b, l, h, kvh, d = 2, 256, 4, 2, 128
    qkv = rng.standard_normal((b, l, (h + 2 * kvh) * d)).astype(np.float32)
    bits = port.f32_to_bf16(qkv)
    t = bits_to_torch(bits, torch.bfloat16)
    q = t[..., : h * d].view(b, l, h, d).permute(0, 2, 1, 3)
    k = t[..., h * d: (h + kvh) * d].view(b, l, kvh, d).permute(0, 2, 1, 3)
    v = t[..., (h + kvh) * d:].view(b, l, kvh, d).permute(0, 2, 1, 3)
    f = port.bf16_to_f32(bits)
    qf = f[..., : h * d].reshape(b, l, h, d).transpose(0, 2, 1, 3).reshape(b, kvh, h // kvh, l, d)
    kf = f[..., h * d: (h + kvh) * d].reshape(b, l, kvh, d).transpose(0, 2, 1, 3)
    vf = f[..., (h + kvh) * d:].reshape(b, l, kvh, d).transpose(0, 2, 1, 3)
    want = port.sdpa(qf, kf, vf, causal=True).reshape(b, h, l, d)
    L.ytcuda_attn_set_path(2)
    try:
        out = api.scaledDotProductAttention(q, k, v, causal=True)
    finally:
        L.ytcuda_attn_set_path(0)
    assert normwise(port.bf16_to_f32(torch_to_bits(out)), want) < H_TOL


def test_config3_full_size_properties(L, api, port):
    """benchmark configuration 3: batch 16, 32 query / 8 kv heads, head_dim 128, seq 4096, causal, bf16.
    Full size through properties: (1) two batch items with the same inputs give the same bits, (2) the first
    256 and the last 128 query rows of one kv head against the oracle, (3) row 0 equals V[0]."""
    g = torch.Generator(device="cuda").manual_seed(2)
    q = torch.randn(16, 32, 4096, 128, device="cuda", generator=g).to(torch.bfloat16)
    k = torch.randn(16, 8, 4096, 128, device="cuda", generator=g).to(torch.bfloat16)
    v = torch.randn(16, 8, 4096, 128, device="cuda", generator=g).to(torch.bfloat16)
    q[15], k[15], v[15] = q[3], k[3], v[3]
    L.ytcuda_attn_set_path(2)
    try:
        out = api.scaledDotProductAttention(q, k, v, causal=True)
    finally:
        L.ytcuda_attn_set_path(0)
    assert L.ytcuda_device_status(None) == 0
    assert torch.equal(out[15], out[3])
    # row 0 sees one key: its softmax weight is 1 up to fp32 round-off, so the output is V[0] within one bf16 step
    v0 = v[:, :, 0, :].repeat_interleave(4, dim=1).float()
    assert torch.all((out[:, :, 0, :].float() - v0).abs() <= v0.abs() * 2.0 ** -7 + 1e-30)
    b2f = port.bf16_to_f32
    qf = b2f(torch_to_bits(q[5, 8:12])).reshape(1, 1, 4, 4096, 128)
    kf = b2f(torch_to_bits(k[5, 2])).reshape(1, 1, 4096, 128)
    vf = b2f(torch_to_bits(v[5, 2])).reshape(1, 1, 4096, 128)
    got = b2f(torch_to_bits(out[5, 8:12])).reshape(1, 1, 4, 4096, 128)
    want_head = port.sdpa(qf[:, :, :, :256], kf[:, :, :256], vf[:, :, :256], causal=True)
    assert normwise(got[:, :, :, :256], want_head) < H_TOL
    want_tail = port.sdpa(qf[:, :, :, -128:], kf, vf, causal=True)  # offset kv_len - q_len: the last 128 rows
    assert normwise(got[:, :, :, -128:], want_tail) < H_TOL


# ------------------------------------------------------------------ fp32 products from bf16 planes (attn_split.cuh)
def _exact(q, k, v, scale, seen=None, bias=None):
    g = q.shape[1] // k.shape[1]
    s = q.double() @ k.double().repeat_interleave(g, 1).transpose(-1, -2) * scale
    s = s if bias is None else s + bias.double()
    s = s if seen is None else s.masked_fill(~seen, float("-inf"))
    return torch.softmax(s, -1) @ v.double().repeat_interleave(g, 1)


def _f32_bound(q, k, v, d, bias=None):
    """Rows of few visible keys average nothing out: a weight is off by the exponential's 2^-22 and by the roundings of its
    score, 2^-24 of the score (log2 units) in the product, the scale and the bias each."""
    s = (q.double() @ k.double().repeat_interleave(q.shape[1] // k.shape[1], 1).transpose(-1, -2)).abs().max() * d ** -0.5
    s = s + (0 if bias is None else bias.abs().max())
    return 2.0 ** -22 * (1 + 1.4427 * s) * v.abs().max()


@pytest.mark.parametrize("b,kvh,g,lq,lk,d,dt,form", [
    (1, 1, 1, 64, 256, 128, "f32", "causal"), (1, 2, 2, 129, 257, 128, "f32", "causal"), (2, 2, 4, 33, 65, 64, "f32", "none"),
    (1, 1, 1, 300, 513, 20, "f32", "causal"), (1, 2, 1, 127, 319, 80, "f32", "bool"), (1, 1, 3, 130, 256, 100, "f32", "bias"),
    (1, 2, 2, 40, 40, 80, "bf16", "causal"), (1, 1, 2, 200, 129, 96, "f16", "none"), (150, 1, 1, 20, 33, 36, "bf16", "none"),
    (1, 40, 2, 160, 270, 128, "f32", "causal")])
def test_planes_against_64_bits(L, api, b, kvh, g, lq, lk, d, dt, form):
    gen = torch.Generator(device="cuda").manual_seed(lq * 1000 + lk)
    t = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[dt]
    # a fused projection's layout: [batch, position, head, d] seen as [batch, head, position, d]
    q, k, v = (torch.randn(b, n, h, d, generator=gen, device="cuda").to(t).transpose(1, 2)
               for n, h in ((lq, kvh * g), (lk, kvh), (lk, kvh)))
    seen = bias = None
    if form == "causal":  # (more queries than keys is allowed: the first rows then see none)
        seen = torch.arange(lk, device="cuda")[None] <= torch.arange(lk - lq, lk, device="cuda")[:, None]
    elif form == "bool":
        seen = torch.rand(lq, lk, generator=gen, device="cuda") < 0.6
        seen[:, 3] = True
    elif form == "bias":
        bias = torch.randn(lq, lk, generator=gen, device="cuda")
    got = api.scaledDotProductAttention(q, k, v, d ** -0.5, seen if form == "bool" else None, bias, causal=form == "causal")
    want = _exact(q, k, v, d ** -0.5, seen, bias)
    # 16 bits: the rounding of the result, in bf16 by the reference's rule (half a unit is added only to an odd result: up to
    # one unit, 2^-7 of the value), in fp16 half a unit.
    bound = _f32_bound(q, k, v, d, bias) if dt == "f32" else {"bf16": 2.0 ** -7, "f16": 2.0 ** -11}[dt] * want.abs().max()
    assert (got.double() - want).abs().max() <= bound
    assert L.ytcuda_device_status(None) == 0


@pytest.mark.parametrize("name,value", [("q", float("inf")), ("k", float("-inf")), ("v", float("nan")), ("v", 3e38)])
def test_planes_leave_special_values_to_ffma(L, api, name, value):
    gen = torch.Generator(device="cuda").manual_seed(5)
    t = {n: torch.randn(1, 2, 300, 64, generator=gen, device="cuda") for n in "qkv"}
    t[name][0, 1, 290, 7] = value
    got = api.scaledDotProductAttention(t["q"], t["k"], t["v"], causal=True)
    L.ytcuda_attn_set_path(1)
    want = api.scaledDotProductAttention(t["q"], t["k"], t["v"], causal=True)
    L.ytcuda_attn_set_path(0)
    assert torch.equal(torch.nan_to_num(got, 7.0, 8.0, 9.0), torch.nan_to_num(want, 7.0, 8.0, 9.0))


def test_planes_step_aside_in_a_capture(api):
    gen = torch.Generator(device="cuda").manual_seed(6)
    q, k, v = (torch.randn(1, 4, 320, 128, generator=gen, device="cuda") for _ in range(3))
    want = api.scaledDotProductAttention(q, k, v, causal=True)
    graph, out = torch.cuda.CUDAGraph(), torch.empty_like(q)
    with torch.cuda.graph(graph):
        out.copy_(api.scaledDotProductAttention(q, k, v, causal=True))
    out.zero_()
    graph.replay()
    assert (out - want).abs().max() <= 2e-6 * want.abs().max()  # (the FFMA kernel: another order of the sums)


@pytest.mark.parametrize("lq,lk,d,dt", [(300, 336, 128, "bf16"), (257, 333, 64, "f16"), (129, 131, 128, "bf16"), (256, 301, 128, "f32"),
                                        (200, 288, 80, "f32")])
@pytest.mark.parametrize("form", ["bool", "bias", "both", "slices"])
def test_masks_and_biases_of_any_alignment(L, api, lq, lk, d, dt, form):
    gen = torch.Generator(device="cuda").manual_seed(lq + lk)
    t = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[dt]
    q, k, v = (torch.randn(1, h, n, d, generator=gen, device="cuda").to(t) for h, n in ((4, lq), (2, lk), (2, lk)))
    seen = torch.rand(lq, lk + 5, generator=gen, device="cuda") < 0.5
    bias = torch.randn(lq, lk + 7, generator=gen, device="cuda")
    seen[7] = False  # a row that sees no key
    seen[lq - 1] = False
    seen[lq - 1, lk - 1] = True
    off = 3 if form == "slices" else 0  # rows that start at odd addresses, strides of the wider tensor
    seen, bias = seen[:, off:off + lk], bias[:, off:off + lk]
    if form != "slices":
        seen, bias = seen.contiguous(), bias.contiguous()
    m, b = (None if form == "bias" else seen), (None if form == "bool" else bias)
    got = api.scaledDotProductAttention(q, k, v, d ** -0.5, m, b)
    want = torch.nan_to_num(_exact(q, k, v, d ** -0.5, m, b))
    # 16 bits: P and the result are rounded to 16 bits
    bound = _f32_bound(q, k, v, d, bias) if dt == "f32" else {"bf16": H_TOL, "f16": 2e-3}[dt] * want.abs().max()
    assert (got.double() - want).abs().max() <= bound
    assert m is None or not got[0, :, 7].any()


@pytest.mark.parametrize("lq,lk,d,dt", [(300, 336, 128, "f32"), (129, 131, 20, "f32"), (40, 70, 80, "bf16")])
def test_bias_of_the_lowest_float(L, api, lq, lk, d, dt):
    """Masks are often written as the lowest float: such a key weighs nothing beside others, and a row that has no other keys
    weighs all of them alike (the score is lost in the rounding of the sum)."""
    gen = torch.Generator(device="cuda").manual_seed(lk)
    t = {"f32": torch.float32, "bf16": torch.bfloat16}[dt]
    q, k, v = (torch.randn(1, h, n, d, generator=gen, device="cuda").to(t) for h, n in ((2, lq), (2, lk), (2, lk)))
    low = torch.finfo(torch.float32).min
    bias = torch.where(torch.rand(lq, lk, generator=gen, device="cuda") < 0.5, low, 0.0)
    bias[5], bias[lq - 1], bias[11, 3:], bias[12] = low, low, float("-inf"), float("-inf")
    bias[11, :3] = low
    bias[17] = torch.where(torch.arange(lk, device="cuda") == 9, -2.6e38, -3.3e38)  # (finite, one far above the others)
    got = api.scaledDotProductAttention(q, k, v, d ** -0.5, None, bias).double()
    s = (q.double() @ k.double().transpose(-1, -2) * d ** -0.5).float() + bias  # the sum in 32 bits
    want = torch.nan_to_num(torch.softmax(s.double(), -1) @ v.double())
    bound = _f32_bound(q, k, v, d) if dt == "f32" else 2.0 ** -7 * want.abs().max()
    assert (got - want).abs().max() <= bound
    assert not got[0, :, 12].any()  # no key at all


@pytest.mark.parametrize("dt", ["f32", "f16"])
@pytest.mark.parametrize("case", ["scores", "sums", "tiny"])
def test_planes_leave_the_ends_of_the_range_to_ffma(L, api, case, dt):
    """Scores and sums beyond the largest float, operands near the smallest: what FFMA makes of them."""
    gen = torch.Generator(device="cuda").manual_seed(8)
    t = {n: torch.randn(1, 2, 300, 96, generator=gen, device="cuda") for n in "qkv"}
    if dt == "f16":
        if case != "scores":
            pytest.skip("fp16 numbers do not reach there")
        t = {n: x.half() for n, x in t.items()}
        scale = 1e37
    else:
        scale = None
        if case == "scores":  # one key whose scores overflow to either infinity: a negative one weighs nothing
            t["q"][0, 1, :, 3:9] *= 2.0 ** 70
            t["k"][0, 1, 290, 3:9] *= 2.0 ** 66
        elif case == "sums":
            t["v"] = t["v"].abs() * 2.0 ** 124
        else:
            t["q"] *= 2.0 ** 60
            t["k"] *= 2.0 ** -60
            t["v"] *= 2.0 ** -119
    run = lambda: api.scaledDotProductAttention(t["q"], t["k"], t["v"], *([scale] if scale else []), causal=True)  # noqa: E731
    got = run()
    L.ytcuda_attn_set_path(1)
    try:
        want = run()
    finally:
        L.ytcuda_attn_set_path(0)
    assert torch.equal(torch.nan_to_num(got, 7.0, 8.0, 9.0), torch.nan_to_num(want, 7.0, 8.0, 9.0))
    assert case == "tiny" or not want.isfinite().all()


@pytest.mark.parametrize("b,kvh,g,lq,lk,d,dt", [(5, 3, 2, 70, 24000, 64, "f32"), (1, 7, 1, 40, 50001, 36, "f32"), (3, 2, 1, 33, 130000, 80, "bf16")])
def test_planes_in_bounded_scratch(L, api, b, kvh, g, lq, lk, d, dt):
    """Keys and values whose planes are more than a stream keeps as scratch go by in groups of heads and batch items."""
    gen = torch.Generator(device="cuda").manual_seed(lk)
    t = {"f32": torch.float32, "bf16": torch.bfloat16}[dt]
    q, k, v = (torch.randn(b, n, h, d, generator=gen, device="cuda").to(t).transpose(1, 2)
               for n, h in ((lq, kvh * g), (lk, kvh), (lk, kvh)))
    got = api.scaledDotProductAttention(q, k, v, causal=True)
    seen = torch.arange(lk, device="cuda")[None] <= torch.arange(lk - lq, lk, device="cuda")[:, None]
    for i in range(b):
        want = _exact(q[i:i + 1], k[i:i + 1], v[i:i + 1], d ** -0.5, seen)
        bound = _f32_bound(q[i:i + 1], k[i:i + 1], v, d) if dt == "f32" else 2.0 ** -7 * want.abs().max()
        assert (got[i:i + 1].double() - want).abs().max() <= bound
    before = L.ytcuda_launch_count()
    api.scaledDotProductAttention(q, k, v, causal=True)
    assert L.ytcuda_launch_count() - before > 3  # (planes, product, check: more than one group)


def test_attention_over_its_queries(L, api):
    """O may lie over Q: an infinity sends the call to the FFMA kernel, which has to find Q as it was."""
    gen = torch.Generator(device="cuda").manual_seed(4)
    q, k, v = (torch.randn(1, 2, 300, 64, generator=gen, device="cuda") for _ in range(3))
    k[0, 1, 299, 5] = float("inf")
    want, out = api.scaledDotProductAttention(q, k, v, causal=True), q.clone()
    import ctypes
    strides = (ctypes.c_int64 * 3)(*q.stride()[:3])
    rc = L.ytcuda_flash_attn_fwd(0, out.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), 1, 2, 1, 300, 300, 64, 64, 0.125, strides,
                                 strides, strides, strides, 1, 0, None, 0, None, 0, 0, torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and torch.equal(torch.nan_to_num(out, 7.0, 8.0, 9.0), torch.nan_to_num(want, 7.0, 8.0, 9.0))
