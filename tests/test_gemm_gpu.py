"""GPU parity tests of ytcuda_gemm / ytcuda_gemm_host against the CPU oracle and the golden vectors.

Tolerances (normwise, max|d| / max|ref|): 1e-5 for fp32, 2e-2 for bf16 / fp16 storage with fp32
accumulation. The bf16 comparison is never bitwise: device and oracle add in different orders and a
one-ulp difference before rounding moves the rounded value."""
import ctypes

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
    lib.ytcuda_gemm_set_path(0)


@pytest.fixture(scope="module")
def api(L):
    from ytensor_b200 import api
    return api


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def status_ok(L):
    assert L.ytcuda_device_status(None) == 0


# ------------------------------------------------------------------ fp32 (FFMA path)
def test_doc_example_exact(L, api, golden):
    c = api.matmul(dev(golden["doc_matmul_a"]), dev(golden["doc_matmul_b"])).cpu().numpy()
    assert np.array_equal(c, golden["doc_matmul_c"])


def test_fp32_golden(L, api, golden):
    a = dev(golden["mm_a"])
    assert normwise(api.matmul(a, dev(golden["mm_b2"])).cpu().numpy(), golden["mm_c_shared"]) < F32_TOL
    assert normwise(api.matmul(a, dev(golden["mm_b3"])).cpu().numpy(), golden["mm_c_batched"]) < F32_TOL
    got = api.matmul(dev(golden["mm_big_a"]), dev(golden["mm_big_b"])).cpu().numpy()
    assert normwise(got, golden["mm_big_c"]) < F32_TOL
    y = api.linear(dev(golden["lin_x"]), dev(golden["lin_w"])).cpu().numpy()
    assert normwise(y, golden["lin_y"]) < F32_TOL


def test_fp32_strided_alpha_beta_golden(L, api, golden):
    a, bt, c0 = dev(golden["sgemm_a"]), dev(golden["sgemm_bt"]), dev(golden["sgemm_c0"])
    out = c0.clone()
    api.matmul(a, bt.t(), out, alpha=0.5, beta=2.0)
    assert normwise(out.cpu().numpy(), golden["sgemm_out"]) < F32_TOL
    out = c0.clone()
    api.matmul(dev(golden["sgemm_at"]).t(), bt.t(), out)
    assert normwise(out.cpu().numpy(), golden["sgemm_out_at"]) < F32_TOL


EDGE = [1, 5, 6, 7, 16, 17, 127, 128, 129]


@pytest.mark.parametrize("m,n,k", [(m, n, k) for m in (1, 6, 129) for n in (1, 17, 128) for k in (1, 7, 127)]
                         + [(1024, 1024, 1024)])
def test_fp32_vs_oracle_shapes(L, api, port, m, n, k):
    rng = np.random.default_rng(m * 10007 + n * 101 + k)
    a = rng.standard_normal((m, k)).astype(np.float32)
    b = rng.standard_normal((k, n)).astype(np.float32)
    want = port.matmul(a, b)
    assert normwise(api.matmul(dev(a), dev(b)).cpu().numpy(), want) < F32_TOL
    # the same product through transposed views of transposed storage
    got = api.matmul(dev(a.T.copy()).t(), dev(b.T.copy()).t()).cpu().numpy()
    assert normwise(got, want) < F32_TOL


def test_fp32_config1_seed0(L, api, port):
    """benchmark configuration 1: C[1024,1024] = A.B, A, B ~ N(0,1) from seed 0, rel err 1e-5 vs the CPU result."""
    rng = np.random.default_rng(0)
    a = rng.standard_normal((1024, 1024)).astype(np.float32)
    b = rng.standard_normal((1024, 1024)).astype(np.float32)
    assert normwise(api.matmul(dev(a), dev(b)).cpu().numpy(), port.matmul(a, b)) < F32_TOL


# ------------------------------------------------------------------ 16-bit storage (tcgen05 path)
@pytest.mark.parametrize("name,dt,tdt", [("bf16", 1, torch.bfloat16), ("f16", 2, torch.float16)])
def test_16bit_golden(L, api, port, golden, name, dt, tdt):
    a, b = golden[f"mm16_{name}_a"], golden[f"mm16_{name}_b"]
    widen = port.bf16_to_f32 if dt == 1 else port.f16_to_f32
    want = widen(golden[f"mm16_{name}_c"])
    for path in (2, 1):  # tcgen05, then FFMA: same contract
        L.ytcuda_gemm_set_path(path)
        got_bits = torch_to_bits(api.matmul(bits_to_torch(a, tdt), bits_to_torch(b, tdt)))
        L.ytcuda_gemm_set_path(0)
        assert normwise(widen(got_bits), want) < H_TOL
        status_ok(L)
        # most outputs are bit-identical; the rest differ by one rounding step
        assert (got_bits == golden[f"mm16_{name}_c"]).mean() > 0.9


LAYOUTS = ["kn", "kk", "mn", "mk"]  # A unit stride along k or m; B unit stride along n or k


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (8, 8, 8), (136, 264, 72), (1000, 776, 200), (256, 128, 4096),
                                   (128, 512, 1088)])
def test_bf16_tcgen05_vs_oracle(L, api, port, layout, m, n, k):
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    a = port.f32_to_bf16(rng.standard_normal((m, k)).astype(np.float32))
    b = port.f32_to_bf16((rng.standard_normal((k, n)) / np.sqrt(k)).astype(np.float32))
    want = port.bf16_to_f32(port.matmul_16(a, b, 1))
    ta = bits_to_torch(a, torch.bfloat16) if layout[0] == "k" else bits_to_torch(a.T.copy(), torch.bfloat16).t()
    tb = bits_to_torch(b, torch.bfloat16) if layout[1] == "n" else bits_to_torch(b.T.copy(), torch.bfloat16).t()
    L.ytcuda_gemm_set_path(2)
    try:
        got = port.bf16_to_f32(torch_to_bits(api.matmul(ta, tb)))
    finally:
        L.ytcuda_gemm_set_path(0)
    status_ok(L)
    assert normwise(got, want) < H_TOL


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (1000, 776, 200), (512, 512, 1088), (264, 520, 72)])
def test_bf16_cta_pair_kernel_vs_oracle(L, api, port, layout, m, n, k):
    """The 2-CTA form (cta_group::2, 256 x 256 tile per CTA pair) forced on, against the oracle."""
    rng = np.random.default_rng(m + 5 * n + 11 * k)
    a = port.f32_to_bf16(rng.standard_normal((m, k)).astype(np.float32))
    b = port.f32_to_bf16((rng.standard_normal((k, n)) / np.sqrt(k)).astype(np.float32))
    want = port.bf16_to_f32(port.matmul_16(a, b, 1))
    ta = bits_to_torch(a, torch.bfloat16) if layout[0] == "k" else bits_to_torch(a.T.copy(), torch.bfloat16).t()
    tb = bits_to_torch(b, torch.bfloat16) if layout[1] == "n" else bits_to_torch(b.T.copy(), torch.bfloat16).t()
    L.ytcuda_gemm_set_path(2)
    L.ytcuda_gemm_set_pair_mode(1)
    try:
        got_pair = torch_to_bits(api.matmul(ta, tb))
        L.ytcuda_gemm_set_pair_mode(2)
        got_single = torch_to_bits(api.matmul(ta, tb))
    finally:
        L.ytcuda_gemm_set_path(0)
        L.ytcuda_gemm_set_pair_mode(0)
    status_ok(L)
    assert normwise(port.bf16_to_f32(got_pair), want) < H_TOL
    assert np.array_equal(got_pair, got_single)  # same products, same order of accumulation along k


def test_bf16_fp32_output_is_tight(L, api, port):
    """With fp32 output the tensor-core result matches the fp32 oracle far inside the 16-bit tolerance."""
    rng = np.random.default_rng(5)
    a = port.f32_to_bf16(rng.standard_normal((256, 384)).astype(np.float32))
    b = port.f32_to_bf16(rng.standard_normal((384, 512)).astype(np.float32))
    want = port.matmul(port.bf16_to_f32(a), port.bf16_to_f32(b))
    L.ytcuda_gemm_set_path(2)
    try:
        got = api.matmul(bits_to_torch(a, torch.bfloat16), bits_to_torch(b, torch.bfloat16),
                         out_dtype=torch.float32).cpu().numpy()
    finally:
        L.ytcuda_gemm_set_path(0)
    assert normwise(got, want) < 1e-5


def test_unqualified_layout_uses_ffma_and_matches(L, api, port):
    """Rows that are not 16-byte aligned cannot be fetched by TMA: the FFMA kernel takes over on the device."""
    rng = np.random.default_rng(9)
    a = port.f32_to_bf16(rng.standard_normal((37, 45)).astype(np.float32))
    b = port.f32_to_bf16(rng.standard_normal((45, 29)).astype(np.float32))
    want = port.bf16_to_f32(port.matmul_16(a, b, 1))
    ta, tb = bits_to_torch(a, torch.bfloat16), bits_to_torch(b, torch.bfloat16)
    assert normwise(port.bf16_to_f32(torch_to_bits(api.matmul(ta, tb))), want) < H_TOL
    from ytensor_b200 import _lib
    L.ytcuda_gemm_set_path(2)
    try:
        with pytest.raises(_lib.YtCudaInvalidArgument):
            api.matmul(ta, tb)
    finally:
        L.ytcuda_gemm_set_path(0)


def test_batched_broadcast_and_views(L, api, port):
    rng = np.random.default_rng(11)
    a = port.f32_to_bf16(rng.standard_normal((2, 3, 72, 136)).astype(np.float32))
    b = port.f32_to_bf16((rng.standard_normal((3, 136, 64)) / 12).astype(np.float32))
    fa, fb = port.bf16_to_f32(a), port.bf16_to_f32(b)
    want = np.stack([np.stack([port.matmul(fa[i, j], fb[j]) for j in range(3)]) for i in range(2)])
    got = api.matmul(bits_to_torch(a, torch.bfloat16), bits_to_torch(b, torch.bfloat16), out_dtype=torch.float32)
    assert normwise(got.cpu().numpy(), want) < 1e-5
    # zero-stride (repeated) left operand, as the attention caller repeats K/V over query groups
    a1 = bits_to_torch(a[0, :1], torch.bfloat16).expand(3, 72, 136)
    got = api.matmul(a1, bits_to_torch(b, torch.bfloat16), out_dtype=torch.float32).cpu().numpy()
    want = np.stack([port.matmul(fa[0, 0], fb[j]) for j in range(3)])
    assert normwise(got, want) < 1e-5


def test_alpha_beta_bf16(L, api, port):
    rng = np.random.default_rng(13)
    a = port.f32_to_bf16(rng.standard_normal((128, 64)).astype(np.float32))
    b = port.f32_to_bf16(rng.standard_normal((64, 256)).astype(np.float32))
    c0 = rng.standard_normal((128, 256)).astype(np.float32)
    want = port.sgemm(port.bf16_to_f32(a), port.bf16_to_f32(b), c0, 0.25, -1.5)
    out = dev(c0)
    api.matmul(bits_to_torch(a, torch.bfloat16), bits_to_torch(b, torch.bfloat16), out, alpha=0.25, beta=-1.5)
    assert normwise(out.cpu().numpy(), want) < 1e-5


@pytest.mark.parametrize("m,n,k,batch", [(1024, 1024, 1024, 1), (300, 264, 520, 3), (129, 8, 8, 1), (512, 768, 2048, 2)])
def test_fp32_on_tensor_cores_vs_oracle(L, api, port, m, n, k, batch):
    """fp32 operands split into three bf16 planes, six tcgen05 products accumulated in fp32: the result keeps fp32
    accuracy (same 1e-5 bound as the FFMA kernel), with alpha / beta and a shared or batched right operand."""
    rng = np.random.default_rng(m + n + k)
    a = rng.standard_normal((batch, m, k)).astype(np.float32)
    b = rng.standard_normal((k, n) if batch != 3 else (batch, k, n)).astype(np.float32)
    want = port.matmul(a, b)
    L.ytcuda_gemm_set_f32_mode(2)
    try:
        n0 = L.ytcuda_launch_count()
        got = api.matmul(dev(a), dev(b))
        launches = L.ytcuda_launch_count() - n0
        assert normwise(got.cpu().numpy(), want) < F32_TOL
        # one launch splits both operands (a right operand shared by several batch items is split on its own first),
        # one product over k' = 6 k
        assert launches == (3 if (batch > 1 and batch != 3) else 2)
        c0 = rng.standard_normal((batch, m, n)).astype(np.float32)
        out = dev(c0)
        api.matmul(dev(a), dev(b), out, alpha=0.5, beta=-2.0)
        assert normwise(out.cpu().numpy(), 0.5 * want - 2.0 * c0) < F32_TOL
        # a transposed view of the left operand goes through the same path (the split reads any strides)
        at = dev(np.ascontiguousarray(a.transpose(0, 2, 1)))
        assert normwise(api.matmul(at.transpose(1, 2), dev(b)).cpu().numpy(), want) < F32_TOL
    finally:
        L.ytcuda_gemm_set_f32_mode(0)
    # the FFMA kernel on the same inputs, for the record of both paths
    L.ytcuda_gemm_set_f32_mode(1)
    try:
        assert normwise(api.matmul(dev(a), dev(b)).cpu().numpy(), want) < F32_TOL
    finally:
        L.ytcuda_gemm_set_f32_mode(0)
    status_ok(L)


@pytest.mark.gpu
def test_fp32_on_tensor_cores_extreme_values(L, api):
    """Values next to the largest float go through the three-plane split exactly (rounding the top plane would
    overflow: it is truncated instead). An infinite operand is the one documented deviation: the tensor-core form
    answers NaN in the outputs it reaches, the FFMA kernel answers the infinity as the reference's sgemm does."""
    rng = np.random.default_rng(5)
    m = n = k = 256
    a = rng.standard_normal((m, k)).astype(np.float32)
    b = np.zeros((k, n), dtype=np.float32)
    b[np.arange(k), np.arange(n)] = 0.5  # C = 0.5 * A: no sums, so huge values stay finite
    big = np.float32(3.4e38)             # above the largest bfloat16 after rounding (3.39e38)
    a[3, 7] = big
    a[200, 100] = -np.float32(np.finfo(np.float32).max)
    L.ytcuda_gemm_set_f32_mode(2)
    try:
        got = api.matmul(dev(a), dev(b)).cpu().numpy()
        assert np.isfinite(got).all()
        assert got[3, 7] == np.float32(0.5) * big and got[200, 100] == -np.float32(np.finfo(np.float32).max) * np.float32(0.5)
        assert normwise(got, 0.5 * a) < F32_TOL
        a[5, 9] = np.inf
        got = api.matmul(dev(a), dev(b)).cpu().numpy()
        assert np.isnan(got[5]).any() and np.isfinite(np.delete(got, 5, axis=0)).all()  # the deviation, row 5 only
    finally:
        L.ytcuda_gemm_set_f32_mode(0)
    L.ytcuda_gemm_set_f32_mode(1)
    try:
        got = api.matmul(dev(a), dev(b)).cpu().numpy()
        assert got[5, 9] == np.inf  # as sgemm: inf * 0.5
    finally:
        L.ytcuda_gemm_set_f32_mode(0)
    status_ok(L)


def test_fp32_split_keeps_extreme_values(L, api):
    """Values far apart in magnitude and 24-bit integers: the three-plane split must not lose them. (Non-finite
    inputs are outside the contract of this path: an infinity times the zero low planes of the other operand gives
    NaN where fp32 arithmetic gives infinity; what is checked is that the result is still not finite.)"""
    L.ytcuda_gemm_set_f32_mode(2)
    try:
        a = np.zeros((256, 256), np.float32)
        b = np.eye(256, dtype=np.float32)
        a[0, :4] = [1.0, 2.0 ** -20, 16777215.0, 3.0e38]
        a[1, 0] = np.inf
        a[2, :3] = [1.0 + 2.0 ** -23, -(1.0 + 2.0 ** -23), 1e-30]
        got = api.matmul(dev(a), dev(b)).cpu().numpy()
        assert np.array_equal(got[0, :4], a[0, :4]) and not np.isfinite(got[1, 0]) and np.array_equal(got[2, :3], a[2, :3])
        assert np.all(got[3:] == 0)
    finally:
        L.ytcuda_gemm_set_f32_mode(0)


def test_masked_matmul_golden_and_16bit(L, api, port, golden):
    """YTensor::masked_matmul: products where the mask holds, the fill value elsewhere (mask shared by the batch)."""
    a, mk = golden["mmask_a"], golden["mmask_mask"]
    tm = dev(mk)
    got = api.masked_matmul(dev(a), dev(golden["mmask_b2"]), tm, -1.5).cpu().numpy()
    assert normwise(got, golden["mmask_c_shared"]) < F32_TOL and np.all(got[:, ~mk] == -1.5)
    got = api.masked_matmul(dev(a), dev(golden["mmask_b3"]), tm, 0.0).cpu().numpy()
    assert normwise(got, golden["mmask_c_batched"]) < F32_TOL and np.all(got[:, ~mk] == 0.0)
    # bf16 on the tensor-core path, a strided mask view, fill value rounded as the reference rounds
    rng = np.random.default_rng(5)
    m, n, k = 256, 264, 128
    A = torch.from_numpy(rng.standard_normal((3, m, k)).astype(np.float32)).cuda().to(torch.bfloat16)
    B = torch.from_numpy(rng.standard_normal((k, n)).astype(np.float32)).cuda().to(torch.bfloat16)
    wide = torch.from_numpy(rng.random((m, 2 * n)) < 0.5).cuda()
    mask = wide[:, :n]
    out = api.masked_matmul(A, B, mask, 0.3).float().cpu().numpy()
    want = port.masked_matmul(A.float().cpu().numpy(), B.float().cpu().numpy(), mask.cpu().numpy(), 0.3)
    keep = mask.cpu().numpy()
    assert normwise(out[:, keep], want[:, keep]) < H_TOL
    fill = port.bf16_to_f32(port.f32_to_bf16(np.array([0.3], np.float32)))[0]
    assert np.all(out[:, ~keep] == fill)
    with pytest.raises(ValueError):
        api.masked_matmul(A, B, mask[:, :-1], 0.0)
    status_ok(L)


def test_empty_and_invalid(L, api):
    from ytensor_b200 import _lib
    n0 = L.ytcuda_launch_count()
    out = api.matmul(torch.empty(0, 8, device="cuda"), torch.empty(8, 4, device="cuda"))
    assert out.shape == (0, 4) and L.ytcuda_launch_count() == n0  # empty dims: success, no launch
    z = api.matmul(torch.empty(3, 0, device="cuda"), torch.empty(0, 4, device="cuda"))
    assert torch.equal(z, torch.zeros(3, 4, device="cuda"))  # k == 0: C = beta*C = 0
    with pytest.raises(ValueError):  # std::invalid_argument in the reference (src/ytensor_math.inl:290-292)
        api.matmul(torch.empty(3, 5, device="cuda"), torch.empty(4, 2, device="cuda"))
    with pytest.raises(_lib.YtCudaInvalidArgument):
        api.matmul(torch.empty(3, 5), torch.empty(5, 2))  # host tensors: no CPU fallback


# ------------------------------------------------------------------ full size (benchmark configuration 2)
def test_config2_full_size_properties(L, api, port):
    """[64,2048,4096] x [4096,4096] bf16. The oracle needs about a minute per batch item, so the full size is
    checked through properties: (1) B = a permutation matrix moves columns exactly (bit-exact);
    (2) sampled rows against the oracle."""
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randn(64, 2048, 4096, device="cuda", generator=g).to(torch.bfloat16)
    perm = torch.randperm(4096, device="cuda", generator=g)
    p = torch.zeros(4096, 4096, device="cuda", dtype=torch.bfloat16)
    p[perm, torch.arange(4096, device="cuda")] = 1  # column j of A.P is column perm[j] of A
    c = api.matmul(a, p)
    status_ok(L)
    assert torch.equal(c, a[:, :, perm])
    b = (torch.randn(4096, 4096, device="cuda", generator=g) / 64).to(torch.bfloat16)
    c = api.matmul(a, b)
    status_ok(L)
    rows = [(0, 0), (21, 777), (42, 1024), (63, 2047)]
    a_rows = np.stack([torch_to_bits(a[i, r]) for i, r in rows])
    want = port.bf16_to_f32(port.matmul_16(a_rows[None], torch_to_bits(b), 1))[0]
    got = np.stack([port.bf16_to_f32(torch_to_bits(c[i, r])) for i, r in rows])
    assert normwise(got, want) < H_TOL


def test_host_buffer_variant_matches_device(L, api):
    from ytensor_b200 import _lib
    g = torch.Generator().manual_seed(3)
    a = torch.randn(6, 512, 1024, generator=g).to(torch.bfloat16).pin_memory()
    b = (torch.randn(1024, 768, generator=g) / 32).to(torch.bfloat16).pin_memory()
    c = torch.empty(6, 512, 768, dtype=torch.bfloat16).pin_memory()
    _lib.check(L.ytcuda_gemm_host(_lib.BF16, _lib.BF16, a.data_ptr(), b.data_ptr(), c.data_ptr(), 512, 768, 1024, 1.0,
                                  0.0, 1024, 1, 768, 1, 768, 1, 6, 512 * 1024, 0, 512 * 768))
    want = api.matmul(a.cuda(), b.cuda()).cpu()
    assert torch.equal(c, want)
    # pageable memory and a C view with a row pitch
    a2, b2 = a.clone(), b.clone()
    cbig = torch.full((6, 512, 800), 7.0, dtype=torch.bfloat16)
    cv = cbig[:, :, :768]
    _lib.check(L.ytcuda_gemm_host(_lib.BF16, _lib.BF16, a2.data_ptr(), b2.data_ptr(), cv.data_ptr(), 512, 768, 1024,
                                  1.0, 0.0, 1024, 1, 768, 1, 800, 1, 6, 512 * 1024, 0, 512 * 800))
    assert torch.equal(cv, want)
    assert torch.all(cbig[:, :, 768:] == 7.0)  # the gap between rows is left alone


# ------------------------------------------------------------------ rewritten operands, k in pieces
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,m,n,k,form", [
    (1, 60, 1001, 1111, "shared"), (1, 257, 513, 1027, "linear"), (3, 129, 255, 777, "batched"), (2, 300, 301, 517, "shared"),
    (1, 16, 4096, 4096, "shared"), (1, 1, 700, 2048, "linear"), (1, 100, 130, 4104, "columns"), (2, 64, 96, 8191, "batched")])
def test_odd_sizes_and_k_pieces(api, dt, batch, m, n, k, form):
    gen = torch.Generator(device="cuda").manual_seed(m * n + k)
    a = torch.randn(batch, m, k, generator=gen, device="cuda").to(dt)
    b = (torch.randn(*([batch] if form == "batched" else []), k, n, generator=gen, device="cuda") * k ** -0.5).to(dt)
    if form == "columns":  # both operands by columns
        a, b = a.transpose(-1, -2).contiguous().transpose(-1, -2), b.transpose(-1, -2).contiguous().transpose(-1, -2)
    if form == "linear":
        got = api.linear(a, b.transpose(-1, -2).contiguous())
    else:
        got = api.matmul(a, b)
    want = a.double() @ b.double()
    # fp32: a rounding per partial sum; 16 bits: the rounding of the result (bf16 by the reference's rule: up to one unit)
    tol = {torch.float32: 2e-6, torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -11}[dt]
    assert (got.double() - want).abs().max() <= tol * want.abs().max()


def test_small_fp32_products_keep_infinities(api):
    gen = torch.Generator(device="cuda").manual_seed(9)
    a, b = torch.randn(64, 2050, generator=gen, device="cuda"), torch.randn(2050, 1500, generator=gen, device="cuda")
    a[5, 9] = float("inf")
    b[:, 77] = 0.0
    want = a.double() @ b.double()
    got = api.matmul(a, b)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    fin = want.isfinite()
    assert (got.double() - want)[fin].abs().max() <= 1e-5 * want[fin].abs().max()


# More than 74 tiles of 256 x 256: the size from which whole products go to the CTA-pair kernel.
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,m,n,k,form", [
    (1, 2048, 2500, 1024, "shared"), (1, 600, 20001, 777, "linear"), (8, 1000, 1001, 1001, "batched"), (1, 2500, 2500, 1300, "columns"),
    (1, 513, 19000, 513, "shared")])
@pytest.mark.parametrize("pair_mode", [0, 1, 2])
def test_large_odd_products(L, api, dt, batch, m, n, k, form, pair_mode):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    # the scratch of this stream holds NaN before: a part of it that is read without having been written shows
    api.matmul(torch.full((300, 8191), float("nan"), device="cuda"), torch.zeros(8191, 1001, device="cuda"))
    a = torch.randn(batch, m, k, generator=gen, device="cuda").to(dt)
    b = (torch.randn(*([batch] if form == "batched" else []), k, n, generator=gen, device="cuda") * k ** -0.5).to(dt)
    if form == "columns":  # both operands by columns
        a, b = a.transpose(-1, -2).contiguous().transpose(-1, -2), b.transpose(-1, -2).contiguous().transpose(-1, -2)
    w = b.transpose(-1, -2).contiguous()
    L.ytcuda_gemm_set_pair_mode(pair_mode)
    try:
        got = api.linear(a, w) if form == "linear" else api.matmul(a, b)
    finally:
        L.ytcuda_gemm_set_pair_mode(0)
    # fp32: a rounding per partial sum; 16 bits: the rounding of the result (bf16 by the reference's rule: up to one unit)
    tol = {torch.float32: 2e-6, torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -11}[dt]
    for i in range(batch):
        want = a[i].double() @ (b[i] if form == "batched" else b).double()
        assert (got[i].double() - want).abs().max() <= tol * want.abs().max()
    assert L.ytcuda_device_status(None) == 0


def _scratch_high():
    """Most bytes that were in use at once in the device's default memory pool (the library's scratch) since the last call."""
    rt, driver = pytest.importorskip("cuda.bindings.runtime"), pytest.importorskip("cuda.bindings.driver")
    pool, attr = rt.cudaDeviceGetDefaultMemPool(0)[1], rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh
    torch.cuda.synchronize()
    high = int(rt.cudaMemPoolGetAttribute(pool, attr)[1])
    rt.cudaMemPoolSetAttribute(pool, attr, driver.cuuint64_t(0))  # (back to what is in use now)
    return high


@pytest.mark.parametrize("batch,m,n,k", [(1, 300, 1001, 30001), (1, 130, 8191, 9000), (1, 2001, 2002, 4099), (40, 150, 701, 3001),
                                         (1, 5001, 6000, 1025)])
def test_odd_products_in_bounded_scratch(api, batch, m, n, k):
    """Small odd fp32 products use no more scratch than a stream keeps, and no more of it when k doubles."""
    gen = torch.Generator(device="cuda").manual_seed(k)
    used = []
    for kk in (k, 2 * k):
        a = torch.randn(batch, m, kk, generator=gen, device="cuda")
        b = torch.randn(kk, n, generator=gen, device="cuda") * kk ** -0.5
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        _scratch_high()
        before = _scratch_high()
        with torch.cuda.stream(stream):
            got = api.matmul(a, b)
        used.append(_scratch_high() - before)
        for i in range(0, batch, 13):
            want = a[i].double() @ b.double()
            assert (got[i].double() - want).abs().max() <= 2e-6 * want.abs().max()
    assert max(used) <= 256 << 20
    assert used[1] <= max(used[0], 250 << 20)


@pytest.mark.parametrize("dt,m,n,k", [(torch.float32, 700, 2501, 1030), (torch.float32, 1024, 2048, 1024), (torch.bfloat16, 1300, 2501, 1111),
                                      (torch.float16, 1300, 2501, 1111), (torch.bfloat16, 128, 8192, 8192)])
def test_products_without_scratch(api, dt, m, n, k):
    """Where the device has no room for scratch the kernels that need none take the product."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    gen = torch.Generator(device="cuda").manual_seed(k)
    a = torch.randn(m, k, generator=gen, device="cuda").to(dt)
    b = (torch.randn(k, n, generator=gen, device="cuda") * k ** -0.5).to(dt)
    out = torch.empty(m, n, dtype=dt, device="cuda")
    torch.cuda.synchronize()
    props = rt.cudaMemPoolProps()
    props.allocType, props.location.type, props.location.id = rt.cudaMemAllocationType.cudaMemAllocationTypePinned, \
        rt.cudaMemLocationType.cudaMemLocationTypeDevice, 0
    props.maxSize = 4 << 20
    err, pool = rt.cudaMemPoolCreate(props)
    assert int(err) == 0
    old = rt.cudaDeviceGetMemPool(0)[1]
    err, handle = rt.cudaStreamCreateWithFlags(1)  # (a stream that has no scratch yet; kept, so that its name is not given again)
    try:
        assert int(rt.cudaDeviceSetMemPool(0, pool)[0]) == 0
        with torch.cuda.stream(torch.cuda.ExternalStream(int(handle))):
            api.matmul(a, b, out)
        torch.cuda.synchronize()
    finally:
        rt.cudaDeviceSetMemPool(0, old)
    want = a.double() @ b.double()
    tol = {torch.float32: 1e-5, torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -11}[dt]
    assert (out.double() - want).abs().max() <= tol * want.abs().max()


@pytest.mark.parametrize("sa,sb", [(2.0 ** 70, 2.0 ** 70), (2.0 ** 64, 2.0 ** 61), (2.0 ** -118, 2.0 ** 20), (2.0 ** -60, 2.0 ** -55)])
@pytest.mark.parametrize("m,n,k", [(70, 1001, 1300), (600, 9001, 515)])
def test_small_and_odd_products_at_the_ends_of_the_range(L, api, sa, sb, m, n, k):
    """Results beyond the largest float are what FFMA says, operands near the smallest lose nothing."""
    gen = torch.Generator(device="cuda").manual_seed(m)
    a, b = torch.randn(m, k, generator=gen, device="cuda"), torch.randn(k, n, generator=gen, device="cuda")
    a[:, 5::3], b[:, 9::2] = a[:, 5::3] * sa, b[:, 9::2] * sb  # (ordinary numbers beside them)
    if sa < 1:
        a[:, 0:5] = 0
        a[:, 6::3] = a[:, 7::3] = 0
    got = api.matmul(a, b)
    L.ytcuda_gemm_set_path(1)
    try:
        ffma = api.matmul(a, b)
    finally:
        L.ytcuda_gemm_set_path(0)
    want, fin = a.double() @ b.double(), ffma.isfinite()
    # (a partial sum may overflow in one order and not in another: where the result is beyond any doubt)
    size = a.double().abs() @ b.double().abs()
    sure = (want.abs() > 2.0 ** 130) | (size < 2.0 ** 126)
    assert torch.equal(got.isnan() & sure, ffma.isnan() & sure) and torch.equal(got.isinf() & sure, ffma.isinf() & sure)
    inf = sure & ffma.isinf()
    assert torch.equal(got[inf], ffma[inf])
    fin = sure & fin
    assert fin.any() and ((got.double() - want)[fin].abs() <= 2e-6 * size[fin]).all()


def test_threads_share_a_stream(api):
    """Two threads that queue products and attention on one stream: each call's launches hand scratch to one another, and none of
    the other thread's may come between them."""
    import threading
    gen = torch.Generator(device="cuda").manual_seed(2)

    def work(i):
        a = torch.randn(30 + 200 * i, 2050, generator=gen, device="cuda")
        b = torch.randn(2050, 601 + 100 * i, generator=gen, device="cuda")
        q, k, v = (torch.randn(1, 2, 200 + 300 * i, 64, generator=gen, device="cuda") for _ in range(3))
        h = torch.randn(16, 8192, generator=gen, device="cuda").bfloat16()
        w = torch.randn(300 + 100 * i, 8192, generator=gen, device="cuda").bfloat16()
        long = torch.randn(2, 3, 40000 + i, generator=gen, device="cuda")
        return [lambda: api.matmul(a, b), lambda: api.scaledDotProductAttention(q, k, v, causal=True), lambda: api.linear(h, w),
                lambda: api.scaledDotProductAttention(q[:, :, -1:], k, v), lambda: api.sum(long, -1)]

    calls = [work(0), work(1)]
    want = [[f() for f in c] for c in calls]
    bad, stream = [], torch.cuda.current_stream()

    def loop(i):
        with torch.cuda.stream(stream):
            for _ in range(60):
                for f, x in zip(calls[i], want[i]):
                    bad.append((f() != x).any())

    threads = [threading.Thread(target=loop, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not torch.stack(bad).any()


@pytest.mark.parametrize("b,m,n,k", [(1, 60, 1001, 180), (1, 777, 1001, 200), (3, 130, 203, 255), (1, 1, 1999, 256), (1, 200, 1501, 181)])
def test_odd_rows_of_one_piece_are_copied_into_place(L, api, b, m, n, k):
    """fp32 products of at most 256 of k whose C has rows off 16 bytes go through partial sums of one piece: 64-bit reference, an infinity
    and a NaN where FFMA answers, C inside a larger tensor, and nothing outside C. fp32 sums of 256 products: the file's tolerance."""
    g = torch.Generator(device="cuda").manual_seed(m + k)
    a, w = torch.randn(b, m, k, generator=g, device="cuda"), torch.randn(k, n, generator=g, device="cuda")
    whole = torch.full((b, m, n + 3), 7.0, device="cuda")
    api.matmul(a, w, whole[:, :, 1:n + 1])
    assert normwise(whole[:, :, 1:n + 1].double().cpu().numpy(), (a.double() @ w.double()).cpu().numpy()) < F32_TOL
    assert bool((whole[:, :, 0] == 7).all()) and bool((whole[:, :, n + 1:] == 7).all())
    a[0, m // 2, 3] = float("inf") if m > 1 else 1.0
    w[k - 1, n // 2] = float("nan")
    got, want = api.matmul(a, w), a.double() @ w.double()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    fine = want.isfinite()
    assert float((got.double() - want)[fine].abs().max()) < F32_TOL * float(want[fine].abs().max())
    status_ok(L)


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("b,m,n,k", [(1, 1, 8, 72), (1, 33, 24, 64), (3, 127, 136, 200), (1, 129, 264, 72), (2, 160, 520, 136),
                                     (1, 4097, 1032, 264), (2, 2304, 1288, 256)])
def test_results_through_tma_stores(L, api, out_dtype, b, m, n, k):
    """C whose rows start at 16 bytes leaves through TMA stores, other C through stores of the lanes: the same bits, and nothing
    outside C, at the edges of tiles of both kernels."""
    dt = torch.float16 if out_dtype == torch.float16 else torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a, w = (torch.randn(s, generator=g, device="cuda").to(dt) for s in ((b, m, k), (k, n)))
    got = []
    for first in (8, 1):  # (an odd place in the row: no 16-byte rows)
        whole = torch.full((b, m + 2, n + 16), 7.0, dtype=out_dtype, device="cuda")
        api.matmul(a, w, whole[:, 1:m + 1, first:first + n])
        got.append(whole[:, 1:m + 1, first:first + n].clone())
        whole[:, 1:m + 1, first:first + n] = 7.0
        assert bool((whole == 7.0).all())
    assert torch.equal(got[0], got[1])
    assert normwise(got[0].double().cpu().numpy(), (a.double() @ w.double()).cpu().numpy()) < (1e-5 if out_dtype == torch.float32 else H_TOL)
    status_ok(L)


@pytest.mark.parametrize("b,m,n,k,dt", [(1, 500, 1024, 2304, "bf16"), (1, 1, 136, 4096, "f16"), (3, 130, 264, 2056, "bf16"), (2, 300, 700, 1088, "f16"),
                                        (1, 1024, 1032, 1032, "bf16"), (1, 1024, 1024, 520, "f32"),
                                        (1, 700, 264, 512, "f32"), (1, 1000, 2000, 256, "f32")])
def test_k_shared_by_a_cluster(L, api, b, m, n, k, dt):
    """Few tiles and a long k: the CTAs of a cluster take a piece of k each. Two and four pieces, planes of fp32
    operands, ragged m, n and k, operands of either order, aligned and other C, alpha and beta. 64-bit reference: fp32 sums of k
    products are off by less than the file's tolerances."""
    t = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}[dt]
    g = torch.Generator(device="cuda").manual_seed(m + k)
    a, w = (torch.randn(s, generator=g, device="cuda").to(t) for s in ((b, m, k), (k, n)))
    want = (a.double() @ w.double()).cpu().numpy()
    tol = F32_TOL if dt == "f32" else H_TOL
    for x in (a, a.transpose(1, 2).contiguous().transpose(1, 2)):
        for y in (w, w.t().contiguous().t()):
            assert normwise(api.matmul(x, y).double().cpu().numpy(), want) < tol
    if dt != "f32":
        wide = api.matmul(a, w, out_dtype=torch.float32)
        assert normwise(wide.double().cpu().numpy(), want) < 1e-5
        assert torch.equal(wide, api.matmul(a, w, out_dtype=torch.float32))
    out = torch.ones(b, m, n + 1, dtype=t, device="cuda")[:, :, 1:]
    api.matmul(a, w, out, alpha=0.5, beta=2.0)
    assert normwise(out.double().cpu().numpy(), 0.5 * want + 2.0) < tol
    status_ok(L)
