"""GPU parity tests of the decoder (ytcuda_qwen3_*) against the reference example model.

Contract: fp32 logits within 1e-4 of the reference's (normwise; fp32 sums in another order over 28 layers), and
argmax-identical greedy tokens for the first 32 decode steps on the Qwen3-0.6B shape with random bf16 weights."""
import hashlib

import numpy as np
import pytest

from _util import normwise

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SMALL = dict(hidden_size=64, num_hidden_layers=2, vocab_size=512, intermediate_size=96, num_attention_heads=4,
             num_key_value_heads=2, head_dim=128, max_position_embeddings=64)


@pytest.fixture(scope="module")
def qwen3_golden():
    from pathlib import Path
    return np.load(Path(__file__).resolve().parent / "golden" / "golden_qwen3.npz")


@pytest.fixture(scope="module")
def Q():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ytensor_b200 import qwen3
    return qwen3


def dev_ids(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.int32)).cuda()


@pytest.mark.parametrize("B", [1, 2])
def test_small_model_logits_match_reference(Q, qwen3_golden, B):
    cfg = Q.Qwen3Config(**SMALL)
    w = Q.random_weights(cfg, seed=4, std=0.05)
    assert hashlib.sha256(w["embed"].tobytes()).hexdigest() == str(qwen3_golden["small_embed_sha256"])
    m = Q.Qwen3ForCausalLM(cfg, batch=B)
    m.load_weights(w)
    want = qwen3_golden[f"small_logits_b{B}"]
    logits = m.forward(dev_ids(qwen3_golden[f"small_ids_b{B}"]))
    for step in range(6):
        got = logits.cpu().numpy()
        assert normwise(got, want[step]) < 1e-4
        assert np.array_equal(got.argmax(1), want[step].argmax(1))
        if step < 5:
            logits = m.forward(dev_ids(want[step].argmax(1).reshape(B, 1)))
    assert m.get_kv_cache_len() == 9 + 5
    m.reset_kv_cache()
    assert m.get_kv_cache_len() == 0
    m.close()


@pytest.mark.parametrize("B", [1, 2, 3, 4, 5, 8, 13, 16, 32])
def test_single_kernel_decode_step_matches_operator_path(Q, B):
    """The persistent step kernel (path 2: up to four sequences without grid barriers, activations exchanged as
    tagged pairs, weights streamed through a shared-memory ring, linear phases on mma.sync from bf16 planes of the
    activations; from five sequences on the kernel with grid barriers and tensor-core linear phases;
    path 3: FFMA linear phases where the kernel with grid barriers runs; path 4: the form without the weight ring;
    path 5: the ring with grid barriers)
    and the one-launch-per-operator forward compute the same logits and leave the same KV cache behind: 70 steps
    after a 40-token prompt (the attention of the step kernel goes from 2 to 4 key chunks), every model fed the
    tokens of the operator path."""
    # (the FFN width is larger than what the step kernel stages at once: the down projection then takes its input in
    # pieces, the last one shorter)
    cfg = Q.Qwen3Config(hidden_size=256, num_hidden_layers=3, vocab_size=1000, intermediate_size=2816,
                        num_attention_heads=4, num_key_value_heads=2, head_dim=128, max_position_embeddings=128)
    w = Q.random_weights(cfg, seed=11, std=0.05)
    ids = dev_ids(np.random.default_rng(B).integers(0, cfg.vocab_size, (B, 40)))
    ms = []
    for path in (1, 2, 3, 4, 5):
        m = Q.Qwen3ForCausalLM(cfg, batch=B)
        m.load_weights(w)
        m.set_decode_path(path)
        ms.append(m)
    # a single token into an empty cache (no prefill before it), then start over with the prompt
    first = ids[:, :1].contiguous()
    fa = ms[0].forward(first).cpu().numpy()
    for m in ms[1:]:
        assert normwise(m.forward(first).cpu().numpy(), fa) < 2e-5
    for m in ms:
        m.reset_kv_cache()
    la = ms[0].forward(ids)  # prefill: the same kernels in all three
    for m in ms[1:]:
        assert torch.equal(la, m.forward(ids))
    count = Q._lib.lib().ytcuda_launch_count
    for step in range(70):
        tok, _ = ms[0].argmax(la)
        tok = tok.reshape(B, 1).contiguous()
        n0 = count()
        la = ms[0].forward(tok)
        assert count() - n0 > 20
        a = la.cpu().numpy()
        for m in ms[1:]:
            n0 = count()
            lb = m.forward(tok)
            assert count() - n0 == 1
            assert normwise(lb.cpu().numpy(), a) < 2e-5, f"step {step}"
    assert all(m.get_kv_cache_len() == 110 for m in ms)
    assert Q._lib.lib().ytcuda_device_status(None) == 0
    for m in ms:
        m.close()
    if B == 32:  # more sequences than the step kernel holds: forcing it is refused, not silently rerouted
        m = Q.Qwen3ForCausalLM(cfg, batch=33)
        m.load_weights(w)
        m.set_decode_path(2)
        m.forward(dev_ids(np.zeros((33, 4))))
        with pytest.raises(Exception):
            m.forward(dev_ids(np.zeros((33, 1))))
        m.close()


@pytest.mark.parametrize("B,heads,kv_heads,inter,prompt,steps", [
    (5, 4, 2, 2816, 30, 3), (6, 4, 4, 256, 1, 2), (7, 8, 2, 768, 12, 3), (8, 4, 4, 256, 1, 2), (9, 8, 2, 768, 62, 3), (16, 4, 2, 2048, 20, 2),
    (17, 16, 8, 512, 7, 2), (31, 8, 8, 1536, 12, 2), (32, 16, 8, 512, 9, 2)])
def test_decode_steps_of_several_sequences_match_the_port(Q, port, B, heads, kv_heads, inter, prompt, steps):
    """Automatic steps of 5 to 32 sequences against the CPU port, from an empty cache and behind a prompt, group sizes 1, 2 and 4. Up to 6
    sequences a step is the one launch of decode_step_kernel, from 7 on one launch per operator, as decode_kernel_name() says.
    fp32 logits: 1e-4, the contract at the head of this file."""
    cfg = Q.Qwen3Config(hidden_size=256 if heads < 16 else 1024, num_hidden_layers=2, vocab_size=500, intermediate_size=inter,
                        num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=128, max_position_embeddings=160)
    w = Q.random_weights(cfg, seed=21, std=0.05)
    ids = np.random.default_rng(B).integers(0, cfg.vocab_size, (B, prompt + steps)).astype(np.int32)
    m = Q.Qwen3ForCausalLM(cfg, batch=B)
    m.load_weights(w)
    assert m.decode_kernel_name().startswith("decode_step_kernel" if B <= 6 else "gemm_tc_kernel")
    count = Q._lib.lib().ytcuda_launch_count
    for first in (0, prompt):  # from an empty cache, then behind the prompt
        ref = port.qwen3(cfg.oracle_dict(), batch=B)
        for key, arr in w.items():
            name, layer = (key, 0) if isinstance(key, str) else key
            ref.set_weight(name, layer, Q.bf16_bits_to_f32(arr) if arr.dtype == np.uint16 else arr)
        m.reset_kv_cache()
        if first:
            m.forward(dev_ids(ids[:, :first]))
            ref.forward(np.ascontiguousarray(ids[:, :first]))
        for t in range(first, first + steps):
            n0 = count()
            got = m.forward(dev_ids(ids[:, t:t + 1]))
            assert count() - n0 == 1 if B <= 6 else count() - n0 > 8 * cfg.num_hidden_layers
            assert normwise(got.cpu().numpy(), ref.forward(np.ascontiguousarray(ids[:, t:t + 1]))) < 1e-4, (first, t)
        ref.close()
    assert Q._lib.lib().ytcuda_device_status(None) == 0
    m.close()


def test_long_prefill_uses_tensor_cores_and_matches_oracle(Q, port):
    """More than 32 rows: activations are split into two bf16 planes and multiplied on tcgen05."""
    cfg = Q.Qwen3Config(**SMALL)
    w = Q.random_weights(cfg, seed=5, std=0.05)
    ids = np.random.default_rng(1).integers(0, cfg.vocab_size, (2, 40)).astype(np.int32)
    om = port.qwen3(cfg.oracle_dict(), 2)
    for key, arr in w.items():
        name, layer = (key, 0) if isinstance(key, str) else key
        om.set_weight(name, layer, Q.bf16_bits_to_f32(arr) if arr.dtype == np.uint16 else arr)
    want = om.forward(ids)
    m = Q.Qwen3ForCausalLM(cfg, batch=2)
    m.load_weights(w)
    got = m.forward(dev_ids(ids)).cpu().numpy()
    assert normwise(got, want) < 1e-4
    nxt = want.argmax(1).astype(np.int32).reshape(2, 1)
    assert normwise(m.forward(dev_ids(nxt)).cpu().numpy(), om.forward(nxt)) < 1e-4
    m.close()
    om.close()


@pytest.mark.parametrize("path", [1, 2])
def test_ring_buffer_cache_past_its_end_matches_reference(Q, path):
    """The reference's KV cache is a ring buffer: past its end a token overwrites the oldest slot, sees every slot and
    takes rotary position 0. Golden logits: 9-token prompt + 19 steps with max_position_embeddings = 16."""
    from pathlib import Path
    from ytensor_b200 import _lib
    g = np.load(Path(__file__).resolve().parent / "golden" / "golden_qwen3_wrap.npz")
    cfg = Q.Qwen3Config(**{**SMALL, "max_position_embeddings": 16})
    m = Q.Qwen3ForCausalLM(cfg, batch=1)
    m.load_weights(Q.random_weights(cfg, seed=4, std=0.05))
    m.set_decode_path(path)
    want = g["wrap_logits"]
    logits = m.forward(dev_ids(g["wrap_ids"]))
    for step in range(20):
        got = logits.cpu().numpy()
        assert normwise(got, want[step]) < 1e-4, step
        assert np.array_equal(got.argmax(1), want[step].argmax(1))
        assert m.get_kv_cache_len() == min(9 + step, 16)
        if step < 19:
            logits = m.forward(dev_ids(want[step].argmax(1).reshape(1, 1)))
    with pytest.raises(_lib.YtCudaInvalidArgument):  # more tokens at once than the ring has slots: refused
        m.forward(dev_ids(np.zeros((1, 17), np.int32)))
    m.close()


def test_several_tokens_per_call_across_the_end_of_the_ring(Q):
    """A forward of several tokens that runs over the end of the cache: every token is appended (the later ones
    overwrite the oldest slots), each query sees the slots that are not younger than itself, and the rotary positions
    restart as in Qwen3Model::forward (reference qwen3.cpp:70-126, 365-375). Golden logits: calls of 9, 5, 6, 3, 1 and
    10 tokens into a ring of 16 slots, two sequences."""
    from pathlib import Path
    g = np.load(Path(__file__).resolve().parent / "golden" / "golden_qwen3_wrap.npz")
    cfg = Q.Qwen3Config(**{**SMALL, "max_position_embeddings": 16})
    m = Q.Qwen3ForCausalLM(cfg, batch=2)
    m.load_weights(Q.random_weights(cfg, seed=4, std=0.05))
    want = g["multi_logits"]
    for i in range(want.shape[0]):
        got = m.forward(dev_ids(g[f"multi_ids_{i}"])).cpu().numpy()
        assert normwise(got, want[i]) < 1e-4, i
        assert np.array_equal(got.argmax(1), want[i].argmax(1)), i
    assert m.get_kv_cache_len() == 16
    m.close()


def test_cache_overflow_is_reported(Q):
    from ytensor_b200 import _lib
    cfg = Q.Qwen3Config(**SMALL)
    m = Q.Qwen3ForCausalLM(cfg, batch=1)
    m.load_weights(Q.random_weights(cfg, seed=4, std=0.05))
    m.forward(dev_ids(np.zeros((1, 60), np.int32)))
    m.forward(dev_ids(np.zeros((1, 5), np.int32)))  # runs over the end of the 64-slot ring: allowed
    assert m.get_kv_cache_len() == 64
    with pytest.raises(_lib.YtCudaInvalidArgument):  # more tokens than the ring has slots
        m.forward(dev_ids(np.zeros((1, 65), np.int32)))
    m.close()


def test_linear_w16_kernels(Q, port):
    from ytensor_b200 import _lib
    L = _lib.lib()
    rng = np.random.default_rng(2)
    for M, N, K in [(1, 1000, 1024), (3, 200, 768), (5, 77, 512), (32, 300, 3072), (100, 256, 1024), (9, 8, 8)]:
        x = rng.standard_normal((M, K)).astype(np.float32)
        wb = Q.f32_to_bf16_bits((rng.standard_normal((N, K)) * 0.05).astype(np.float32))
        want = port.matmul(x, np.ascontiguousarray(Q.bf16_bits_to_f32(wb).T))
        tx = torch.from_numpy(x).cuda()
        tw = torch.from_numpy(wb.view(np.int16)).cuda()
        y = torch.empty(M, N, device="cuda")
        scratch = torch.empty(4 * M * K, dtype=torch.uint8, device="cuda")
        _lib.check(L.ytcuda_linear_w16(tx.data_ptr(), K, tw.data_ptr(), y.data_ptr(), N, M, N, K, 0,
                                       scratch.data_ptr(), None))
        assert normwise(y.cpu().numpy(), want) < 2e-5
        _lib.check(L.ytcuda_linear_w16(tx.data_ptr(), K, tw.data_ptr(), y.data_ptr(), N, M, N, K, 1,
                                       scratch.data_ptr(), None))
        assert normwise(y.cpu().numpy(), 2 * want) < 2e-5


def test_full_model_greedy_tokens_match_reference(Q, qwen3_golden):
    """benchmark configuration 5, batch 1: 512-token prompt, 32 greedy steps, tokens identical to the reference's."""
    cfg = Q.Qwen3Config(max_position_embeddings=768)
    w = Q.random_weights(cfg, seed=4)
    assert hashlib.sha256(w["embed"].tobytes()).hexdigest() == str(qwen3_golden["full_embed_sha256"])
    m = Q.Qwen3ForCausalLM(cfg, batch=1)
    m.load_weights(w)
    logits = m.forward(dev_ids(qwen3_golden["full_prompt"]))
    want_tok, top_i, top_v = qwen3_golden["full_tokens"], qwen3_golden["full_top8_indices"], qwen3_golden["full_top8_values"]
    for s in range(32):
        tok, _ = m.argmax(logits)
        got = logits[0].cpu().numpy()
        assert int(tok[0]) == int(want_tok[s]), f"step {s}: margin in the reference was {qwen3_golden['full_margins'][s]}"
        assert np.abs(got[top_i[s]] - top_v[s]).max() < 1e-3
        if s < 31:
            logits = m.forward(tok.reshape(1, 1).contiguous())
    # batch 2 with the same prompt twice gives the same tokens in both rows
    m.close()
    m2 = Q.Qwen3ForCausalLM(cfg, batch=2)
    m2.load_weights(w)
    p2 = np.repeat(qwen3_golden["full_prompt"], 2, axis=0)
    toks = m2.generate_greedy(dev_ids(p2), 8).cpu().numpy()
    assert np.array_equal(toks[0], want_tok[:8]) and np.array_equal(toks[1], want_tok[:8])
    m2.close()


def qkv_post(Q, qkv, qn, kn, cos, sin, B, T, H, G, max_len, pos0, slot0, eps, off):
    """ytcuda_qwen3_qkv_post on numpy arrays, every tensor `off` floats behind a 16-byte boundary -> q, k_cache, v_cache (7 where
    nothing was written)."""
    from ytensor_b200 import _lib

    def place(shape, a=None):
        t = torch.full((off + int(np.prod(shape)),), 7.0, device="cuda")[off:].reshape(shape)
        return t if a is None else t.copy_(torch.from_numpy(np.ascontiguousarray(a, np.float32)))

    q, kc, vc = place((B, H, T, 128)), place((B, G, max_len, 128)), place((B, G, max_len, 128))
    ins = [place(a.shape, a) for a in (qkv, qn, kn, cos, sin)]
    _lib.check(_lib.lib().ytcuda_qwen3_qkv_post(ins[0].data_ptr(), q.data_ptr(), kc.data_ptr(), vc.data_ptr(),
                                                *(t.data_ptr() for t in ins[1:]), B, T, H, G, 128, max_len, pos0, slot0, eps,
                                                torch.cuda.current_stream().cuda_stream))
    return [t.cpu().numpy() for t in (q, kc, vc)]


# up to 2367 groups of four heads a warp takes one head, from 2368 on (16 warps an SM) four; heads that four does not divide
QKV_POST = [(1, 3, 4, 2, 0), (2, 5, 3, 1, 1), (1, 1183, 5, 1, 0), (1, 1184, 5, 1, 0), (2, 700, 3, 1, 0), (1, 1300, 5, 1, 3), (3, 200, 14, 2, 0)]


@pytest.mark.parametrize("B,T,H,G,off", QKV_POST)
def test_norms_behind_the_qkv_projection_round_as_fp32_does(Q, B, T, H, G, off):
    """Small whole numbers make the sums of squares exact, and cos = 1, sin = 0 leave the norm alone: (x / rms) * w in fp32, to the bit.
    The ring ends inside the new tokens."""
    rng = np.random.default_rng(T)
    qkv = rng.integers(-8, 9, (B, T, H + 2 * G, 128)).astype(np.float32)
    qn, kn = (rng.uniform(0.5, 1.5, 128).astype(np.float32) for _ in range(2))
    max_len, pos0, slot0, eps = T + 9, 4, T + 7, np.float32(1e-6)
    cos, sin = np.ones((max_len, 128), np.float32), np.zeros((max_len, 128), np.float32)
    q, kc, vc = qkv_post(Q, qkv, qn, kn, cos, sin, B, T, H, G, max_len, pos0, slot0, eps, off)
    rms = np.sqrt((qkv * qkv).sum(-1, keepdims=True) / np.float32(128) + eps)
    x = (qkv / rms).transpose(0, 2, 1, 3)
    slots = (slot0 + np.arange(T)) % max_len
    assert np.array_equal(q, x[:, :H] * qn)
    assert np.array_equal(kc[:, :, slots], x[:, H:H + G] * kn)
    assert np.array_equal(vc[:, :, slots], qkv.transpose(0, 2, 1, 3)[:, H + G:])
    rest = np.setdiff1d(np.arange(max_len), slots)
    assert (kc[:, :, rest] == 7).all() and (vc[:, :, rest] == 7).all()


@pytest.mark.parametrize("B,T,H,G,off", QKV_POST)
def test_rotation_reads_the_first_half_of_the_tables(Q, B, T, H, G, off):
    """Rotate-half RoPE against float64: 1e-6 normwise (fp32 products, one rounding each of x / rms, times w and two of the rotation).
    Values 64 .. 127 of a row of the tables are not read: NaN there changes nothing."""
    rng = np.random.default_rng(T + 1)
    qkv = rng.standard_normal((B, T, H + 2 * G, 128)).astype(np.float32)
    qn, kn = (rng.uniform(0.5, 1.5, 128).astype(np.float32) for _ in range(2))
    max_len, pos0, slot0 = T + 9, 4, 2
    angle = rng.uniform(0, 6, (max_len, 64))
    cos, sin = (np.concatenate([f(angle), np.full_like(angle, np.nan)], 1).astype(np.float32) for f in (np.cos, np.sin))
    q, kc, _ = qkv_post(Q, qkv, qn, kn, cos, sin, B, T, H, G, max_len, pos0, slot0, 1e-6, off)
    x = qkv.astype(np.float64).transpose(0, 2, 1, 3)
    x = x / np.sqrt((x * x).mean(-1, keepdims=True) + 1e-6)
    c, s = (t[pos0:pos0 + T, :64].astype(np.float64) for t in (cos, sin))
    turned = lambda v: np.concatenate([v[..., :64] * c - v[..., 64:] * s, v[..., 64:] * c + v[..., :64] * s], -1)  # noqa: E731
    assert normwise(q, turned(x[:, :H] * qn)) < 1e-6
    assert normwise(kc[:, :, slot0:slot0 + T], turned(x[:, H:H + G] * kn)) < 1e-6


def test_full_model_32_sequences_match_reference(Q):
    """benchmark configuration 5 at batch 32: the operator path that 32 sequences take (tcgen05 linears on hi + lo bf16 planes
    with split-k pieces, attn_decode_fast_kernel, fused glue) against the reference run with 32 distinct prompts.
    The reference's prompt is 16 tokens per sequence (its prefill of 32 x 512 tokens would take most of an hour on the
    CPU); the 32 greedy decode steps are the full count. Tokens must be identical wherever the reference's own margin
    between its two best logits is above the fp32 noise of the comparison, and the logits of the reference's four
    best tokens must agree to 1e-3 at every step; the device is fed the reference's tokens, so that one near-tie
    cannot hide the steps after it."""
    from pathlib import Path
    g = np.load(Path(__file__).resolve().parent / "golden" / "golden_qwen3_b32.npz")
    cfg = Q.Qwen3Config(max_position_embeddings=64)
    w = Q.random_weights(cfg, seed=4)
    assert hashlib.sha256(w["embed"].tobytes()).hexdigest() == str(g["embed_sha256"])
    m = Q.Qwen3ForCausalLM(cfg, batch=32)
    m.load_weights(w)
    want_tok, margins, top_i, top_v = g["tokens"], g["margins"], g["top4_indices"], g["top4_values"]
    logits = m.forward(dev_ids(g["prompt"]))
    free_running_equal = True
    fed = None
    for s in range(32):
        tok, _ = m.argmax(logits)
        got_tok = tok.cpu().numpy()
        got = logits.cpu().numpy()
        picked = np.take_along_axis(got, top_i[:, s, :].astype(np.int64), axis=1)
        assert np.abs(picked - top_v[:, s, :]).max() < 1e-3, s
        clear = margins[:, s] > 2e-3
        assert np.array_equal(got_tok[clear], want_tok[clear, s]), (s, got_tok, want_tok[:, s])
        free_running_equal &= bool(np.array_equal(got_tok, want_tok[:, s]))
        if s < 31:
            fed = dev_ids(want_tok[:, s].reshape(32, 1))
            logits = m.forward(fed)
    assert (margins > 2e-3).mean() > 0.97  # the check above covered nearly every token
    assert free_running_equal or (margins <= 2e-3).any()
    m.close()


def test_long_prompts_of_wide_models(Q):
    """A hidden size above what the norm that writes planes takes: one prompt of 130 tokens, and the same in two parts."""
    cfg = Q.Qwen3Config(**{**SMALL, "hidden_size": 16392, "num_hidden_layers": 1, "vocab_size": 64, "num_attention_heads": 1,
                           "num_key_value_heads": 1, "max_position_embeddings": 256})
    m = Q.Qwen3ForCausalLM(cfg)
    m.load_weights(Q.random_weights(cfg, seed=3, std=0.01))
    ids = np.random.default_rng(1).integers(0, 64, (1, 130))
    m.forward(dev_ids(ids[:, :100]))
    want = m.forward(dev_ids(ids[:, 100:])).cpu().numpy()
    m.reset_kv_cache()
    assert normwise(m.forward(dev_ids(ids)).cpu().numpy(), want) < 1e-4
    m.close()


@pytest.mark.parametrize("inter,rows", [(2816, 1100), (2824, 1025), (4104, 600)])
def test_activation_in_the_products_epilogue(Q, inter, rows):
    """Prompts long enough for CTA pairs: swish(gate) * up and its planes come from the gate / up product itself, at FFN widths that
    end inside a tile of 128 outputs and rows that end inside one of 256. The same prompt in parts of 100 rows takes the other
    kernels; both keep two planes and fp32 sums."""
    cfg = Q.Qwen3Config(**{**SMALL, "hidden_size": 256, "intermediate_size": inter, "max_position_embeddings": 1200})
    m = Q.Qwen3ForCausalLM(cfg)
    m.load_weights(Q.random_weights(cfg, seed=3, std=0.05))
    ids = np.random.default_rng(1).integers(0, 512, (1, rows))
    for i in range(0, rows, 100):
        want = m.forward(dev_ids(ids[:, i:i + 100])).cpu().numpy()
    m.reset_kv_cache()
    assert normwise(m.forward(dev_ids(ids)).cpu().numpy(), want) < 2e-5
    m.close()


@pytest.mark.parametrize("hidden,rows", [(256, 300), (1024, 1100), (2048, 2400), (264, 131)])
def test_residual_stream_of_a_long_prompt_keeps_every_fp32_number(Q, hidden, rows):
    """Embeddings below 2^-126 through a layer whose o and down projections are zero: the stream stays what it was, whichever kernel adds
    to it in memory (k shared by a cluster, one CTA a tile, CTA pairs, columns that end inside a tile). The final norm, whose root is
    that of its eps, and an output matrix of its own show it: 2e-5, two bf16 planes."""
    cfg = Q.Qwen3Config(**{**SMALL, "hidden_size": hidden, "num_hidden_layers": 1, "intermediate_size": 512, "max_position_embeddings": 2400})
    w = Q.random_weights(cfg, seed=3, std=0.05)
    rng = np.random.default_rng(rows)
    w["lm_head"] = w["embed"]
    w["embed"] = Q.f32_to_bf16_bits((rng.uniform(0.25, 1, w["embed"].shape) * rng.choice([-1, 1], w["embed"].shape) * 2.0 ** -127).astype(np.float32)).reshape(w["embed"].shape)
    w["norm"] = np.full(hidden, 2.0 ** 100, np.float32)
    for name in ("o", "down"):
        w[(name, 0)] = np.zeros_like(w[(name, 0)])
    m = Q.Qwen3ForCausalLM(cfg)
    m.load_weights(w)
    ids = rng.integers(0, 512, (1, rows))
    got = m.forward(dev_ids(ids)).cpu().numpy()[0]
    x = Q.bf16_bits_to_f32(w["embed"])[ids[0, -1]].astype(np.float64) / np.sqrt(cfg.rms_norm_eps) * 2.0 ** 100
    assert normwise(got, Q.bf16_bits_to_f32(w["lm_head"]).astype(np.float64) @ x) < 2e-5
    m.close()


def test_long_prompts_of_an_odd_share_of_the_ffn(Q):
    """A rank whose share of the FFN has rows that do not start at 16 bytes (40 / 2 columns) computes what one GPU does with
    the same weights and columns of zeros behind them. The sums over the ranks are left out."""
    cfg = Q.Qwen3Config(**{**SMALL, "num_attention_heads": 2, "intermediate_size": 40, "max_position_embeddings": 256})
    w = Q.random_weights(cfg, seed=3, std=0.05)
    m = Q.Qwen3ForCausalLM(cfg, tp_rank=0, tp_world=2, connect_peers=False)
    m._cb = Q._ALLREDUCE_T(lambda buf, count, user: 0)
    assert m.L.ytcuda_qwen3_set_allreduce(m.h, Q.C.cast(m._cb, Q.C.c_void_p), None) == 0
    m.load_weights(w)
    one = Q.Qwen3Config(**{**SMALL, "num_attention_heads": 1, "num_key_value_heads": 1, "intermediate_size": 24,
                           "max_position_embeddings": 256})
    part = {}
    for key, x in w.items():
        name = key if isinstance(key, str) else key[0]
        x = Q.shard_weight(cfg, name, x, 0, 2)
        if name == "gate_up":
            x = np.concatenate([np.pad(x[:20], ((0, 4), (0, 0))), np.pad(x[20:], ((0, 4), (0, 0)))])
        part[key] = np.pad(x, ((0, 0), (0, 4))) if name == "down" else x
    n = Q.Qwen3ForCausalLM(one)
    n.load_weights(part)
    ids = np.random.default_rng(1).integers(0, 512, (1, 150))
    got, want = m.forward(dev_ids(ids)).cpu().numpy(), n.forward(dev_ids(ids)).cpu().numpy()
    assert normwise(got, want[:, :256]) < 1e-4
    m.close()
    n.close()
