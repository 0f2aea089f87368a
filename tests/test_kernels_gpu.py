"""CUDA kernels vs the fp32 PyTorch reference of the same op (run on a B200)."""
import math

import pytest
import torch

from vllm_metax_b200 import _custom_ops as ops
from vllm_metax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def cos_diff(a, b):
    a, b = a.float().flatten(), b.float().flatten()
    return 1.0 - float(torch.dot(a, b) / (a.norm() * b.norm() + 1e-12))


@pytest.fixture(autouse=True)
def _status(kernel_status_ok):
    yield


# ------------------------------------------------------------------ GEMM
@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (1000, 1536, 4096), (4096, 6144, 4096),
                                   (333, 264, 520), (129, 4096, 14336)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gemm_tcgen05(M, N, K, dtype):
    a = torch.randn(M, K, device=DEV, dtype=dtype)
    w = torch.randn(N, K, device=DEV, dtype=dtype) * 0.05
    want = (a.float() @ w.float().t())
    got = ops.gemm(a, w)
    torch.cuda.synchronize()
    assert got.shape == (M, N)
    err = (got.float() - want).abs().max() / want.abs().max()
    assert err < 1.5e-2, err
    assert cos_diff(got, want) < 1e-5


@pytest.mark.parametrize("force_bn", [256, 128, 64, 32, -16, -32, -64])
def test_gemm_every_tile_config(force_bn):
    M = 48 if force_bn < 0 else 300
    N, K = 1280, 1024
    a = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(N, K, device=DEV, dtype=torch.bfloat16) * 0.05
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    res = torch.randn(M, N, device=DEV, dtype=torch.bfloat16)
    want = a.float() @ w.float().t() + bias.float() + res.float()
    got = ops.gemm(a, w, bias, res, force_bn=force_bn)
    assert (got.float() - want).abs().max() / want.abs().max() < 1.5e-2


@pytest.mark.parametrize("M", [1, 7, 16, 33, 64])
def test_gemm_small_m_swap(M):
    a = torch.randn(M, 4096, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(6144, 4096, device=DEV, dtype=torch.bfloat16) * 0.05
    want = a.float() @ w.float().t()
    got = ops.gemm(a, w)
    assert (got.float() - want).abs().max() / want.abs().max() < 1.5e-2


def test_gemm_strided_input_view():
    big = torch.randn(200, 3 * 512, device=DEV, dtype=torch.bfloat16)
    a = big[:, 512:1024]
    w = torch.randn(384, 512, device=DEV, dtype=torch.bfloat16) * 0.05
    want = a.float() @ w.float().t()
    assert (ops.gemm(a, w).float() - want).abs().max() / want.abs().max() < 1.5e-2


# ------------------------------------------------------------------ norms
@pytest.mark.parametrize("T,H", [(1, 256), (7, 4096), (300, 8192), (5, 7168), (3, 520)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_rms_norm(T, H, dtype):
    x = torch.randn(T, H, device=DEV, dtype=dtype)
    w = torch.randn(H, device=DEV, dtype=dtype)
    torch.testing.assert_close(ops.rms_norm(x, w, 1e-5), ref.rms_norm(x, w, 1e-5), rtol=2e-2, atol=2e-2)
    r = torch.randn(T, H, device=DEV, dtype=dtype)
    wy, wr = ref.fused_add_rms_norm(x, r, w, 1e-5)
    x2, r2 = x.clone(), r.clone()
    ops.fused_add_rms_norm(x2, r2, w, 1e-5)
    torch.testing.assert_close(r2, wr, rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(x2, wy, rtol=2e-2, atol=2e-2)


def test_head_rms_norm():
    T, H, D = 9, 6, 128
    x = torch.randn(T, H * D + 256, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(D, device=DEV, dtype=torch.bfloat16)
    want = ref.rms_norm(x[:, : H * D].reshape(T, H, D), w, 1e-6).reshape(T, -1)
    tail = x[:, H * D:].clone()
    ops.head_rms_norm(x, w, 1e-6, H, D)
    torch.testing.assert_close(x[:, : H * D], want, rtol=2e-2, atol=2e-2)
    assert torch.equal(x[:, H * D:], tail)


@pytest.mark.parametrize("with_res", [False, True])
def test_rms_norm_quant_variants(with_res):
    T, H = 11, 2048
    x = torch.randn(T, H, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(H, device=DEV, dtype=torch.bfloat16)
    res = torch.randn(T, H, device=DEV, dtype=torch.bfloat16) if with_res else None
    # per-token fp8
    q, s = ops.rms_norm_dynamic_per_token_quant(x, w, 1e-5, residual=None if res is None else res.clone())
    wq, ws, _ = ref.rms_norm_dynamic_per_token_quant(x, w, 1e-5, residual=res)
    torch.testing.assert_close(s, ws, rtol=2e-2, atol=1e-6)
    assert cos_diff(q.float() * s, wq.float() * ws) < 1e-3
    # per-token int8
    q, s = ops.rms_norm_dynamic_per_token_quant(x, w, 1e-5, torch.int8, residual=None if res is None else res.clone())
    wq, ws, _ = ref.rms_norm_dynamic_per_token_quant(x, w, 1e-5, torch.int8, residual=res)
    assert cos_diff(q.float() * s, wq.float() * ws) < 1e-3
    # per-128 block fp8
    q, s = ops.rms_norm_per_block_quant(x, w, 1e-5, 128, residual=None if res is None else res.clone())
    wq, ws, _ = ref.rms_norm_per_block_quant(x, w, 1e-5, 128, residual=res)
    torch.testing.assert_close(s, ws, rtol=2e-2, atol=1e-6)
    deq = (q.float().reshape(T, -1, 128) * s[..., None]).reshape(T, H)
    wdeq = (wq.float().reshape(T, -1, 128) * ws[..., None]).reshape(T, H)
    assert cos_diff(deq, wdeq) < 1e-3
    # static fp8
    sc = torch.tensor([0.02], device=DEV)
    q = ops.rms_norm_static_fp8_quant(x, w, sc, 1e-5)
    assert cos_diff(q.float(), ref.rms_norm_static_fp8_quant(x, w, sc, 1e-5).float()) < 1e-3


# ------------------------------------------------------------------ activations
@pytest.mark.parametrize("act", ["silu", "gelu", "gelu_tanh", "relu2", "mul_silu", "swigluoai", "swiglustep"])
def test_act_and_mul(act):
    x = torch.randn(13, 2 * 1536, device=DEV, dtype=torch.bfloat16)
    got = ops.act_and_mul(x, act)
    want = ops.act_and_mul(x.cpu(), act).to(DEV)
    torch.testing.assert_close(got, want, rtol=2e-2, atol=2e-2)


def test_silu_mul_block_quant():
    x = torch.randn(10, 2 * 1024, device=DEV, dtype=torch.bfloat16)
    q, s = ops.silu_and_mul_per_block_quant(x, 128)
    wq, ws = ref.silu_and_mul_per_block_quant(x, 128)
    torch.testing.assert_close(s, ws, rtol=2e-2, atol=1e-7)
    a = (q.float().reshape(10, -1, 128) * s[..., None])
    b = (wq.float().reshape(10, -1, 128) * ws[..., None])
    assert cos_diff(a, b) < 1e-3


# ------------------------------------------------------------------ rope + cache
@pytest.mark.parametrize("neox", [True, False])
@pytest.mark.parametrize("D,rot", [(128, 128), (64, 64), (128, 64), (256, 128)])
def test_rotary_embedding(neox, D, rot):
    T, Hq, Hk = 17, 8, 2
    q = torch.randn(T, Hq * D, device=DEV, dtype=torch.bfloat16)
    k = torch.randn(T, Hk * D, device=DEV, dtype=torch.bfloat16)
    pos = torch.randint(0, 500, (T,), device=DEV)
    cache = ref.build_rope_cache(rot, 512, 10000.0).to(DEV)
    wq, wk = ref.rotary_embedding(pos, q, k, D, cache, neox)
    ops.rotary_embedding(pos, q, k, D, cache, neox)
    torch.testing.assert_close(q, wq, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(k, wk, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("kind", ["bf16", "fp8_static", "int8_per_token_head", "fp8_per_token_head"])
def test_rope_and_cache_write(kind):
    T, Hq, Hk, D, bs, nb = 40, 8, 2, 128, 16, 12
    qkv = torch.randn(T, (Hq + 2 * Hk) * D, device=DEV, dtype=torch.bfloat16)
    q, k, v = qkv[:, : Hq * D], qkv[:, Hq * D:(Hq + Hk) * D], qkv[:, (Hq + Hk) * D:]
    pos = torch.arange(T, device=DEV)
    slots = torch.randperm(nb * bs, device=DEV)[:T]
    slots[3] = -1
    cos_sin = ref.build_rope_cache(D, 64, 10000.0).to(DEV)
    dt = {"bf16": torch.bfloat16, "fp8_static": torch.float8_e4m3fn, "int8_per_token_head": torch.int8,
          "fp8_per_token_head": torch.float8_e4m3fn}[kind]
    cache = torch.zeros(nb, 2, bs, Hk, D, device=DEV, dtype=dt)
    scales = torch.ones(nb, 2, bs, Hk, device=DEV) if kind.endswith("head") else None
    wcache, wscales = cache.clone(), None if scales is None else scales.clone()
    wq, wk = ref.rotary_embedding(pos, q.contiguous(), k.contiguous(), D, cos_sin, True)
    ref.reshape_and_cache(wk.reshape(T, Hk, D), v.reshape(T, Hk, D), wcache, slots, wscales, 0.05, 0.07)
    ops.rope_and_cache(pos, q, k, v, D, cos_sin, True, cache, slots, scales, 0.05, 0.07)
    torch.testing.assert_close(q, wq, rtol=2e-2, atol=2e-2)
    if scales is not None:
        torch.testing.assert_close(scales, wscales, rtol=1e-2, atol=1e-6)
        assert cos_diff(cache.float() * scales[..., None], wcache.float() * wscales[..., None]) < 2e-3
    else:
        assert cos_diff(cache.float(), wcache.float()) < 2e-3


def test_concat_and_cache_mla_both_formats():
    T, bs, nb = 19, 64, 4
    kv_c = torch.randn(T, 512, device=DEV, dtype=torch.bfloat16)
    k_pe = torch.randn(T, 64, device=DEV, dtype=torch.bfloat16)
    slots = torch.randperm(nb * bs, device=DEV)[:T]
    c = torch.zeros(nb, bs, 576, device=DEV, dtype=torch.bfloat16)
    wc = c.clone()
    ops.concat_and_cache_mla(kv_c, k_pe, c, slots)
    ref.concat_and_cache_mla(kv_c, k_pe, wc, slots)
    assert torch.equal(c, wc)
    c8 = torch.zeros(nb, bs, 656, device=DEV, dtype=torch.uint8)
    w8 = c8.clone()
    ops.concat_and_cache_mla(kv_c, k_pe, c8, slots)
    ref.concat_and_cache_mla(kv_c, k_pe, w8, slots)
    a, b = ref.unpack_ds_mla(c8.reshape(-1, 656)), ref.unpack_ds_mla(w8.reshape(-1, 656))
    assert cos_diff(a, b) < 1e-4
    assert torch.equal(c8[..., 528:], w8[..., 528:])


def test_indexer_k_quant_and_cache():
    T, bs, nb = 33, 64, 3
    k = torch.randn(T, 128, device=DEV, dtype=torch.bfloat16)
    slots = torch.randperm(nb * bs, device=DEV)[:T]
    c = torch.zeros(nb, bs * 132, device=DEV, dtype=torch.uint8)
    w = c.clone()
    ops.indexer_k_quant_and_cache(k, c, slots, bs)
    ref.indexer_k_quant_and_cache(k, w, slots)
    bt = torch.arange(nb, device=DEV, dtype=torch.int32)
    kq, sc = ref.gather_indexer_k(c, bt, nb * bs)
    wq, wsc = ref.gather_indexer_k(w, bt, nb * bs)
    torch.testing.assert_close(sc, wsc, rtol=1e-3, atol=1e-8)
    assert cos_diff(kq * sc[:, None], wq * wsc[:, None]) < 1e-4


def test_copy_blocks():
    c = torch.randn(10, 2, 16, 2, 64, device=DEV, dtype=torch.bfloat16)
    w = c.clone()
    pairs = torch.tensor([[0, 5], [1, 7], [2, 9]], device=DEV)
    ops.copy_blocks([c], pairs)
    ref.copy_blocks([w], pairs)
    assert torch.equal(c, w)


# ------------------------------------------------------------------ attention
def make_paged(B, lens, Hkv, D, bs, dtype, kind="same", extra_blocks=3):
    """Random paged cache + block tables for sequences of the given kv lengths."""
    nblk = [(l + bs - 1) // bs for l in lens]
    total = sum(nblk) + extra_blocks
    perm = torch.randperm(total)
    bt = torch.zeros(B, max(nblk), dtype=torch.int32)
    o = 0
    for b in range(B):
        bt[b, : nblk[b]] = perm[o:o + nblk[b]].to(torch.int32)
        o += nblk[b]
    kv = torch.randn(total, 2, bs, Hkv, D)
    scales = None
    if kind == "same":
        cache = kv.to(dtype)
    elif kind == "int8":
        sc = kv.abs().amax(-1) / 127.0
        cache = torch.round(kv / sc[..., None]).clamp(-128, 127).to(torch.int8)
        scales = sc.float()
    elif kind == "fp8":
        sc = kv.abs().amax(-1) / 448.0
        cache = (kv / sc[..., None]).to(torch.float8_e4m3fn)
        scales = sc.float()
    return cache.to(DEV), (None if scales is None else scales.to(DEV)), bt.to(DEV)


@pytest.mark.parametrize("Hq,Hkv,D", [(32, 8, 128), (8, 8, 64), (16, 2, 128), (4, 1, 256)])
@pytest.mark.parametrize("bs", [16, 64])
@pytest.mark.parametrize("splits", [1, 4])
def test_paged_decode(Hq, Hkv, D, bs, splits):
    lens = [1, 17, 300, 1025, 64]
    B = len(lens)
    cache, _, bt = make_paged(B, lens, Hkv, D, bs, torch.bfloat16)
    q = torch.randn(B, Hq, D, device=DEV, dtype=torch.bfloat16)
    sl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    scale = D ** -0.5
    got = ops.paged_attention_decode(q, cache, bt, sl, scale, num_splits=splits)
    qsl = torch.arange(B + 1, dtype=torch.int32, device=DEV)
    want = ref.paged_attention(q, cache, bt, sl, qsl, scale)
    assert cos_diff(got, want) < 2e-4
    torch.testing.assert_close(got.float(), want.float(), rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("kind", ["int8", "fp8"])
def test_paged_decode_quantised_kv(kind):
    Hq, Hkv, D, bs = 32, 8, 128, 16
    lens = [5, 130, 777]
    cache, scales, bt = make_paged(3, lens, Hkv, D, bs, torch.bfloat16, kind)
    q = torch.randn(3, Hq, D, device=DEV, dtype=torch.bfloat16)
    sl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    got = ops.paged_attention_decode(q, cache, bt, sl, D ** -0.5, kv_scales=scales, num_splits=2)
    want = ref.paged_attention(q, cache, bt, sl, torch.arange(4, dtype=torch.int32, device=DEV), D ** -0.5,
                               kv_scales=scales)
    assert cos_diff(got, want) < 5e-4


def test_paged_decode_window_softcap_sinks_multitoken():
    Hq, Hkv, D, bs = 8, 2, 128, 16
    lens = [40, 200]
    qlens = [3, 2]
    cache, _, bt = make_paged(2, lens, Hkv, D, bs, torch.bfloat16)
    T = sum(qlens)
    q = torch.randn(T, Hq, D, device=DEV, dtype=torch.bfloat16)
    sl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    qsl = torch.tensor([0, 3, 5], dtype=torch.int32, device=DEV)
    sinks = torch.randn(Hq, device=DEV)
    lse = torch.empty(Hq, T, device=DEV)
    got = ops.paged_attention_decode(q, cache, bt, sl, D ** -0.5, query_start_loc=qsl, max_q_len=3, window=64,
                                     softcap=30.0, sinks=sinks, lse_out=lse, num_splits=1)
    want = ref.paged_attention(q, cache, bt, sl, qsl, D ** -0.5, window=64, softcap=30.0, sinks=sinks)
    assert cos_diff(got, want) < 3e-4


@pytest.mark.parametrize("Hq,Hkv,D", [(32, 8, 128), (4, 4, 64), (28, 4, 128)])
@pytest.mark.parametrize("bs", [16, 64, 128])
def test_prefill_tcgen05_paged(Hq, Hkv, D, bs):
    # (q_len, kv_len): pure prefill, chunked prefill with context, short and ragged cases
    cases = [(200, 200), (64, 300), (1, 1), (129, 129), (257, 1000)]
    lens = [c[1] for c in cases]
    B = len(cases)
    cache, _, bt = make_paged(B, lens, Hkv, D, bs, torch.bfloat16)
    T = sum(c[0] for c in cases)
    q = torch.randn(T, Hq, D, device=DEV, dtype=torch.bfloat16)
    qsl = torch.tensor([0] + list(torch.tensor([c[0] for c in cases]).cumsum(0)), dtype=torch.int32, device=DEV)
    sl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    lse = torch.empty(Hq, T, device=DEV)
    got = ops.paged_attention_prefill(q, cache, bt, sl, qsl, D ** -0.5, max_q_len=257, lse_out=lse)
    want, wlse = ref.paged_attention(q, cache, bt, sl, qsl, D ** -0.5, return_lse=True)
    assert cos_diff(got, want) < 3e-4
    torch.testing.assert_close(got.float(), want.float(), rtol=4e-2, atol=4e-2)
    torch.testing.assert_close(lse, wlse, rtol=2e-2, atol=2e-2)


def test_prefill_window_softcap_sinks():
    Hq, Hkv, D, bs = 8, 2, 128, 64
    cases = [(300, 300), (100, 400)]
    lens = [c[1] for c in cases]
    cache, _, bt = make_paged(2, lens, Hkv, D, bs, torch.bfloat16)
    q = torch.randn(400, Hq, D, device=DEV, dtype=torch.bfloat16)
    qsl = torch.tensor([0, 300, 400], dtype=torch.int32, device=DEV)
    sl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    sinks = torch.randn(Hq, device=DEV)
    got = ops.paged_attention_prefill(q, cache, bt, sl, qsl, D ** -0.5, max_q_len=300, window=128, softcap=50.0,
                                      sinks=sinks)
    want = ref.paged_attention(q, cache, bt, sl, qsl, D ** -0.5, window=128, softcap=50.0, sinks=sinks)
    assert cos_diff(got, want) < 3e-4


def test_prefill_quantised_cache_falls_to_split_kernel():
    Hq, Hkv, D, bs = 16, 4, 128, 16
    cases = [(50, 50), (20, 90)]
    lens = [c[1] for c in cases]
    cache, scales, bt = make_paged(2, lens, Hkv, D, bs, torch.bfloat16, "int8")
    q = torch.randn(70, Hq, D, device=DEV, dtype=torch.bfloat16)
    qsl = torch.tensor([0, 50, 70], dtype=torch.int32, device=DEV)
    sl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    got = ops.paged_attention_prefill(q, cache, bt, sl, qsl, D ** -0.5, kv_scales=scales, max_q_len=50)
    want = ref.paged_attention(q, cache, bt, sl, qsl, D ** -0.5, kv_scales=scales)
    assert cos_diff(got, want) < 5e-4


@pytest.mark.parametrize("dqk,dv", [(128, 128), (192, 128)])
def test_varlen_attention_contiguous(dqk, dv):
    H = 16
    lq, lk = [100, 37, 256], [100, 200, 256]
    q = torch.randn(sum(lq), H, dqk, device=DEV, dtype=torch.bfloat16)
    k = torch.randn(sum(lk), H, dqk, device=DEV, dtype=torch.bfloat16)
    v = torch.randn(sum(lk), H, dv, device=DEV, dtype=torch.bfloat16)
    cq = torch.tensor([0, 100, 137, 393], dtype=torch.int32, device=DEV)
    ck = torch.tensor([0, 100, 300, 556], dtype=torch.int32, device=DEV)
    got = ops.varlen_attention(q, k, v, cq, ck, dqk ** -0.5, max_q_len=256)
    want = ops.varlen_attention(q.cpu(), k.cpu(), v.cpu(), cq.cpu(), ck.cpu(), dqk ** -0.5).to(DEV)
    assert cos_diff(got, want) < 3e-4


# ------------------------------------------------------------------ sampling
def test_argmax_and_greedy_sample():
    logits = torch.randn(37, 128256, device=DEV, dtype=torch.bfloat16)
    assert torch.equal(ops.argmax(logits), logits.float().argmax(-1))
    t = torch.zeros(37, device=DEV)
    u = torch.rand(37, device=DEV)
    assert torch.equal(ops.sample(logits, t, None, None, None, u), logits.float().argmax(-1))


def _topk_then_topp_keep(probs, k, p):
    """Upstream's order: top-k, renormalise over the kept tokens, then top-p.  Returns (sorted ids, keep mask by rank,
    renormalised probabilities by rank)."""
    sp, si = probs.sort(-1, descending=True)
    V = probs.shape[-1]
    in_k = torch.arange(V, device=probs.device)[None] < k
    pk = torch.where(in_k, sp, torch.zeros_like(sp))
    pk = pk / pk.sum(-1, keepdim=True)
    keep = in_k & ((pk.cumsum(-1) - pk) < p)
    final = torch.where(keep, pk, torch.zeros_like(pk))
    return si, keep, final / final.sum(-1, keepdim=True)


def test_sample_respects_topk_topp():
    V = 5000
    logits = torch.randn(64, V, device=DEV)
    temp = torch.full((64,), 0.8, device=DEV)
    top_k = torch.full((64,), 50, device=DEV, dtype=torch.int32)
    top_p = torch.full((64,), 0.9, device=DEV)
    si, keep, _ = _topk_then_topp_keep(torch.softmax(logits / 0.8, -1), 50, 0.9)
    for trial in range(8):
        u = torch.rand(64, device=DEV)
        tok = ops.sample(logits, temp, top_k, top_p, None, u)
        rank = (si == tok[:, None]).float().argmax(-1)
        assert bool(keep.gather(1, rank[:, None]).all())


def test_sample_topk_then_topp_distribution():
    """With both cuts active the kept set is the one of the sort-based oracle (top-p over the renormalised top-k
    distribution), and tokens are drawn in proportion inside it."""
    V, n = 64, 16384
    row = torch.randn(1, V, device=DEV)
    logits = row.repeat(n, 1)
    temp = torch.ones(n, device=DEV)
    si, keep, final = _topk_then_topp_keep(torch.softmax(row, -1), 16, 0.8)
    tok = ops.sample(logits, temp, torch.full((n,), 16, device=DEV, dtype=torch.int32),
                     torch.full((n,), 0.8, device=DEV), None, torch.rand(n, device=DEV))
    emp = torch.bincount(tok, minlength=V).float() / n
    want = torch.zeros(V, device=DEV)
    want[si[0]] = final[0]
    assert float(emp[want == 0].sum()) == 0.0
    assert (emp - want).abs().max() < 0.03


def test_sample_distribution_matches():
    V = 50
    logits = torch.randn(1, V, device=DEV).repeat(4096, 1)
    temp = torch.ones(4096, device=DEV)
    u = torch.rand(4096, device=DEV)
    tok = ops.sample(logits, temp, None, None, None, u)
    emp = torch.bincount(tok, minlength=V).float() / 4096
    assert (emp - torch.softmax(logits[0], -1)).abs().max() < 0.04


def test_penalties_and_advance_and_embedding():
    B, V = 5, 1000
    logits = torch.randn(B, V, device=DEV)
    counts = torch.randint(0, 3, (B, V), device=DEV, dtype=torch.int32)
    pm = torch.randint(0, 2, (B, V), device=DEV, dtype=torch.int32)
    rep = torch.full((B,), 1.3, device=DEV)
    pres = torch.full((B,), 0.2, device=DEV)
    freq = torch.full((B,), 0.1, device=DEV)
    want = ops.apply_penalties(logits.cpu().clone(), pm.cpu(), counts.cpu(), rep.cpu(), pres.cpu(), freq.cpu())
    got = ops.apply_penalties(logits.clone(), pm, counts, rep, pres, freq)
    torch.testing.assert_close(got.cpu(), want, rtol=1e-5, atol=1e-5)
    table = torch.randn(300, 256, device=DEV, dtype=torch.bfloat16)
    ids = torch.randint(0, 300, (40,), device=DEV)
    assert torch.equal(ops.embedding(table, ids), table[ids])
    # advance
    bs, MB = 16, 8
    bt = torch.randint(0, 100, (B, MB), device=DEV, dtype=torch.int32)
    pos = torch.tensor([0, 15, 16, 31, 100], device=DEV)
    ids2 = torch.zeros(B, dtype=torch.int64, device=DEV)
    sl = (pos + 1).to(torch.int32)
    slots = torch.zeros(B, dtype=torch.int64, device=DEV)
    sampled = torch.arange(B, device=DEV) + 7
    ops.advance_step(ids2, pos, sl, slots, sampled, bt, bs, B)
    assert torch.equal(ids2, sampled)
    assert pos.tolist() == [1, 16, 17, 32, 101]
    assert sl.tolist() == [2, 17, 18, 33, 102]
    exp = [int(bt[i, p // bs]) * bs + p % bs for i, p in enumerate([1, 16, 17, 32, 101])]
    assert slots.tolist() == exp


@pytest.mark.parametrize("M", [5, 48, 256, 1000])
def test_gemm_fused_silu_gate_epilogue(M):
    K, I = 1024, 1408
    a = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(2 * I, K, device=DEV, dtype=torch.bfloat16) * 0.05
    got = ops.gemm_silu_mul(a, w)
    want = ops.gemm_silu_mul(a.cpu(), w.cpu()).to(DEV)
    assert got.shape == (M, I)
    assert cos_diff(got, want) < 1e-4
    torch.testing.assert_close(got.float(), want.float(), rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("M,N,K", [(512, 512, 256), (1024, 1536, 4096), (1000, 1288, 520), (8192, 6144, 4096)])
def test_gemm_cta_pair(M, N, K):
    a = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(N, K, device=DEV, dtype=torch.bfloat16) * 0.05
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    res = torch.randn(M, N, device=DEV, dtype=torch.bfloat16)
    want = a.float() @ w.float().t() + bias.float() + res.float()
    got = ops.gemm(a, w, bias, res, force_bn=512)
    assert (got.float() - want).abs().max() / want.abs().max() < 1.5e-2
    assert cos_diff(got, want) < 1e-5


@pytest.mark.parametrize("D", [64, 128])
def test_alibi_bias_in_prefill_and_decode(D):
    """ALiBi slopes: score += slope[h] * (kv position - query position), both attention kernels."""
    torch.manual_seed(9)
    Hq, Hkv, bs = 8, 2, 16
    lens, qlens = [70, 33, 130], [70, 1, 17]          # fresh prefill, decode, chunked prefill
    B = len(lens)
    nblk = [(l + bs - 1) // bs for l in lens]
    bt = torch.zeros(B, max(nblk), dtype=torch.int32)
    perm = torch.randperm(sum(nblk) + 1)
    o = 0
    for b in range(B):
        bt[b, : nblk[b]] = perm[o:o + nblk[b]].int()
        o += nblk[b]
    cache = torch.randn(sum(nblk) + 1, 2, bs, Hkv, D).bfloat16()
    q = torch.randn(sum(qlens), Hq, D).bfloat16()
    slopes = torch.tensor([2.0 ** (-(i + 1)) for i in range(Hq)])
    sl = torch.tensor(lens, dtype=torch.int32)
    qsl = torch.tensor([0] + list(torch.tensor(qlens).cumsum(0)), dtype=torch.int32)
    want = ref.paged_attention(q.float(), cache.float(), bt, sl, qsl, D ** -0.5, alibi_slopes=slopes)
    plain = ref.paged_attention(q.float(), cache.float(), bt, sl, qsl, D ** -0.5)
    assert (want - plain).abs().max() > 1e-2          # the bias matters in this case
    got_p = ops.paged_attention_prefill(q.cuda(), cache.cuda(), bt.cuda(), sl.cuda(), qsl.cuda(), D ** -0.5,
                                        max_q_len=max(qlens), alibi_slopes=slopes.cuda())
    torch.testing.assert_close(got_p.float().cpu(), want, rtol=3e-2, atol=3e-2)
    got_d = ops.paged_attention_decode(q.cuda(), cache.cuda(), bt.cuda(), sl.cuda(), D ** -0.5, query_start_loc=qsl.cuda(),
                                       max_q_len=max(qlens), max_seq_len=max(lens), alibi_slopes=slopes.cuda())
    torch.testing.assert_close(got_d.float().cpu(), want, rtol=3e-2, atol=3e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[1], [900], [0, 1, 64, 65, 0, 3], [17] * 300, [5000, 3, 129, 1, 700, 64], [2048 - 13 * i for i in range(48)]])
@pytest.mark.parametrize("Hq,Hkv,D,kind", [(32, 8, 128, 0), (64, 8, 128, 1), (16, 2, 256, 0), (24, 2, 128, 0), (32, 2, 128, 1), (6, 6, 64, 0),
                                           (5, 1, 80, 0)])
def test_decode_shared_out_evenly(lens, Hq, Hkv, D, kind, kernel_status_ok):
    """One token per sequence: ranges that end inside sequences and hold many, sequences cut into many parts, empty ones, fewer
    units than CTAs, windows, sinks, capped scores; 16-bit and int8 caches, 8 and 16 rows of heads, padded head sizes; a scratch
    that is kept, whose counters are zero again after each call."""
    g = torch.Generator().manual_seed(len(lens) + D)
    bs, B = 64, len(lens)
    nb = [-(-n // bs) for n in lens]
    table = torch.zeros(B, max(nb) + 1, dtype=torch.int32)
    perm, at = torch.randperm(sum(nb) + 1, generator=g), 0
    for i, n in enumerate(nb):
        table[i, :n] = perm[at: at + n]
        at += n
    q = torch.randn(B, Hq, D, generator=g).bfloat16()
    sl = torch.tensor(lens, dtype=torch.int32)
    scales = None
    if kind:
        cache = torch.randint(-127, 128, (sum(nb) + 1, 2, bs, Hkv, D), generator=g, dtype=torch.int8)
        scales = torch.rand(sum(nb) + 1, 2, bs, Hkv, generator=g) * 0.012 + 0.004
        deq = cache.float() * scales[..., None]
    else:
        cache = torch.randn(sum(nb) + 1, 2, bs, Hkv, D, generator=g).bfloat16()
        deq = cache.float()
    sinks = torch.randn(Hq, generator=g)
    scratch = ops.decode_scratch(Hq, Hkv, D, "cuda")
    for kw in (dict(), dict(window=100, softcap=20.0), dict(sinks=sinks), dict(scratch=scratch), dict(scratch=scratch, window=70)):
        lse = None if kw.get("sinks") is not None else torch.empty(Hq, B, device="cuda")
        kc = {k: v.cuda() if torch.is_tensor(v) else v for k, v in kw.items()}
        got = ops.paged_attention_decode(q.cuda(), cache.cuda(), table.cuda(), sl.cuda(), D ** -0.5, kv_scales=None if scales is None else scales.cuda(),
                                         lse_out=lse, max_seq_len=max(lens), **kc).float().cpu()
        assert not bool(scratch[:16384].any())
        for i, n in enumerate(lens):
            if n == 0:
                assert float(got[i].abs().max()) == 0.0
                continue
            rows = deq[table[i, : nb[i]].long()]
            k, v = (rows[:, j].reshape(-1, Hkv, D)[:n].repeat_interleave(Hq // Hkv, 1) for j in (0, 1))
            s = torch.einsum("hd,nhd->hn", q[i].float(), k) * D ** -0.5
            if kw.get("softcap"):
                s = kw["softcap"] * torch.tanh(s / kw["softcap"])
            if kw.get("window"):
                s[:, : max(0, n - kw["window"])] = float("-inf")
            full = torch.cat([s, sinks[:, None]], 1) if kw.get("sinks") is not None else s
            p = full.softmax(-1)[:, :n]
            want = torch.einsum("hn,nhd->hd", p, v)
            # weights are rounded to bf16 (2^-9 each, at random signs), the result once more
            bound = 2.0 ** -8 * want.abs() + 2.0 ** -8 * torch.einsum("hn,nhd->hd", p, v.abs())
            assert bool(((got[i] - want).abs() <= bound + 1e-5).all()), (i, n, float((got[i] - want).abs().max()))
            if lse is not None:
                torch.testing.assert_close(lse[:, i].cpu(), full.logsumexp(-1), rtol=1e-4, atol=2e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("bs", [16, 64, 128])
@pytest.mark.parametrize("Hq,Hkv", [(16, 2), (6, 2)])
@pytest.mark.parametrize("kw", [dict(), dict(window=70), dict(softcap=15.0), dict(causal=False)])
def test_prefill_of_256_wide_heads(bs, Hq, Hkv, kw, kernel_status_ok):
    """The one-tile tcgen05 kernel on paged 256-wide heads, portions behind context and without, lengths around its tiles (16
    tokens of 8 heads or 128 of one, 64 keys), against the decode kernel's 16-row tiles on the same cache."""
    g = torch.Generator().manual_seed(bs + Hq)
    qlens, past = [1, 15, 16, 129, 63, 200], [0, 64, 3, 0, 129, 1]
    lens = [a + b for a, b in zip(qlens, past)]
    nb = [-(-n // bs) for n in lens]
    table, perm, at = torch.zeros(len(lens), max(nb), dtype=torch.int32), torch.randperm(sum(nb), generator=g), 0
    for i, n in enumerate(nb):
        table[i, :n] = perm[at: at + n]
        at += n
    q = torch.randn(sum(qlens), Hq, 256, generator=g).bfloat16().cuda()
    cache = torch.randn(sum(nb), 2, bs, Hkv, 256, generator=g).bfloat16().cuda()
    qsl = torch.tensor([0] + list(torch.tensor(qlens).cumsum(0)), dtype=torch.int32).cuda()
    sl = torch.tensor(lens, dtype=torch.int32).cuda()
    l1, l2 = (torch.empty(Hq, q.shape[0], device="cuda") for _ in range(2))
    args, sizes = (q, cache, table.cuda(), sl), dict(max_q_len=max(qlens), max_seq_len=max(lens))
    got = ops.paged_attention_prefill(*args, qsl, 256 ** -0.5, **sizes, **kw)
    want = ops.paged_attention_decode(*args, 256 ** -0.5, query_start_loc=qsl, lse_out=l2, **sizes, **kw)
    # both round weights to bf16 (2^-9 of each, weights of 1 / n random values of size 1) and the result (2^-9)
    torch.testing.assert_close(got.float(), want.float(), rtol=2.0 ** -6, atol=2.0 ** -6)
    # with the log-sum-exp: the decode kernel itself
    assert torch.equal(ops.paged_attention_prefill(*args, qsl, 256 ** -0.5, lse_out=l1, **sizes, **kw), want) and torch.equal(l1, l2)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K", [(640, 2048), (6144, 4096), (1000, 1000), (1008, 1000), (28672, 512), (576, 14336)])
def test_few_tokens_against_a_weight(dtype, M, N, K, kernel_status_ok):
    """Rows that do not fill a CTA's eight, a contraction that ends inside a warp's piece, bias, residual and gated rows: sums of
    products exact in fp32, rounded once (gated: the two factors first)."""
    g = torch.Generator().manual_seed(N + M)
    a = torch.randn(M, K, generator=g).to(dtype).cuda()
    w = (torch.randn(N, K, generator=g) / K ** 0.5).to(dtype).cuda()
    b = torch.randn(N, generator=g).to(dtype).cuda()
    r = torch.randn(M, N, generator=g).to(dtype).cuda()
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    want = a.double() @ w.double().T
    torch.testing.assert_close(ops.gemm(a, w).double(), want, rtol=eps, atol=1e-5)
    torch.testing.assert_close(ops.gemm(a, w, bias=b, residual=r).double(), want + b.double() + r.double(), rtol=eps, atol=1e-5)
    if N % 16 == 0:
        f = lambda x: x.to(dtype).double()
        gate, up = f(want[:, 0::2]), f(want[:, 1::2])
        got = ops.gemm_silu_mul(a, w).double()
        # either factor may be the neighbouring number of its type, then one rounding
        torch.testing.assert_close(got, torch.nn.functional.silu(gate) * up, rtol=5 * eps, atol=1e-4)


def _decode_case(Hq, Hkv, dqk, dv, lens, dtype, int8=False, bs=64, seed=0):
    """Queries of one token per sequence, a shuffled cache (16 bits: pages for ``_decode_views``), and the result in fp32 from the
    cache's numbers with a bound."""
    g = torch.Generator().manual_seed(seed + Hq * dqk)
    nb = [-(-n // bs) for n in lens]
    table, perm, at = torch.zeros(len(lens), max(nb) + 1, dtype=torch.int32), torch.randperm(sum(nb) + 1, generator=g), 0
    for i, n in enumerate(nb):
        table[i, :n] = perm[at: at + n]
        at += n
    q = torch.randn(len(lens), Hq, dqk, generator=g).to(dtype)
    scales = None
    if int8:
        kv = torch.randint(-127, 128, (sum(nb) + 1, 2, bs, Hkv, dqk), generator=g, dtype=torch.int8)
        scales = torch.rand(sum(nb) + 1, 2, bs, Hkv, generator=g) * 0.012 + 0.004
        k, v = (kv[:, j].float() * scales[:, j, ..., None] for j in (0, 1))
        cache = kv
    else:
        cache = torch.randn(sum(nb) + 1, bs * Hkv * (dqk + dv), generator=g).to(dtype)       # a page: keys, then values
        k, v = (t.float() for t in _decode_views(cache, bs, Hkv, dqk, dv))
    want, mass = torch.zeros(len(lens), Hq, dv), torch.zeros(len(lens), Hq, dv)
    for i, n in enumerate(lens):
        if n:
            kk, vv = (t[table[i, : nb[i]].long()].reshape(-1, Hkv, t.shape[-1])[:n].repeat_interleave(Hq // Hkv, 1) for t in (k, v))
            p = (torch.einsum("hd,nhd->hn", q[i].float(), kk) * dqk ** -0.5).softmax(-1)
            want[i], mass[i] = torch.einsum("hn,nhd->hd", p, vv), torch.einsum("hn,nhd->hd", p, vv.abs())
    # a weight is rounded to 16 bits, and once more the result
    u = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    return q, cache, scales, table, torch.tensor(lens, dtype=torch.int32), want, 2 * u * want.abs() + 2 * u * mass + 1e-5


def _decode_views(pages, bs, Hkv, dqk, dv):
    n = bs * Hkv * dqk
    return pages[:, :n].unflatten(1, (bs, Hkv, dqk)), pages[:, n:].unflatten(1, (bs, Hkv, dv))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Hq,Hkv,dqk,dv", [(8, 1, 256, 256), (10, 1, 256, 256), (16, 1, 256, 256), (24, 2, 192, 192), (18, 2, 160, 160),
                                           (12, 1, 256, 128), (9, 1, 128, 136), (17, 1, 256, 256)])
def test_decode_of_wide_heads_in_large_groups(dtype, Hq, Hkv, dqk, dv):
    """Heads wider than 128 in groups around 8 and 16 query heads per key head, where the kernels for one token per sequence part:
    a call of its own, one with a kept scratch, and a replayed graph."""
    lens = [1, 900, 0, 65, 64, 2100, 17]
    q, cache, _, table, sl, want, bound = _decode_case(Hq, Hkv, dqk, dv, lens, dtype)
    qd, td, ld, cd = q.cuda(), table.cuda(), sl.cuda(), _decode_views(cache.cuda(), 64, Hkv, dqk, dv)
    out = torch.full((len(lens), Hq, dv), float("nan"), dtype=dtype, device="cuda")
    ws = torch.empty(32 * len(lens) * Hq * (dv + 1), device="cuda")
    run = lambda **kw: ops.paged_attention_decode(qd, cd, td, ld, dqk ** -0.5, out=out, max_seq_len=max(lens), workspace=ws, **kw)
    check = lambda: bool(((out.float().cpu() - want).abs() <= bound).all())
    for kw in ({}, dict(scratch=ops.decode_scratch(Hq, Hkv, max(dqk, dv), "cuda"))):
        out.fill_(float("nan"))
        run(**kw)
        assert check()
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            run(**kw)
        for _ in range(2):
            out.fill_(float("nan"))
            graph.replay()
            assert check()


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("N,K", [(8, 8), (1024, 1016), (1032, 1016), (4096, 4096), (4104, 4096), (4096, 4104), (8192, 1024),
                                 (8192, 8192), (8200, 8192)])
def test_few_tokens_around_the_choice_of_kernel(M, N, K):
    """Sizes on either side of where the products of one to four tokens change kernels, and a contraction that ends inside a
    warp's piece: sums of products exact in fp32, rounded once."""
    g = torch.Generator(device=DEV).manual_seed(N + M)
    a = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(N, K, generator=g, device=DEV) / K ** 0.5).bfloat16()
    b, r = (torch.randn(*s, generator=g, device=DEV).bfloat16() for s in ((N,), (M, N)))
    want = a.double() @ w.double().T
    torch.testing.assert_close(ops.gemm(a, w).double(), want, rtol=2.0 ** -8, atol=1e-5)
    torch.testing.assert_close(ops.gemm(a, w, bias=b, residual=r).double(), want + b.double() + r.double(), rtol=2.0 ** -8, atol=1e-5)


@pytest.mark.parametrize("M", [1, 32, 33, 64, 65])
@pytest.mark.parametrize("N,K", [(8, 32), (512, 4096), (520, 4096), (64, 16384), (64, 16416), (64, 32768), (16, 65536)])
def test_narrow_products_around_the_choice_of_kernel(M, N, K):
    """Sizes on either side of where narrow products of a decode batch change kernels: one rounding behind fp32 sums."""
    g = torch.Generator(device=DEV).manual_seed(N + M)
    a = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(N, K, generator=g, device=DEV) / K ** 0.5).bfloat16()
    b = torch.randn(N, generator=g, device=DEV).bfloat16()
    want = a.double() @ w.double().T
    torch.testing.assert_close(ops.gemm(a, w).double(), want, rtol=2.0 ** -8, atol=2e-5)
    torch.testing.assert_close(ops.gemm(a, w, bias=b).double(), want + b.double(), rtol=2.0 ** -8, atol=2e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Hq,Hkv,D,int8", [(32, 8, 128, False), (16, 8, 64, False), (8, 1, 128, False), (4, 4, 256, False), (16, 2, 128, True),
                                           (24, 2, 128, True)])
@pytest.mark.parametrize("lens", [[128] * 32, [150, 64, 1, 192] * 20, [192, 193] * 40, [700] * 30 + [650], [3000, 10, 5] * 3, [64] * 300,
                                  [2000], [1, 4000], [1024, 64, 700, 320, 900, 0, 128, 200]])
def test_decode_ranges(dtype, Hq, Hkv, D, int8, lens):
    """The ways in which the CTAs share out the sequences: a part of one each, a whole one each, ranges that end where short
    sequences do and ranges that end anywhere; both 16-bit types, int8 rows widened to either; a kept scratch is zero again."""
    q, cache, scales, table, sl, want, bound = _decode_case(Hq, Hkv, D, D, lens, dtype, int8)
    cd = cache.cuda() if int8 else _decode_views(cache.cuda(), 64, Hkv, D, D)
    scratch = ops.decode_scratch(Hq, Hkv, D, "cuda")
    got = [ops.paged_attention_decode(q.cuda(), cd, table.cuda(), sl.cuda(), D ** -0.5, max_seq_len=max(lens), scratch=scratch,
                                      kv_scales=None if scales is None else scales.cuda()).float().cpu() for _ in range(2)]
    assert torch.equal(got[0], got[1]) and not bool(scratch[:16384].any())
    assert bool(((got[0] - want).abs() <= bound).all()), float((got[0] - want).abs().max())
