"""Mixture-of-experts: routing, alignment, grouped GEMM pipeline and the Qwen3-MoE model."""
import pytest
import torch

from vllm_metax_b200 import LLM, ModelConfig, SamplingParams
from vllm_metax_b200 import _custom_ops as ops
from vllm_metax_b200.layers.fused_moe import fused_experts, reference_moe
from vllm_metax_b200.ops import reference as ref


def moe_cfg(**kw):
    d = dict(architecture="Qwen3MoeForCausalLM", vocab_size=512, hidden_size=128, intermediate_size=256,
             num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2, head_dim=32, qk_norm=True,
             num_experts=8, num_experts_per_tok=2, moe_intermediate_size=64, norm_topk_prob=True,
             max_position_embeddings=256, dtype=torch.float32, seed=0)
    d.update(kw)
    return ModelConfig(**d)


def test_align_gather_combine_roundtrip_cpu():
    T, E, k, H = 37, 8, 2, 64
    ids = torch.randint(0, E, (T, k), dtype=torch.int32)
    sorted_ids, block_expert, total, inv = ops.moe_align_block_size(ids, 128, E, want_inverse=True)
    assert int(total) % 128 == 0
    flat = ids.reshape(-1)
    for b in range(int(total) // 128):
        rows = sorted_ids[b * 128:(b + 1) * 128]
        valid = rows[rows < T * k].long()
        assert bool((flat[valid] == block_expert[b]).all())
    assert bool((sorted_ids[inv.long()] == torch.arange(T * k, dtype=torch.int32)).all())
    x = torch.randn(T, H)
    a = ops.moe_gather(x, sorted_ids, total, k)
    w = torch.rand(T, k)
    out = ops.moe_combine(a, w, inv, T)
    torch.testing.assert_close(out, x * w.sum(-1, keepdim=True), rtol=1e-5, atol=1e-5)


def test_expert_map_drops_remote_pairs_cpu():
    T, E, k = 20, 8, 2
    ids = torch.randint(0, E, (T, k), dtype=torch.int32)
    emap = torch.full((E,), -1, dtype=torch.int32)
    emap[4:8] = torch.arange(4, dtype=torch.int32)
    _, block_expert, total, inv = ops.moe_align_block_size(ids, 128, 4, emap, want_inverse=True)
    remote = ids.reshape(-1) < 4
    assert bool((inv[remote] == -1).all()) and bool((inv[~remote] >= 0).all())


def test_fused_experts_matches_reference_cpu():
    T, E, k, H, I = 50, 8, 2, 64, 32
    x = torch.randn(T, H)
    w13 = torch.randn(E, 2 * I, H) * 0.1
    w2 = torch.randn(E, H, I) * 0.1
    w, ids = ops.topk_gating(torch.randn(T, E), k, True)
    got = fused_experts(x, w13, w2, w, ids, E)
    torch.testing.assert_close(got, reference_moe(x, w13, w2, w, ids), rtol=1e-4, atol=1e-4)
    # two "EP ranks" each computing their half sum to the same result
    parts = []
    for r in range(2):
        emap = torch.full((E,), -1, dtype=torch.int32)
        emap[r * 4:(r + 1) * 4] = torch.arange(4, dtype=torch.int32)
        parts.append(fused_experts(x, w13[r * 4:(r + 1) * 4], w2[r * 4:(r + 1) * 4], w, ids, 4, emap))
    torch.testing.assert_close(parts[0] + parts[1], got, rtol=1e-4, atol=1e-4)


def test_qwen3_moe_generates_cpu():
    llm = LLM(moe_cfg(), device="cpu", block_size=16, max_model_len=128, max_num_seqs=4, max_num_batched_tokens=64,
              num_gpu_blocks=32)
    g = torch.Generator().manual_seed(0)
    prompts = [torch.randint(0, 512, (n,), generator=g).tolist() for n in (19, 33)]
    outs = llm.generate(prompts, SamplingParams(max_tokens=6, ignore_eos=True))
    assert all(len(o.outputs[0].token_ids) == 6 for o in outs)
    # chunked prefill must not change the result
    llm2 = LLM(moe_cfg(), device="cpu", block_size=16, max_model_len=128, max_num_seqs=4, max_num_batched_tokens=16,
               num_gpu_blocks=32)
    llm2.engine.runner.model.load_state_dict(llm.engine.runner.model.state_dict())
    outs2 = llm2.generate(prompts, SamplingParams(max_tokens=6, ignore_eos=True))
    assert [o.outputs[0].token_ids for o in outs] == [o.outputs[0].token_ids for o in outs2]


# ------------------------------------------------------------------ GPU kernels
gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("E,k,scoring", [(128, 8, "softmax"), (256, 8, "sigmoid"), (64, 6, "sqrtsoftplus"), (8, 2, "softmax")])
def test_topk_gating_gpu(E, k, scoring, kernel_status_ok):
    g = torch.randn(77, E, device="cuda", dtype=torch.float32)   # fp32: no exact ties between experts
    bias = torch.randn(E, device="cuda") * 0.1 if scoring != "softmax" else None
    w, ids = ops.topk_gating(g, k, True, scoring, bias, 2.5)
    ww, wids = ops.topk_gating(g.cpu().float(), k, True, scoring, None if bias is None else bias.cpu(), 2.5)
    assert torch.equal(ids.cpu().sort(-1)[0], wids.sort(-1)[0])
    torch.testing.assert_close(w.cpu().sort(-1)[0], ww.sort(-1)[0], rtol=2e-2, atol=1e-3)


@gpu
def test_grouped_topk_gpu(kernel_status_ok):
    g = torch.randn(50, 256, device="cuda", dtype=torch.float32)
    bias = torch.randn(256, device="cuda") * 0.1
    w, ids = ops.grouped_topk(g, 8, True, 8, 4, "sigmoid", bias, 2.5)
    ww, wids = ref.grouped_topk(g.cpu(), 8, True, 8, 4, "sigmoid", bias.cpu(), 2.5)
    assert torch.equal(ids.cpu().sort(-1)[0], wids.sort(-1)[0])
    torch.testing.assert_close(w.cpu().sort(-1)[0], ww.sort(-1)[0], rtol=1e-3, atol=1e-4)


@gpu
@pytest.mark.parametrize("T,E,k,H,I", [(300, 16, 4, 1024, 512), (9, 128, 8, 2048, 768), (2000, 8, 2, 512, 1024)])
def test_fused_experts_gpu(T, E, k, H, I, kernel_status_ok):
    x = torch.randn(T, H, device="cuda", dtype=torch.bfloat16)
    w13 = (torch.randn(E, 2 * I, H, device="cuda") * 0.05).to(torch.bfloat16)
    w2 = (torch.randn(E, H, I, device="cuda") * 0.05).to(torch.bfloat16)
    w, ids = ops.topk_gating(torch.randn(T, E, device="cuda"), k, True)
    got = fused_experts(x, w13, w2, w, ids, E)
    want = reference_moe(x.cpu().float(), w13.cpu().float(), w2.cpu().float(), w.cpu(), ids.cpu())
    a, b = got.float().cpu().flatten(), want.flatten()
    assert 1 - float(torch.dot(a, b) / (a.norm() * b.norm())) < 1e-3


@gpu
def test_qwen3_moe_gpu_tracks_cpu(kernel_status_ok):
    cfg = dict(hidden_size=512, head_dim=128, num_attention_heads=4, num_key_value_heads=2, moe_intermediate_size=256,
               num_experts=16, num_experts_per_tok=4, vocab_size=1024)
    kw = dict(block_size=64, max_model_len=256, max_num_seqs=4, max_num_batched_tokens=512, num_gpu_blocks=32)
    cpu = LLM(moe_cfg(**cfg), device="cpu", **kw)
    gpu_llm = LLM(moe_cfg(**cfg, dtype=torch.bfloat16), device="cuda", enforce_eager=True, **kw)
    sd = {k: v.to(torch.bfloat16) for k, v in cpu.engine.runner.model.state_dict().items()}
    gpu_llm.engine.runner.model.load_state_dict(sd)
    cpu.engine.runner.model.load_state_dict({k: v.float() for k, v in sd.items()})
    from tests.test_e2e_gpu import lockstep

    g = torch.Generator().manual_seed(0)
    prompts = [torch.randint(0, 1024, (n,), generator=g).tolist() for n in (70, 130)]
    lockstep(cpu, gpu_llm, prompts, steps=4, tol=2e-2)


def test_moe_chunked_over_tokens_equals_one_pass(monkeypatch):
    """B200_FUSED_MOE_CHUNK_SIZE: a long step goes through the experts in pieces with the same result."""
    import torch

    from vllm_metax_b200.layers.fused_moe import FusedMoE

    torch.manual_seed(0)
    moe = FusedMoE(8, 2, 32, 16, dtype=torch.float32)
    moe.w13_weight.data.normal_(0, 0.2)
    moe.w2_weight.data.normal_(0, 0.2)
    x, logits, shared = torch.randn(70, 32), torch.randn(70, 8), torch.randn(70, 32)
    want = moe.forward(x, logits, shared)
    monkeypatch.setenv("B200_FUSED_MOE_CHUNK_SIZE", "16")
    torch.testing.assert_close(moe.forward(x, logits, shared), want, rtol=1e-5, atol=1e-5)
    monkeypatch.setenv("B200_FUSED_MOE_CHUNK_SIZE", "0")
    torch.testing.assert_close(moe.forward(x, logits, None), moe.forward(x, logits, shared) - shared, rtol=1e-5, atol=1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("numel,experts,block", [(4096, 128, 128), (4104, 3, 16), (9000, 64, 128), (70001, 128, 128),
                                                 (200003, 1024, 64)])
@pytest.mark.parametrize("mapped", [False, True])
def test_moe_align_by_several_ctas(numel, experts, block, mapped):
    """The order of one CTA's placement and of many's against the stable sort: around the size where they part, segments that
    end early, experts without pairs, pairs routed elsewhere."""
    from vllm_metax_b200 import _custom_ops as ops

    g = torch.Generator().manual_seed(numel)
    ids = (torch.rand(numel, generator=g).pow(3) * experts).to(torch.int32)      # the first experts get most
    emap = None
    if mapped:
        emap = torch.arange(experts, dtype=torch.int32)
        emap[::3] = -1
    want = ops.moe_align_block_size(ids, block, experts, emap, want_inverse=True)
    got = ops.moe_align_block_size(ids.cuda(), block, experts, None if emap is None else emap.cuda(), want_inverse=True)
    for a, b in zip(got, want):
        assert torch.equal(a.cpu().reshape(-1), b.reshape(-1))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,topk,hidden,experts", [(1, 8, 2048, 16), (37, 3, 2176, 8), (300, 10, 7168, 64), (5, 1, 264, 4)])
def test_moe_rows_from_the_pairs(dtype, tokens, topk, hidden, experts):
    """Scattered rows equal gathered ones (padding apart), as they are, weighted and quantised; combined rows equal the sum in
    fp32 in the order of the pairs, rounded once."""
    from vllm_metax_b200 import _custom_ops as ops

    g = torch.Generator().manual_seed(tokens)
    x = torch.randn(tokens, hidden, generator=g).to(dtype).cuda()
    ids = torch.stack([torch.randperm(experts, generator=g)[:topk] if topk <= experts else
                       torch.randint(0, experts, (topk,), generator=g) for _ in range(tokens)]).to(torch.int32).cuda()
    emap = torch.arange(experts, dtype=torch.int32).cuda()
    emap[0] = -1                                            # one expert is elsewhere
    w = torch.rand(tokens, topk, generator=g).cuda()
    sorted_ids, be, total, inv = ops.moe_align_block_size(ids, 128, experts, emap, want_inverse=True)
    real = sorted_ids < ids.numel()
    for weights in (None, w):
        got, want = ops.moe_scatter(x, inv, sorted_ids, total, topk, weights), ops.moe_gather(x, sorted_ids, total, topk, weights)
        assert torch.equal(got[real], want[real])
    if hidden % 128 == 0:
        q, s = ops.moe_scatter_fp8(x, inv, sorted_ids, total, topk)
        wq, ws = ops.per_token_group_quant_fp8(ops.moe_gather(x, sorted_ids, total, topk), 128)
        assert torch.equal(q[real].view(torch.uint8), wq[real].view(torch.uint8)) and torch.equal(s[real], ws[real])
        h = torch.cat([want, want.flip(1)], 1)
        a, b = ops.silu_and_mul_per_block_quant(h, 128), ops.silu_and_mul_per_block_quant(h, 128, sorted_ids=sorted_ids, numel=ids.numel())
        assert torch.equal(a[0][real].view(torch.uint8), b[0][real].view(torch.uint8)) and torch.equal(a[1][real], b[1][real])
    shared = torch.randn(tokens, hidden, generator=g).to(dtype).cuda()
    y = torch.randn(sorted_ids.numel(), hidden, generator=g).to(dtype).cuda()
    out = ops.moe_combine(y, w, inv, tokens, shared)
    acc, iv = shared.float(), inv.view(tokens, topk).long()
    for k in range(topk):
        acc = torch.where((iv[:, k] >= 0)[:, None], acc + w[:, k: k + 1] * y[iv[:, k].clamp_min(0)].float(), acc)
    torch.testing.assert_close(out.float(), acc, rtol=2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10, atol=1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("T,topk,E,N,K,epi", [(3, 2, 4, 256, 128, 0), (64, 8, 128, 1536, 256, 1), (500, 3, 5, 300, 72, 0)])
def test_grouped_products_without_padding(T, topk, E, N, K, epi):
    """One, a few and all rows of a block, both tile widths, a ragged contraction: padding rows hold NaN, are not read, and the
    others equal those of the call that takes every row."""
    g = torch.Generator().manual_seed(T)
    ids = torch.stack([torch.randperm(E, generator=g)[:topk] for _ in range(T)]).to(torch.int32).cuda()
    sorted_ids, be, total, inv = ops.moe_align_block_size(ids, 128, E, want_inverse=True)
    real = sorted_ids < ids.numel()
    x = torch.randn(T, K, generator=g).bfloat16().cuda()
    a = ops.moe_scatter(x, inv, sorted_ids, total, topk)
    a[~real] = float("nan")
    w = torch.randn(E, N, K, generator=g).bfloat16().cuda()
    got = ops.gemm_grouped(a, w, be, total, epi, None, sorted_ids, ids.numel())
    want = ops.gemm_grouped(torch.where(real[:, None], a, torch.zeros_like(a)), w, be, total, epi)
    assert torch.equal(got[real], want[real]) and bool(torch.isfinite(got[real]).all())
    ops.check_kernel_status(0)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,K,N", [(1, 8, 8), (64, 2048, 2048), (5, 3000, 4104)])
def test_gate_of_a_shared_expert(dtype, T, K, N):
    """Rows shorter than a CTA and longer than one pass of it, strided tokens: an exact product up to fp32 sums, one rounding."""
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, 2 * K, generator=g).to(dtype).cuda()[:, :K]
    w = (torch.randn(1, K, generator=g) / K ** 0.5).to(dtype).cuda()
    y = torch.randn(T, N, generator=g).to(dtype).cuda()
    with torch.no_grad():
        got = ops.sigmoid_dot_scale(x, w, y)
    want = torch.sigmoid(x.double() @ w.double().T) * y.double()
    # one rounding to the type, of 8 or 11 significant bits; the sigmoid's exponential and the sum to 2^-18
    torch.testing.assert_close(got.double(), want, rtol=(2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.05, atol=1e-6)


def test_kernels_that_start_early_wait_before_their_loads():
    """A kernel that may run beside the one in front of it waits first, and its loads are none that a compiler may move in front
    of the wait: those through const pointers with ``__restrict__``."""
    import pathlib
    import re

    found = 0
    for src in sorted((pathlib.Path(ops.__file__).parent / "csrc").glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", src.read_text())
        early = set(re.findall(r"pdl_run\((\w+)", text)) - {"kern"} | set(re.findall(r"auto kern = (\w+)", text) if "pdl_" in text else [])
        for head, body in re.findall(r"__global__([^{;]*)\{(.*?)\n\}", text, re.S):
            name = re.findall(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", head))[0]
            if name not in early and "pdl_wait" not in body and "pdl_trigger" not in body:
                continue
            found += 1
            assert "pdl_wait();" in body, (src.name, name)
            assert "__restrict__" not in head, (src.name, name)
    assert found >= 9


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,N,K", [(1, 2048, 512), (2, 2048, 4096), (3, 7168, 2048), (4, 512, 2048), (33, 512, 2048), (64, 256, 512)])
def test_gate_behind_a_product_in_a_graph(dtype, T, N, K, kernel_status_ok):
    """The gate starts while the product in front of it, which makes its rows, still runs: replays over changing inputs give what
    the two calls give one after the other."""
    g = torch.Generator().manual_seed(T)
    h = torch.empty(T, K, dtype=dtype, device="cuda")
    x = torch.empty(T, 2048, dtype=dtype, device="cuda")
    w = (torch.randn(N, K, generator=g) / K ** 0.5).to(dtype).cuda()
    gate = (torch.randn(1, 2048, generator=g) / 50).to(dtype).cuda()
    first = lambda a: torch.mul(a, 2.0)                     # (a kernel in front of the product, so that this starts early too)
    step = lambda: ops.sigmoid_dot_scale(x, gate, ops.gemm(first(h), w))
    with torch.no_grad():
        h.zero_(), x.zero_()
        step()
        torch.cuda.synchronize()
        graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(4):                              # (several in a row: the one in front of a product is a gate)
                out = step()
        for _ in range(20):
            h.copy_(torch.randn(T, K, generator=g))
            x.copy_(torch.randn(T, 2048, generator=g))
            want = step().clone()
            graph.replay()
            assert torch.equal(out, want)


@pytest.mark.gpu
@pytest.mark.parametrize("T,topk,E,N,K,epi", [(255, 2, 4, 256, 128, 0), (256, 2, 4, 256, 128, 1), (257, 2, 4, 1024, 192, 0), (1500, 3, 5, 300, 72, 0),
                                              (900, 2, 2, 512, 128, 1)])
def test_grouped_products_of_full_blocks(T, topk, E, N, K, epi):
    """Around the mean of 128 rows per expert from which whole blocks are read, with experts that get far fewer: padding rows hold NaN
    and touch nothing, the others equal those of the call that takes every row."""
    g = torch.Generator().manual_seed(T)
    ids = torch.stack([torch.multinomial(torch.arange(1, E + 1).float() ** 2, topk, generator=g) for _ in range(T)]).to(torch.int32).cuda()
    sorted_ids, be, total, inv = ops.moe_align_block_size(ids, 128, E, want_inverse=True)
    real = sorted_ids < ids.numel()
    x = torch.randn(T, K, generator=g).bfloat16().cuda()
    a = ops.moe_scatter(x, inv, sorted_ids, total, topk)
    a[~real] = float("nan")
    w = torch.randn(E, N, K, generator=g).bfloat16().cuda()
    got = ops.gemm_grouped(a, w, be, total, epi, None, sorted_ids, ids.numel())
    want = ops.gemm_grouped(torch.where(real[:, None], a, torch.zeros_like(a)), w, be, total, epi)
    assert torch.equal(got[real], want[real]) and bool(torch.isfinite(got[real]).all())
    ops.check_kernel_status(0)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,topk,hidden", [(4095, 2, 4096), (4096, 2, 4096), (4097, 5, 2056), (5000, 1, 264)])
def test_combined_rows_of_many_tokens(tokens, topk, hidden):
    """Around the number of tokens from which a CTA walks its whole row: sums in fp32 in the order of the pairs, rounded once."""
    g = torch.Generator(device="cuda").manual_seed(tokens)
    y = torch.randn(tokens * topk, hidden, generator=g, device="cuda").bfloat16()
    w = torch.rand(tokens, topk, generator=g, device="cuda")
    inv = torch.randperm(tokens * topk, generator=g, device="cuda").to(torch.int32)
    inv[::11] = -1
    shared = torch.randn(tokens, hidden, generator=g, device="cuda").bfloat16()
    acc, iv = shared.float(), inv.view(tokens, topk).long()
    for k in range(topk):
        acc = torch.where((iv[:, k] >= 0)[:, None], acc + w[:, k: k + 1] * y[iv[:, k].clamp_min(0)].float(), acc)
    torch.testing.assert_close(ops.moe_combine(y, w, inv, tokens, shared).float(), acc, rtol=2.0 ** -7, atol=1e-5)
