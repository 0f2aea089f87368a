"""Gated delta rule (recurrent kernel vs the fp32 recurrence) and bidirectional encoder attention."""
import os
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

gpu = pytest.mark.gpu


def _gdn_case(dtype, seed=0, Hq=2, Hv=4, lens=(5, 1, 33)):
    g_ = torch.Generator().manual_seed(seed)
    T = sum(lens)
    q = torch.randn(T, Hq, 128, generator=g_).to(dtype)
    k = torch.randn(T, Hq, 128, generator=g_).to(dtype)
    v = torch.randn(T, Hv, 128, generator=g_).to(dtype)
    g = -torch.rand(T, Hv, generator=g_) * 0.5
    beta = torch.rand(T, Hv, generator=g_)
    qsl = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    state = torch.randn(4, Hv, 128, 128, generator=g_) * 0.1
    idx = torch.tensor([2, 0, 3], dtype=torch.int32)
    has = torch.tensor([1, 0, 1], dtype=torch.int32)
    return q, k, v, g, beta, qsl, state, idx, has


def test_gdn_reference_properties():
    from vllm_metax_b200.ops.gdn import gated_delta_rule

    q, k, v, g, beta, qsl, state, idx, has = _gdn_case(torch.float32)
    s1 = state.clone()
    o_all = gated_delta_rule(q, k, v, g, beta, qsl, s1, idx, has)
    # the same tokens fed in two calls (chunked prefill) continue from the stored state
    s2 = state.clone()
    cut = torch.tensor([0, 3, 4, 20], dtype=torch.int32)                  # first 3 / 1 / 16 tokens of each sequence
    first = torch.cat([torch.arange(0, 3), torch.arange(5, 6), torch.arange(6, 22)])
    o_a = gated_delta_rule(q[first], k[first], v[first], g[first], beta[first], cut, s2, idx, has)
    rest = torch.cat([torch.arange(3, 5), torch.arange(22, 39)])
    cut2 = torch.tensor([0, 2, 2, 19], dtype=torch.int32)
    o_b = gated_delta_rule(q[rest], k[rest], v[rest], g[rest], beta[rest], cut2, s2, idx, torch.ones(3, dtype=torch.int32))
    torch.testing.assert_close(o_a, o_all[first], rtol=1e-4, atol=1e-4)
    torch.testing.assert_close(o_b, o_all[rest], rtol=1e-4, atol=1e-4)
    torch.testing.assert_close(s2, s1, rtol=1e-4, atol=1e-4)
    assert torch.equal(s1[1], state[1])                                   # an unused slot is untouched


@pytest.mark.parametrize("lens,chunk", [((5, 1, 33), 64), ((200, 64, 129), 64), ((70, 3, 17), 16)])
def test_gdn_chunked_form_equals_the_recurrence(lens, chunk):
    """The matrix form over chunks (what prefill uses when switched on) against the token-by-token recurrence:
    sequences shorter than, equal to and not a multiple of the chunk, initial states, stored final states."""
    from vllm_metax_b200.ops.gdn import gated_delta_rule_chunked, gated_delta_rule_ref

    q, k, v, g, beta, qsl, state, idx, has = _gdn_case(torch.float32, seed=4, lens=lens)
    s_ref, s_chk = state.clone(), state.clone()
    want = gated_delta_rule_ref(q, k, v, g, beta, qsl, s_ref, idx, has)
    got = gated_delta_rule_chunked(q, k, v, g, beta, qsl, s_chk, idx, has, chunk=chunk)
    torch.testing.assert_close(got, want, rtol=2e-4, atol=2e-4)
    torch.testing.assert_close(s_chk, s_ref, rtol=2e-4, atol=2e-4)
    assert torch.equal(s_chk[1], state[1])
    # strong decay and beta = 1 (the stiffest case for the triangular solve)
    g2, b2 = g * 8, torch.ones_like(beta)
    s_ref, s_chk = state.clone(), state.clone()
    want = gated_delta_rule_ref(q, k, v, g2, b2, qsl, s_ref, idx, has)
    got = gated_delta_rule_chunked(q, k, v, g2, b2, qsl, s_chk, idx, has, chunk=chunk)
    torch.testing.assert_close(got, want, rtol=5e-4, atol=5e-4)


def test_gdn_dispatch_takes_the_chunked_form_when_switched_on(monkeypatch):
    from vllm_metax_b200.ops import gdn

    q, k, v, g, beta, qsl, state, idx, has = _gdn_case(torch.float32, seed=2, lens=(300, 2, 40))
    calls = []
    real = gdn.gated_delta_rule_chunked
    monkeypatch.setattr(gdn, "gated_delta_rule_chunked", lambda *a, **kw: (calls.append(1), real(*a, **kw))[1])
    s0 = state.clone()
    want = gdn.gated_delta_rule(q, k, v, g, beta, qsl, s0, idx, has)
    assert not calls
    monkeypatch.setenv("B200_GDN_CHUNKED", "1")
    s1 = state.clone()
    got = gdn.gated_delta_rule(q, k, v, g, beta, qsl, s1, idx, has)
    assert calls == [1]
    torch.testing.assert_close(got, want, rtol=2e-4, atol=2e-4)
    torch.testing.assert_close(s1, s0, rtol=2e-4, atol=2e-4)
    short = torch.tensor([0, 5, 6, 39], dtype=torch.int32)                # no long chunk in the batch: recurrent
    gdn.gated_delta_rule(q[:39], k[:39], v[:39], g[:39], beta[:39], short, state.clone(), idx, has)
    assert calls == [1]


@gpu
def test_gdn_kernel_matches_reference():
    from vllm_metax_b200.ops.gdn import gated_delta_rule, gated_delta_rule_ref

    q, k, v, g, beta, qsl, state, idx, has = _gdn_case(torch.bfloat16, seed=1)
    s_ref = state.clone()
    want = gated_delta_rule_ref(q, k, v, g, beta, qsl, s_ref, idx, has)
    s_gpu = state.clone().cuda()
    got = gated_delta_rule(q.cuda(), k.cuda(), v.cuda(), g.cuda(), beta.cuda(), qsl.cuda(), s_gpu, idx.cuda(), has.cuda())
    torch.testing.assert_close(got.float().cpu(), want.float(), rtol=3e-2, atol=3e-2)
    torch.testing.assert_close(s_gpu.cpu(), s_ref, rtol=2e-3, atol=2e-3)
    # no state pool: every sequence starts from zero and nothing is stored
    o2 = gated_delta_rule(q.cuda(), k.cuda(), v.cuda(), g.cuda(), beta.cuda(), qsl.cuda())
    w2 = gated_delta_rule_ref(q, k, v, g, beta, qsl)
    torch.testing.assert_close(o2.float().cpu(), w2.float(), rtol=3e-2, atol=3e-2)


def _vit_ref(q, k, v, cu, scale):
    out = torch.zeros_like(q, dtype=torch.float32)
    for a, b in zip(cu[:-1].tolist(), cu[1:].tolist()):
        s = torch.einsum("qhd,khd->hqk", q[a:b].float(), k[a:b].float()) * scale
        out[a:b] = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), v[a:b].float())
    return out


def test_encoder_attention_cpu():
    from vllm_metax_b200.layers.mm_encoder_attention import MMEncoderAttention

    g = torch.Generator().manual_seed(0)
    H, D = 4, 64
    cu = torch.tensor([0, 9, 9 + 16, 9 + 16 + 5], dtype=torch.int32)
    q, k, v = (torch.randn(30, H * D, generator=g) for _ in range(3))
    attn = MMEncoderAttention(H, D)
    out = attn(q, k, v, cu, 16)
    want = _vit_ref(q.view(30, H, D), k.view(30, H, D), v.view(30, H, D), cu, D ** -0.5)
    torch.testing.assert_close(out.float(), want, rtol=1e-4, atol=1e-4)
    # batched [B, S, H, D] form without cu_seqlens: every image is one sequence
    qb = torch.randn(2, 7, H, D, generator=g)
    ob = attn(qb, qb, qb)
    wb = _vit_ref(qb.reshape(14, H, D), qb.reshape(14, H, D), qb.reshape(14, H, D), torch.tensor([0, 7, 14]), D ** -0.5)
    torch.testing.assert_close(ob.reshape(14, H, D).float(), wb, rtol=1e-4, atol=1e-4)


@gpu
@pytest.mark.parametrize("D", [64, 128])
def test_encoder_attention_gpu(D):
    from vllm_metax_b200.layers.mm_encoder_attention import MMEncoderAttention

    g = torch.Generator().manual_seed(1)
    H = 8
    lens = [200, 64, 1, 333]
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    T = sum(lens)
    q, k, v = (torch.randn(T, H, D, generator=g).to(torch.bfloat16) for _ in range(3))
    out = MMEncoderAttention(H, D)(q.cuda(), k.cuda(), v.cuda(), cu.cuda(), max(lens))
    torch.testing.assert_close(out.float().cpu(), _vit_ref(q, k, v, cu, D ** -0.5), rtol=3e-2, atol=3e-2)


# ------------------------------------------------------------------------------------------ short causal convolution
def _conv_case(dtype, seed=0, C=384, K=4, lens=(5, 1, 70, 2)):
    g_ = torch.Generator().manual_seed(seed)
    T = sum(lens)
    x = torch.randn(T, C + 64, generator=g_).to(dtype)[:, :C]            # row pitch larger than C
    w = (torch.randn(C, K, generator=g_) * 0.5).to(dtype)
    bias = (torch.randn(C, generator=g_) * 0.1).to(dtype)
    qsl = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    state = torch.randn(6, K - 1, C, generator=g_).to(dtype)
    idx = torch.tensor([4, 1, 0, 5], dtype=torch.int32)
    has = torch.tensor([1, 1, 0, 1], dtype=torch.int32)
    return x, w, bias, qsl, state, idx, has


def test_causal_conv1d_reference_is_a_streaming_convolution():
    """Feeding a sequence in pieces through the carry gives the same outputs as feeding it at once."""
    from vllm_metax_b200.ops.gdn import causal_conv1d

    x, w, bias, *_ = _conv_case(torch.float32, lens=(40,))
    one = torch.tensor([0], dtype=torch.int32)
    whole = causal_conv1d(x, w, bias, torch.zeros(1, 3, x.shape[1]), torch.tensor([0, 40], dtype=torch.int32), one,
                          torch.tensor([0], dtype=torch.int32))
    st = torch.zeros(1, 3, x.shape[1])
    parts, pos = [], 0
    for n in (1, 2, 17, 1, 19):
        parts.append(causal_conv1d(x[pos:pos + n], w, bias, st, torch.tensor([0, n], dtype=torch.int32), one,
                                   torch.tensor([1 if pos else 0], dtype=torch.int32)))
        pos += n
    torch.testing.assert_close(torch.cat(parts), whole, atol=1e-5, rtol=1e-5)
    # and against torch's own depthwise convolution
    ref = torch.nn.functional.conv1d(x.t()[None], w[:, None], bias, padding=3, groups=x.shape[1])[0, :, :40].t()
    torch.testing.assert_close(whole, torch.nn.functional.silu(ref), atol=1e-5, rtol=1e-5)


@gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("K", [2, 4])
def test_causal_conv1d_kernel_matches_reference(dtype, K):
    from vllm_metax_b200.ops.gdn import causal_conv1d, causal_conv1d_ref

    x, w, bias, qsl, state, idx, has = _conv_case(dtype, K=K)
    st_ref = state.clone()
    want = causal_conv1d_ref(x, w, bias, st_ref, qsl, idx, has)
    st = state.cuda()
    got = causal_conv1d(x.cuda(), w.cuda(), bias.cuda(), st, qsl.cuda(), idx.cuda(), has.cuda())
    tol = 2e-2 if dtype == torch.bfloat16 else 1e-5
    torch.testing.assert_close(got.float().cpu(), want.float(), atol=tol, rtol=tol)
    torch.testing.assert_close(st.float().cpu(), st_ref.float(), atol=0, rtol=0)          # carries are copies of inputs
    # no carry: every sequence starts from zeros and nothing is written back
    got2 = causal_conv1d(x.cuda(), w.cuda(), None, None, qsl.cuda(), None, None, silu=False)
    want2 = causal_conv1d_ref(x, w, None, None, qsl, None, None, silu=False)
    torch.testing.assert_close(got2.float().cpu(), want2.float(), atol=tol, rtol=tol)


@gpu
def test_qwen3_next_engine_on_gpu_graphs_match_eager():
    """Hybrid model end to end on the GPU kernels (delta-rule head size 128, attention head size 128): decode steps
    replayed from CUDA graphs must give the tokens of the eager run, with requests spread over several state slots."""
    from vllm_metax_b200 import LLM, SamplingParams
    from vllm_metax_b200.config import ModelConfig

    hf = dict(architectures=["Qwen3NextForCausalLM"], vocab_size=1024, hidden_size=256, num_hidden_layers=4,
              num_attention_heads=4, num_key_value_heads=2, head_dim=128, max_position_embeddings=512,
              intermediate_size=512, moe_intermediate_size=128, shared_expert_intermediate_size=128, num_experts=8,
              num_experts_per_tok=2, linear_num_value_heads=4, linear_num_key_heads=2, linear_key_head_dim=128,
              linear_value_head_dim=128, linear_conv_kernel_dim=4, norm_topk_prob=True, torch_dtype="bfloat16")
    g = torch.Generator().manual_seed(0)
    prompts = [torch.randint(0, 1024, (n,), generator=g).tolist() for n in (37, 5, 130, 64, 9)]
    sp = SamplingParams(max_tokens=12, temperature=0.0, ignore_eos=True)
    outs = []
    for eager in (True, False):
        llm = LLM(ModelConfig.from_hf_dict(hf, seed=3), max_model_len=256, max_num_seqs=4, max_num_batched_tokens=128,
                  num_gpu_blocks=64, enforce_eager=eager, load_format="dummy")
        outs.append([list(o.outputs[0].token_ids) for o in llm.generate(prompts, sp)])
        assert not llm.engine.runner.state_slots
        del llm
        torch.cuda.empty_cache()
    assert outs[0] == outs[1]
    assert all(len(t) == 12 for t in outs[0])


def _gdn_f64(q, k, v, g, beta, lens, state, idx, has, l2norm=True):
    qf, kf, vf = q.double(), k.double(), v.double()
    if l2norm:
        qf = qf * torch.rsqrt(qf.pow(2).sum(-1, keepdim=True) + 1e-6)
        kf = kf * torch.rsqrt(kf.pow(2).sum(-1, keepdim=True) + 1e-6)
    rep = v.shape[1] // q.shape[1]
    qf, kf = qf.repeat_interleave(rep, 1) * 128 ** -0.5, kf.repeat_interleave(rep, 1)
    out, state, t = torch.zeros_like(vf), state.double(), 0
    for b, n in enumerate(lens):
        S = state[idx[b]].clone() if has[b] else torch.zeros_like(state[0])
        for t in range(t, t + n):
            S = S * torch.exp(g[t].double())[:, None, None]
            u = beta[t].double()[:, None] * (vf[t] - torch.einsum("hkv,hk->hv", S, kf[t]))
            S = S + torch.einsum("hk,hv->hkv", kf[t], u)
            out[t] = torch.einsum("hkv,hk->hv", S, qf[t])
        t = t + 1 if n else t
        if n:
            state[idx[b]] = S
    return out, state


@gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens", [(1, 1, 1), (4, 16, 1), (3, 0, 17), (33, 5, 64), (31, 2, 100)])
@pytest.mark.parametrize("pitch", [0, 8, 3])               # rows behind one another, on 16 bytes, on 2 bytes only
def test_gdn_groups_of_tokens(dtype, lens, pitch):
    """Steps of one token and groups of four: sequences that end inside a group or a stage, empty ones, strided rows, strong decay.
    Outputs are rounded once (half a unit of 2^-8 or 2^-11) behind sums of 128 fp32 products: fp32 state within 1e-5."""
    from vllm_metax_b200.ops.gdn import gated_delta_rule

    q, k, v, g, beta, qsl, state, idx, has = _gdn_case(dtype, seed=7, lens=lens)
    g[::3] *= 60                                            # e^-30 in one token
    want, s_want = _gdn_f64(q, k, v, g, beta, lens, state, idx, has)
    wide = lambda x: torch.cat([x.flatten(1), x.new_zeros(x.shape[0], pitch)], 1).cuda()[:, : x[0].numel()].unflatten(1, x.shape[1:])
    s_got = state.cuda()
    got = gated_delta_rule(wide(q), wide(k), wide(v), g.cuda(), beta.cuda(), qsl.cuda(), s_got, idx.cuda(), has.cuda())
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    torch.testing.assert_close(got.cpu().double(), want, rtol=eps, atol=1e-5)
    torch.testing.assert_close(s_got.cpu().double(), s_want, rtol=1e-5, atol=1e-5)


@gpu
def test_gdn_gates_and_norm_in_the_kernels():
    """``ba`` of a projection instead of decays and betas, the grouped projection as the convolution's input, and the gated
    norm of a view, against the same from plain tensors."""
    from vllm_metax_b200.ops import gdn

    gen = torch.Generator().manual_seed(3)
    for lens in ((1, 1, 1), (40, 3, 9)):
        T, nk, rep, d = sum(lens), 2, 2, 128
        qkvz = torch.randn(T, nk * 6 * d, generator=gen).bfloat16().cuda()
        ba = torch.randn(T, nk * 2 * rep, generator=gen).bfloat16().cuda()
        a_log, dt = torch.rand(4, generator=gen).cuda(), torch.randn(4, generator=gen).cuda()
        w = torch.randn(nk * 4 * d, 4, generator=gen).bfloat16().cuda()
        qsl = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32).cuda()
        idx, has = torch.tensor([2, 0, 3], dtype=torch.int32).cuda(), torch.tensor([1, 0, 1], dtype=torch.int32).cuda()
        conv = torch.randn(4, 3, nk * 4 * d, generator=gen).bfloat16().cuda()
        flat = torch.cat([t.flatten(1) for t in qkvz.view(T, nk, -1).split([d, d, rep * d, rep * d], -1)[:3]], -1)
        c1, c2 = conv.clone(), conv.clone()
        got = gdn.causal_conv1d(qkvz, w, None, c1, qsl, idx, has, heads=(nk, d, rep * d))
        assert torch.equal(got, gdn.causal_conv1d(flat, w, None, c2, qsl, idx, has)) and torch.equal(c1, c2)
        ref = gdn.causal_conv1d_ref(flat.cpu(), w.cpu(), None, conv.cpu().clone(), qsl.cpu(), idx.cpu(), has.cpu())
        torch.testing.assert_close(got.cpu(), ref, rtol=2.0 ** -7, atol=1e-3)
        q, k, v = (t.unflatten(1, (-1, d)) for t in got.split([nk * d, nk * d, nk * rep * d], -1))
        b, a = ba.view(T, nk, 2 * rep).chunk(2, -1)
        beta = torch.sigmoid(b.reshape(T, -1).float())
        g = -torch.exp(a_log) * torch.nn.functional.softplus(a.reshape(T, -1).float() + dt)
        s0 = torch.randn(4, 4, d, d, generator=gen).cuda() * 0.1
        s1, s2 = s0.clone(), s0.clone()
        o1 = gdn.gated_delta_rule_ba(q, k, v, ba, a_log, dt, qsl, s1, idx, has)
        o2 = gdn.gated_delta_rule(q, k, v, g, beta, qsl, s2, idx, has)
        torch.testing.assert_close(o1, o2, rtol=2.0 ** -7, atol=1e-5)
        torch.testing.assert_close(s1, s2, rtol=1e-5, atol=1e-5)
        z = qkvz.view(T, nk, -1)[..., 4 * d:]
        nw = torch.randn(d, generator=gen).bfloat16().cuda()
        y = gdn.gated_head_norm(o1.reshape(T, -1), z, nw, d, 1e-6)
        n = o1.float() * torch.rsqrt(o1.float().pow(2).mean(-1, keepdim=True) + 1e-6) * nw.float()
        want = n.bfloat16().float() * torch.nn.functional.silu(z.reshape(T, -1, d).float())
        # the normed value may round to the next bf16 (2^-7 at most of it), the product rounds once more (2^-8)
        torch.testing.assert_close(y.view(T, -1, d).float(), want, rtol=2.0 ** -7 + 2.0 ** -8, atol=1e-5)
        y = gdn.gated_head_norm(o1.reshape(T, -1), z, None, d)
        want = o1.float() * torch.sigmoid(z.reshape(T, -1, d).float())
        torch.testing.assert_close(y.view(T, -1, d).float(), want, rtol=2.0 ** -7, atol=1e-6)


@gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gdn_rows_alone_and_in_company(dtype, monkeypatch):
    """With results that must not depend on the batch, a decode row and a prompt have the same outputs and states, bit for bit,
    alone, beside one another, and with the prompt cut in two."""
    from vllm_metax_b200 import _custom_ops as ops
    from vllm_metax_b200.ops.gdn import gated_delta_rule, gated_delta_rule_ba

    monkeypatch.setattr(ops, "_batch_invariant", True)
    q, k, v, g, beta, _, state, _, _ = _gdn_case(dtype, seed=11, lens=(1, 50))
    ba = torch.randn(51, 8, generator=torch.Generator().manual_seed(12)).to(dtype)
    a_log, dt = torch.zeros(4), torch.ones(4)
    cuda = lambda *ts: [t.cuda() for t in ts]
    ints = lambda *x: torch.tensor(x, dtype=torch.int32, device="cuda")
    q, k, v, g, beta, ba, a_log, dt = cuda(q, k, v, g, beta, ba, a_log, dt)
    for gates in (lambda r: (gated_delta_rule, (g[r], beta[r])), lambda r: (gated_delta_rule_ba, (ba[r], a_log, dt))):
        def run(lo, hi, qsl, slots, s):
            fn, more = gates(slice(lo, hi))
            return fn(q[lo:hi], k[lo:hi], v[lo:hi], *more, qsl, s, slots, torch.ones_like(slots))

        s_all, s_cut = state.cuda(), state.cuda()
        want = run(0, 51, ints(0, 1, 51), ints(2, 0), s_all)
        parts = [run(0, 1, ints(0, 1), ints(2), s_cut), run(1, 20, ints(0, 19), ints(0), s_cut), run(20, 51, ints(0, 31), ints(0), s_cut)]
        assert torch.equal(torch.cat(parts), want) and torch.equal(s_cut, s_all)


@gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("at", [0, 1, 6, 15, 16, 30])
def test_gdn_tokens_in_front_of_a_bad_one(dtype, bad, at):
    """An infinity or NaN in a token changes no bit of the outputs of those before it, of other columns (a bad value), of other
    heads or of other sequences (a bad key or decay)."""
    from vllm_metax_b200.ops.gdn import gated_delta_rule

    q, k, v, g, beta, qsl, state, idx, has = (t.cuda() for t in _gdn_case(dtype, seed=5, lens=(31, 3, 17)))
    run = lambda k_, v_, g_: gated_delta_rule(q, k_, v_, g_, beta, qsl, state.clone(), idx, has)
    want = run(k, v, g)
    assert bool(torch.isfinite(want).all())
    v2, k2, g2 = v.clone(), k.clone(), g.clone()
    v2[at, 1, 40] = bad
    got = run(k, v2, g)
    assert torch.equal(got[:at], want[:at]) and torch.equal(got[31:], want[31:]) and not bool(torch.isfinite(got[at, 1, 40]))
    others = torch.arange(128, device="cuda") != 40
    assert torch.equal(got[..., others], want[..., others]) and torch.equal(got[:, [0, 2, 3]], want[:, [0, 2, 3]])
    k2[at, 1, 7] = bad
    g2[at, 2] = bad
    for got, same in ((run(k2, v, g), [0, 1]), (run(k, v, g2), [0, 1, 3])):
        assert torch.equal(got[:at], want[:at]) and torch.equal(got[31:], want[31:]) and torch.equal(got[:, same], want[:, same])


@gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens", [(1,) * 90 + (40,), (7, 8, 5, 6) * 20, (3, 0, 5) * 30, (2,) * 4, (5, 6, 7, 8), (1, 1, 1, 26), (8,) * 80,
                                  (0, 33) + (5,) * 80 + (17, 6)])
@pytest.mark.parametrize("known", [False, True])
def test_gdn_short_sequences_beside_long_ones(dtype, lens, known):
    """Sequences of 5 to 8 tokens, around where they change from a token at a time to chunks or groups; few and many of them, alone
    and beside longer ones, with the longest length known or not.  Outputs rounded once, fp32 state within 1e-5."""
    from vllm_metax_b200.ops.gdn import gated_delta_rule

    q, k, v, g, beta, qsl, _, _, _ = _gdn_case(dtype, seed=len(lens), lens=lens)
    gen = torch.Generator().manual_seed(9)
    state = torch.randn(len(lens) + 1, 4, 128, 128, generator=gen) * 0.1
    idx = torch.randperm(len(lens) + 1, generator=gen)[:len(lens)].to(torch.int32)
    has = (torch.rand(len(lens), generator=gen) < 0.7).to(torch.int32)
    want, s_want = _gdn_f64(q, k, v, g, beta, lens, state, idx, has)
    s_got = state.cuda()
    got = gated_delta_rule(*(t.cuda() for t in (q, k, v, g, beta, qsl)), s_got, idx.cuda(), has.cuda(), max_len=max(lens) if known else 0)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    torch.testing.assert_close(got.cpu().double(), want, rtol=eps, atol=1e-5)
    torch.testing.assert_close(s_got.cpu().double(), s_want, rtol=1e-5, atol=1e-5)


@gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,C", [(64, 8192), (65, 8192), (80, 8192), (81, 8192), (160, 4096), (161, 4096), (513, 8192), (1, 8)])
@pytest.mark.parametrize("K", [2, 4])
def test_convolution_around_the_choice_of_kernel(dtype, T, C, K):
    """Steps on either side of where threads take several channels and tokens, sequences of one token and of many, with and without
    a carry: products of 16-bit numbers summed in fp32 in the order of the taps, one rounding (and the silu's exponential)."""
    from vllm_metax_b200.ops import gdn

    g = torch.Generator().manual_seed(T)
    lens = [1] * min(T, 40) + ([T - 40] if T > 40 else [])
    B = len(lens)
    x, w = torch.randn(T, C, generator=g).to(dtype), torch.randn(C, K, generator=g).to(dtype)
    state = torch.randn(B + 1, K - 1, C, generator=g).to(dtype)
    qsl = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    idx, has = torch.randperm(B + 1, generator=g)[:B].to(torch.int32), (torch.rand(B, generator=g) < 0.6).to(torch.int32)
    s1, s2 = state.clone(), state.cuda()
    want = gdn.causal_conv1d_ref(x, w, None, s1, qsl, idx, has)
    got = gdn.causal_conv1d(*(t.cuda() for t in (x, w)), None, s2, qsl.cuda(), idx.cuda(), has.cuda())
    assert torch.equal(s2.cpu(), s1)
    torch.testing.assert_close(got.cpu(), want, rtol=2.0 ** (-7 if dtype == torch.bfloat16 else -9), atol=1e-3)


@gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gdn_of_a_long_prompt(dtype):
    """2048 tokens of one sequence, where errors of the recurrence would add up: outputs rounded once, and the fp32 state within 1e-5
    (its entries decay, so that an error of 2^-24 per token does not grow)."""
    from vllm_metax_b200.ops.gdn import gated_delta_rule

    q, k, v, g, beta, qsl, state, idx, has = _gdn_case(dtype, seed=21, lens=(2048, 1, 700))
    want, s_want = _gdn_f64(q, k, v, g, beta, (2048, 1, 700), state, idx, has)
    s_got = state.cuda()
    got = gated_delta_rule(*(t.cuda() for t in (q, k, v, g, beta, qsl)), s_got, idx.cuda(), has.cuda())
    torch.testing.assert_close(got.cpu().double(), want, rtol=2.0 ** (-8 if dtype == torch.bfloat16 else -11), atol=1e-5)
    torch.testing.assert_close(s_got.cpu().double(), s_want, rtol=1e-5, atol=1e-5)
