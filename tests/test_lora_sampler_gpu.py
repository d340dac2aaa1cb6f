"""GPU numerics of the multi-LoRA, sampler and router kernels against their fp32 PyTorch restatements, plus the
native sampler and a LoRA training step end to end on the device."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def E():
    from twinkle_b200 import ops
    e = ops.ext()
    e.read_and_clear_error()
    yield e
    assert e.read_and_clear_error() == 0


def rel(a, b):
    a, b = a.float(), b.float()
    return float((a - b).norm() / (b.norm() + 1e-12))


def _tiny():
    from twinkle_b200.models import preset
    return preset('qwen3-8b', num_hidden_layers=2, hidden_size=512, intermediate_size=1024, num_attention_heads=4,
                  num_key_value_heads=2, vocab_size=1024)


def test_grouped_gemm_group_map(E):
    torch.manual_seed(1)
    G, N, K = 5, 96, 256
    w = (torch.randn(G, N, K, device='cuda') * 0.1).bfloat16()
    lens = [130, 0, 257, 64, 33]
    gmap = [3, 0, 1, 4, 3]  # segment i multiplies by weight gmap[i]; a weight may serve two segments
    off = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device='cuda')
    x = torch.randn(sum(lens), K, device='cuda').bfloat16()
    y = E.grouped_gemm(x, w, off, 'nt', torch.tensor(gmap, dtype=torch.int32, device='cuda'))
    lo = 0
    for n, g in zip(lens, gmap):
        if n:
            assert rel(y[lo:lo + n], x[lo:lo + n].float() @ w[g].float().t()) < 4e-3
        lo += n


@pytest.mark.parametrize('T', [777, 4096, 40000])     # 40000: segments long enough for the split-K weight gradients
def test_sgmv_forward_backward(E, T):
    from twinkle_b200 import ops
    torch.manual_seed(2)
    S, R, K, N = 4, 32, 512, 384
    a = (torch.randn(S, R, K, device='cuda') * 0.05).bfloat16().requires_grad_(True)
    b = (torch.randn(S, N, R, device='cuda') * 0.05).bfloat16().requires_grad_(True)
    cuts = sorted({0, T} | {int(v) for v in torch.randint(1, T, (4, ))})
    nseg = len(cuts) - 1
    slots = [2, -1, 0, 2, 3][:nseg]
    ranks = [32, 0, 8, 32, 16][:nseg]
    scales = [2.0, 0.0, 0.5, 2.0, 1.0][:nseg]
    dev = dict(device='cuda')
    st = torch.tensor(cuts, dtype=torch.int32, **dev)
    sl = torch.tensor(slots, dtype=torch.int32, **dev)
    rk = torch.tensor(ranks, dtype=torch.int32, **dev)
    sc = torch.tensor(scales, dtype=torch.float32, **dev)
    x = torch.randn(T, K, device='cuda').bfloat16().requires_grad_(True)
    y = ops.sgmv(x, a, b, st, sl, rk, sc)
    g = torch.randn_like(y)
    y.backward(g)

    xr, ar, br = (t.detach().float().requires_grad_(True) for t in (x, a, b))
    yr = ops._sgmv_autograd_cpu(xr, ar, br, st, sl, rk, sc)
    yr.backward(g.float())
    assert rel(y, yr) < 6e-3
    assert rel(x.grad, xr.grad) < 8e-3
    assert rel(a.grad, ar.grad) < 8e-3
    assert rel(b.grad, br.grad) < 8e-3
    # rows of slots nobody used and rank rows beyond a segment's rank get no gradient
    assert float(a.grad[1].abs().max()) == 0.0 and float(b.grad[1].abs().max()) == 0.0


def test_sgmv_into_base_output_with_rank_stacked_pools(E):
    """The form the fused q|k|v projection uses: pools of two projections stacked along the rank axis (block-diagonal
    ``B``), the delta accumulated into the base output in place; against base + per-projection deltas in fp32."""
    import torch.nn.functional as F
    from twinkle_b200 import ops
    torch.manual_seed(5)
    T, S, R, K, n1, n2 = 1500, 3, 16, 256, 384, 128
    a1, a2 = ((torch.randn(S, R, K, device='cuda') * 0.05).bfloat16().requires_grad_(True) for _ in range(2))
    b1 = (torch.randn(S, n1, R, device='cuda') * 0.05).bfloat16().requires_grad_(True)
    b2 = (torch.randn(S, n2, R, device='cuda') * 0.05).bfloat16().requires_grad_(True)
    cuts, slots, ranks, scales = [0, 400, 900, T], [1, -1, 2], [16, 0, 8], [2.0, 0.0, 0.5]
    st = torch.tensor(cuts, dtype=torch.int32, device='cuda')
    sl = torch.tensor(slots, dtype=torch.int32, device='cuda')
    rk = torch.tensor(ranks, dtype=torch.int32, device='cuda')
    sc = torch.tensor(scales, dtype=torch.float32, device='cuda')
    host = [(cuts[i], cuts[i + 1], slots[i], ranks[i], scales[i]) for i in range(3)]
    x = torch.randn(T, K, device='cuda').bfloat16().requires_grad_(True)
    base = torch.randn(T, n1 + n2, device='cuda').bfloat16().requires_grad_(True)
    y0 = base * 1.0                                            # a non-leaf, as the projection's output is
    a = torch.cat([a1, a2], 1)
    b = torch.cat([F.pad(b1, (0, R)), F.pad(b2, (R, 0))], 1)
    y = ops.sgmv(x, a, b, st, sl, rk, sc, host, out=y0, repeat=2)
    assert y.data_ptr() == y0.data_ptr()
    g = torch.randn_like(y)
    y.backward(g)
    xr, a1r, a2r, b1r, b2r, baser = (t.detach().float().requires_grad_(True) for t in (x, a1, a2, b1, b2, base))
    yr = baser + torch.cat([ops._sgmv_autograd_cpu(xr, a1r, b1r, st, sl, rk, sc), ops._sgmv_autograd_cpu(xr, a2r, b2r, st, sl, rk, sc)], 1)
    yr.backward(g.float())
    assert rel(y, yr) < 6e-3 and rel(base.grad, baser.grad) == 0.0
    for got, want in ((x.grad, xr.grad), (a1.grad, a1r.grad), (a2.grad, a2r.grad), (b1.grad, b1r.grad), (b2.grad, b2r.grad)):
        assert rel(got, want) < 8e-3
    assert torch.equal(y[400:900], base.detach()[400:900])      # the segment without an adapter keeps the base rows


def test_paged_decode(E):
    from twinkle_b200 import ops
    torch.manual_seed(3)
    B, Hq, Hkv, D, bs, nblocks = 5, 16, 4, 128, 16, 64
    kc = torch.randn(nblocks, bs, Hkv, D, device='cuda').bfloat16()
    vc = torch.randn(nblocks, bs, Hkv, D, device='cuda').bfloat16()
    lens = torch.tensor([1, 17, 160, 33, 200], dtype=torch.int32, device='cuda')
    perm = torch.randperm(nblocks, device='cuda').int()
    tables = torch.zeros(B, 13, dtype=torch.int32, device='cuda')
    used = 0
    for i in range(B):
        nb = (int(lens[i]) + bs - 1) // bs
        tables[i, :nb] = perm[used:used + nb]
        used += nb
    q = torch.randn(B, Hq, D, device='cuda').bfloat16()
    o = ops.paged_attention_decode(q, kc, vc, tables, lens)
    r = ops.ref.paged_attention_decode(q, kc, vc, tables, lens)
    assert rel(o, r) < 6e-3


@pytest.mark.parametrize('hq,hkv,D,bs,cap', [(32, 8, 128, 16, 8), (16, 1, 128, 16, 256), (40, 4, 64, 8, 700), (12, 3, 64, 24, 40), (8, 1, 128, 1, 600), (6, 2, 64, 24, 40)])
def test_paged_decode_splits(E, hq, hkv, D, bs, cap):
    """Contexts around tile (16), warp and cluster boundaries, tables wide enough for one to eight CTAs per key head, groups of 3 (the vector kernel) to 16 heads."""
    from twinkle_b200 import ops
    torch.manual_seed(hq + D)
    lens = [n for n in (0, 1, 15, 16, 17, 63, 64, 65, 127, 128, 513, 1025, 2000) if n <= bs * cap]
    need = [(n + bs - 1) // bs for n in lens]
    nblocks = sum(need) + 1
    kc, vc = (torch.randn(nblocks, bs, hkv, D, device='cuda').bfloat16() for _ in range(2))
    kc[0], vc[0] = float('nan'), float('nan')                       # nobody's block
    perm, tables, used = (torch.randperm(nblocks - 1) + 1).int(), torch.zeros(len(lens), cap, dtype=torch.int32), 0
    for i, nb in enumerate(need):
        tables[i, :nb] = perm[used:used + nb]
        used += nb
    q = torch.randn(len(lens), hq, D, device='cuda').bfloat16()
    o = ops.paged_attention_decode(q, kc, vc, tables.cuda(), torch.tensor(lens, dtype=torch.int32, device='cuda')).double()
    for i, (n, nb) in enumerate(zip(lens, need)):
        if n == 0:
            assert not o[i].any()
            continue
        at = tables[i, :nb].long().cuda()
        k, v = (c[at].flatten(0, 1)[:n].double().repeat_interleave(hq // hkv, 1) for c in (kc, vc))
        w = torch.softmax(torch.einsum('hd,nhd->hn', q[i].double(), k) * D ** -0.5, -1)
        assert rel(o[i], torch.einsum('hn,nhd->hd', w, v)) < 2.5e-3, n      # rounding of the result to bf16: 2^-9 = 2e-3 at most


def test_router(E):
    from twinkle_b200 import ops
    torch.manual_seed(4)
    for (T, Ex, k, renorm) in [(1000, 128, 8, True), (257, 8, 2, False), (64, 64, 6, True)]:
        lg = torch.randn(T, Ex, device='cuda').bfloat16().requires_grad_(True)
        w, idx, probs, hist = ops.moe_router(lg, k, renorm)
        lr = lg.detach().float().requires_grad_(True)
        wr, ir, pr = ops.ref.moe_router(lr, k, renorm)
        assert torch.equal(idx.sort(-1).values, ir.sort(-1).values)
        order, order_r = idx.argsort(-1), ir.argsort(-1)
        assert torch.allclose(w.gather(-1, order), wr.gather(-1, order_r), atol=1e-5, rtol=1e-4)
        assert torch.allclose(probs, pr, atol=1e-6, rtol=1e-4)
        assert torch.equal(hist.long(), torch.bincount(ir.flatten(), minlength=Ex))
        gw, gp = torch.randn_like(w), torch.randn_like(probs)
        ((w.gather(-1, order) * gw).sum() + (probs * gp).sum()).backward()
        ((wr.gather(-1, order_r) * gw).sum() + (pr * gp).sum()).backward()
        assert rel(lg.grad, lr.grad) < 1e-2  # bf16 gradient storage


def test_sampling(E):
    from twinkle_b200 import ops
    torch.manual_seed(5)
    B, V = 64, 50000
    lg = torch.randn(B, V, device='cuda') * 3
    seeds = torch.arange(B, device='cuda', dtype=torch.int64) + 11
    # greedy
    tok, lp = ops.sample_tokens(lg, 0.0, -1, 1.0, seeds=seeds)
    assert torch.equal(tok, lg.argmax(-1))
    # top-k: every draw inside the k largest, log-prob renormalised over them
    k = 20
    tok, lp = ops.sample_tokens(lg, 0.8, k, 1.0, seeds=seeds)
    topv, topi = (lg / 0.8).topk(k, -1)
    assert bool((topi == tok[:, None]).any(-1).all())
    want = torch.log_softmax(topv, -1).gather(-1, (topi == tok[:, None]).float().argmax(-1, keepdim=True)).squeeze(-1)
    assert torch.allclose(lp, want, atol=2e-3)
    # same seeds → same tokens; other seeds → some differ
    tok2, _ = ops.sample_tokens(lg, 0.8, k, 1.0, seeds=seeds)
    tok3, _ = ops.sample_tokens(lg, 0.8, k, 1.0, seeds=seeds + 1000)
    assert torch.equal(tok, tok2) and not torch.equal(tok, tok3)
    # top-p: draws stay inside the nucleus
    p = 0.5
    tok, lp = ops.sample_tokens(lg, 1.0, -1, p, seeds=seeds)
    probs = torch.softmax(lg, -1)
    sp, si = probs.sort(-1, descending=True)
    inside = (sp.cumsum(-1) - sp) < p
    nucleus = torch.zeros_like(probs, dtype=torch.bool).scatter(-1, si, inside)
    assert bool(nucleus.gather(-1, tok[:, None]).all())
    # the empirical distribution of one row follows softmax (chi-square-free check on the top entries)
    row = torch.randn(1, 32, device='cuda') * 2
    n = 20000
    draws, _ = ops.sample_tokens(row.expand(n, -1).contiguous(), 1.0, -1, 1.0, seeds=torch.arange(n, device='cuda', dtype=torch.int64))
    freq = torch.bincount(draws, minlength=32).float() / n
    assert float((freq - torch.softmax(row[0], -1)).abs().max()) < 0.015


def test_sampler_greedy_matches_full_forward(E):
    """Greedy decode through the paged-KV engine equals argmax of a full-sequence forward at every step."""
    from twinkle_b200.models import build_model, preset
    from twinkle_b200.data_format import SamplingParams
    from twinkle_b200.models.decoder import PackedBatch
    from twinkle_b200.sampler.engine import NativeEngine
    torch.manual_seed(6)
    cfg = _tiny()
    model = build_model(cfg, device='cuda', dtype=torch.bfloat16, seed=0)
    eng = NativeEngine(model, cfg, num_blocks=64, block_size=16)
    prompts = [[5, 9, 33, 2, 17], [7, 7, 100, 42, 3, 1, 250, 11, 90]]
    outs = eng.generate(prompts, [SamplingParams(max_tokens=6, temperature=0.0) for _ in prompts])
    for prompt, resp in zip(prompts, outs):
        toks = list(prompt)
        for t in resp.sequences[0].tokens:
            n = len(toks)
            batch = PackedBatch(torch.tensor(toks, device='cuda'), torch.arange(n, device='cuda'),
                                torch.tensor([0, n], dtype=torch.int32, device='cuda'), n)
            with torch.no_grad():
                logits = model.logits(model(batch))[-1].float()
            top2 = logits.topk(2).values
            if float(top2[0] - top2[1]) > 0.05:  # ties within bf16 noise may legitimately flip
                assert int(logits.argmax()) == t
            toks.append(t)


def test_lora_training_step_on_gpu(E):
    """Two tenants, different ranks, one fused step each: losses fall and the base weights stay untouched."""
    from twinkle_b200.model import LoraConfig, MultiLoraTransformersModel
    torch.manual_seed(7)
    m = MultiLoraTransformersModel(config=_tiny(), device='cuda', max_loras=3, max_r=16)
    base = {k: v.detach().clone() for k, v in m.model.named_parameters() if 'lora' not in k}
    for name, r in (('a', 8), ('b', 16)):
        m.add_adapter_to_model(name, LoraConfig(r=r, lora_alpha=2 * r, target_modules='all-linear'))
        m.set_optimizer('AdamW', lr=5e-3, adapter_name=name)
    g = torch.Generator().manual_seed(0)
    feats = []
    for _ in range(4):
        ids = torch.randint(0, 256, (49, ), generator=g)
        feats.append({'input_ids': ids[:-1].tolist(), 'labels': ids[1:].tolist()})
    first, last = {}, {}
    for it in range(6):
        for name in ('a', 'b'):
            out = m.forward_backward(inputs=feats, adapter_name=name)
            m.clip_grad_and_step(adapter_name=name)
            (first if it == 0 else last)[name] = float(out['loss'])
    for name in ('a', 'b'):
        assert last[name] < first[name] - 0.05, (name, first, last)
    for k, v in m.model.named_parameters():
        if 'lora' not in k:
            assert torch.equal(v, base[k]), k


def _tiny_moe():
    from twinkle_b200.models import preset
    return preset('qwen3-30b-a3b', num_hidden_layers=2, hidden_size=512, num_attention_heads=4, num_key_value_heads=2,
                  vocab_size=1024, num_experts=8, num_experts_per_tok=2, moe_intermediate_size=256)


def test_moe_model_matches_cpu_reference(E):
    """Router kernel + 128-aligned expert layout + grouped tcgen05 GEMMs (fwd, dgrad, per-expert wgrad) vs fp32 CPU."""
    from twinkle_b200.models import PackedBatch, build_model
    cfg = _tiny_moe()
    ref_model = build_model(cfg, device='cpu', dtype=torch.float32, seed=5)
    gpu_model = build_model(cfg, device='cuda', dtype=torch.bfloat16, seed=5)
    with torch.no_grad():
        for (_, p), (_, pc) in zip(gpu_model.named_parameters(), ref_model.named_parameters()):
            p.copy_(pc)
            pc.copy_(p.float().cpu())
    g = torch.Generator().manual_seed(0)
    lens = [150, 106]
    ids = torch.randint(0, cfg.vocab_size, (sum(lens), ), generator=g)
    labels = torch.randint(0, cfg.vocab_size, (sum(lens), ), generator=g)
    pos = torch.cat([torch.arange(n) for n in lens])
    cu = torch.tensor([0, 150, 256], dtype=torch.int32)
    # pin the routing to the CPU model's choice so a bf16 near-tie in the router cannot send a token elsewhere
    ref_model.set_record_routing(True)

    def run(m, dev, routed=None):
        b = PackedBatch(ids.to(dev), pos.to(dev), cu.to(dev), 150, labels.to(dev), routed_experts=routed)
        h = m(b)
        lp, _ = m.token_logprobs(h, b.labels)
        loss = -lp.mean()
        loss.backward()
        ex = m.layers[1].mlp.experts
        return float(loss), ex.down_proj.grad.float().cpu(), ex.gate_up_proj.grad.float().cpu(), m.layers[0].mlp.gate.weight.grad.float().cpu()

    lc, gdc, gguc, ggc = run(ref_model, 'cpu')
    routed = [r.to('cuda') for r in ref_model.collect_routed_experts()]
    lg, gdg, ggug, ggg = run(gpu_model, 'cuda', routed)
    assert abs(lc - lg) < 3e-2, (lc, lg)
    assert rel(gdg, gdc) < 4e-2 and rel(ggug, gguc) < 4e-2 and rel(ggg, ggc) < 6e-2


def test_moe_expert_lora_trains_on_gpu(E):
    from twinkle_b200.model import LoraConfig, MultiLoraTransformersModel
    torch.manual_seed(9)
    m = MultiLoraTransformersModel(config=_tiny_moe(), device='cuda', max_loras=2, max_r=16)
    m.add_adapter_to_model('t', LoraConfig(r=16, lora_alpha=32, target_modules='all-linear'))
    m.set_optimizer('AdamW', lr=5e-3, adapter_name='t')
    g = torch.Generator().manual_seed(0)
    feats = []
    for _ in range(4):
        ids = torch.randint(0, 256, (65, ), generator=g)
        feats.append({'input_ids': ids[:-1].tolist(), 'labels': ids[1:].tolist()})
    losses = []
    for _ in range(6):
        out = m.forward_backward(inputs=feats, adapter_name='t')
        m.clip_grad_and_step(adapter_name='t')
        losses.append(float(out['loss']))
    assert losses[-1] < losses[0] - 0.05, losses
    ex = m.model.layers[0].mlp.experts
    assert float(ex.lora['down_B'][0].abs().max()) > 0  # the expert adapters actually moved


def test_decode_cuda_graph_matches_eager(E):
    """The captured decode step (bucketed batch, static inputs) generates the same greedy tokens and log-probs as the
    eager step, across a batch that shrinks as sequences finish."""
    from twinkle_b200.data_format import SamplingParams
    from twinkle_b200.models import build_model
    from twinkle_b200.sampler.engine import NativeEngine
    cfg = _tiny()
    model = build_model(cfg, device='cuda', dtype=torch.bfloat16, seed=0)
    prompts = [[5, 9, 33, 2, 17], [7, 7, 100, 42, 3, 1, 250, 11, 90], [1, 2, 3]]
    params = [SamplingParams(max_tokens=n, temperature=0.0, logprobs=1) for n in (20, 7, 12)]  # crosses a 16-token block boundary
    outs = {}
    for graphs in (True, False):
        eng = NativeEngine(model, cfg, num_blocks=64, block_size=16)
        eng.use_cuda_graphs = graphs
        res = eng.generate(prompts, params)
        outs[graphs] = [(r.sequences[0].tokens, r.sequences[0].logprobs) for r in res]
        assert bool(eng._graphs) == graphs
    for (t1, l1), (t0, l0) in zip(outs[True], outs[False]):
        assert t1 == t0
        assert max(abs(a - b) for a, b in zip(l1, l0)) < 1e-3


@pytest.mark.parametrize('V', [1, 7, 33, 4099, 32000, 151936, 400001])
@pytest.mark.parametrize('kind', ['flat', 'normal', 'peaked', 'masked'])
def test_sampling_thresholds(E, V, kind):
    """What is kept, from sorted fp64 probabilities, for rows that leave parts of a cluster empty, fill its shared memory, exceed it (400001), whose
    bracket holds everything (flat) or nothing but the largest (peaked), and with tokens ruled out."""
    from twinkle_b200 import ops
    g = torch.Generator(device='cuda').manual_seed(V)
    x = torch.randn(6, V, device='cuda', generator=g)
    if kind == 'flat':
        x *= 1e-3
    elif kind == 'peaked':
        x[:, V // 2] += 60.0
    elif kind == 'masked':
        x *= 3
        x[:, 1:][torch.rand(6, V - 1, device='cuda', generator=g) < 0.7] = float('-inf')
    seeds = torch.arange(6, device='cuda')
    for temp, k, p in [(1.0, -1, 0.9), (0.7, 5, 1.0), (1.0, 50, 0.8), (1.3, -1, 1.0), (1.0, -1, 0.2)]:
        tok, lp = ops.sample_tokens(x, temp, k, p, seeds=seeds)
        prob = torch.softmax(x.double() / temp, -1)
        top, _ = prob.sort(-1, descending=True)
        tau = torch.zeros(6, dtype=torch.float64, device='cuda')
        if 0 < k < V:
            tau = torch.maximum(tau, top[:, k - 1])
        if p < 1:
            tau = torch.maximum(tau, top.gather(1, (top.cumsum(-1) < p).sum(-1, keepdim=True).clamp_max(V - 1))[:, 0])
        mine = prob.gather(1, tok[:, None])[:, 0]
        step = top[:, 0] * 2.0 ** -32 + tau * 1e-5            # resolution of the search, and of fp32 probabilities
        assert (mine >= tau - step).all()
        low, high = (torch.where(prob >= (tau + s * step)[:, None], prob, 0).sum(-1) for s in (1, -1))     # mass kept, but for the tokens at the border
        want = mine.log()
        assert (lp >= want - high.log() - 2e-5).all() and (lp <= want - torch.maximum(low, top[:, 0]).log() + 2e-5).all()
        again, lp2 = ops.sample_tokens(x, temp, k, p, seeds=seeds)
        assert torch.equal(tok, again) and torch.equal(lp, lp2)


@pytest.mark.parametrize('M', [1, 7, 8, 9, 120, 127, 128, 129, 300])
@pytest.mark.parametrize('N,K', [(16, 64), (40, 192), (1000, 320), (1024, 3072), (6144, 1024), (520, 8192), (4096, 12288)])
def test_gemm_few_rows(E, M, N, K):
    """Narrow tiles for few rows: the bits of the wide tiles where K is not split, fp64 to the rounding of sums otherwise; ragged rows and columns,
    strided operands, both result types, accumulation."""
    g = torch.Generator(device='cuda').manual_seed(M * 7 + N)
    x = torch.randn(M, K + 64, device='cuda', generator=g).bfloat16()[:, :K]
    w = torch.randn(N, K, device='cuda', generator=g).bfloat16()
    want = x.double() @ w.double().t()
    for dt in (torch.bfloat16, torch.float32):
        y = E.gemm(x, w, 'nt', None, False, dt)
        E.set_gemm_pair(0)
        wide = E.gemm(x, w, 'nt', None, False, dt)
        E.set_gemm_pair(1)
        if K < 8192:
            assert torch.equal(y, wide)
        # fp32 accumulation of K products of unit variance: K·2^-24 of √K at worst; one rounding to bf16 is 2^-9 of a value
        bound = K * 2.0 ** -24 * K ** 0.5 * 4 + (want.abs() * 2.0 ** -8 if dt == torch.bfloat16 else 0.0)
        assert ((y.double() - want).abs() <= bound).all()
        out = torch.randn(M, N + 8, device='cuda', generator=g).to(dt)
        before, ref = out.clone(), out.clone()
        E.gemm(x, w, 'nt', out[:, :N], True)
        E.set_gemm_pair(0)
        E.gemm(x, w, 'nt', ref[:, :N], True)
        E.set_gemm_pair(1)
        assert torch.equal(out[:, N:], before[:, N:])
        assert torch.equal(out, ref) if K < 8192 else rel(out, ref) < 4e-3
    assert E.read_and_clear_error() == 0


@pytest.mark.parametrize('hq,hkv', [(4, 4), (8, 1), (6, 2), (16, 4), (64, 32)])
@pytest.mark.parametrize('lens,klens', [((1, 63, 64, 65), None), ((127, 128, 129), None), ((300, 1, 515), None), ((1024, ), None), ((5, 130, 1), (260, 130, 129))])
@pytest.mark.parametrize('causal', [True, False])
def test_flash_backward_tiles(E, hq, hkv, lens, klens, causal):
    """Gradients around tile edges (128), for heads that are and are not shared out over a cluster (groups of 1, 3, 4, 8; few and many tiles), keys that
    are longer than their queries."""
    from twinkle_b200 import ops
    g = torch.Generator(device='cuda').manual_seed(hq + sum(lens))
    klens = klens or lens
    D, T, Tk = 128, sum(lens), sum(klens)
    q, k, v, do = (torch.randn(n, h, D, device='cuda', generator=g).bfloat16() for n, h in ((T, hq), (Tk, hkv), (Tk, hkv), (T, hq)))
    cu, cuk = (torch.tensor([0] + list(x), device='cuda').cumsum(0).int() for x in (lens, klens))
    leaves = [t.clone().requires_grad_() for t in (q, k, v)]
    o = ops.flash_attn_varlen(*leaves, cu, max(lens), causal=causal, cu_seqlens_k=cuk, max_seqlen_k=max(klens))
    got = torch.autograd.grad(o, leaves, do)
    ref = [t.double().requires_grad_() for t in (q, k, v)]
    outs, a, b = [], 0, 0
    for n, m in zip(lens, klens):
        kk, vv = (t[b:b + m].repeat_interleave(hq // hkv, 1) for t in ref[1:])
        s = torch.einsum('qhd,khd->hqk', ref[0][a:a + n], kk) * D ** -0.5
        if causal:
            s = s.masked_fill(torch.ones(n, m, dtype=torch.bool, device='cuda').triu(m - n + 1), float('-inf'))
        outs.append(torch.einsum('hqk,khd->qhd', torch.softmax(s, -1), vv))
        a, b = a + n, b + m
    want = torch.autograd.grad(torch.cat(outs), ref, do.double())
    for x, y in zip(got, want):
        assert rel(x, y) < 8e-3        # P and dS rounded to bf16 (2^-9 each at most) and the result too
    assert E.read_and_clear_error() == 0


@pytest.mark.parametrize('d,e', [(128, 128), (64, 64), (40, 128), (104, 24)])
@pytest.mark.parametrize('lens,klens', [((1, 127, 128, 129), None), ((255, 256, 257, 1, 700), None), ((3, 130, 300), (3, 400, 301)), ((400, 260), (100, 300))])
@pytest.mark.parametrize('window,chunk', [(0, 0), (70, 0), (0, 200), (300, 0)])
def test_flash_forward_pairs(E, d, e, lens, klens, window, chunk):
    """Sequences that end in the first or second tile of a pair, keys longer and shorter than their queries, bounds that leave a tile's first blocks unseen."""
    g = torch.Generator(device='cuda').manual_seed(d + sum(lens))
    klens, hq, hkv = klens or lens, 6, 2
    q, k, v = (torch.randn(n, h, w, device='cuda', generator=g).bfloat16() for n, h, w in ((sum(lens), hq, d), (sum(klens), hkv, d), (sum(klens), hkv, e)))
    cu, cuk = (torch.tensor([0] + list(x), device='cuda').cumsum(0).int() for x in (lens, klens))
    o, lse = E.flash_attn_fwd(q, k, v, cu, max(lens), True, d ** -0.5, cuk, None, None, window, chunk)
    a = b = 0
    for n, m in zip(lens, klens):
        kk, vv = (t[b:b + m].double().repeat_interleave(hq // hkv, 1) for t in (k, v))
        s = torch.einsum('qhd,khd->hqk', q[a:a + n].double(), kk) * d ** -0.5
        i, j = torch.arange(n, device='cuda')[:, None] + m - n, torch.arange(m, device='cuda')[None]
        seen = j <= i
        if window:
            seen &= j > i - window
        if chunk:
            seen &= j >= i // chunk * chunk
        live = seen.any(-1)                        # a query without keys has no defined result
        s = s.masked_fill(~seen, float('-inf'))
        want = torch.einsum('hqk,khe->qhe', torch.softmax(s, -1), vv)
        if live.any():
            assert rel(o[a:a + n][live], want[live]) < 6e-3            # weights and results rounded to bf16
            assert (lse[:, a:a + n][:, live].double() - torch.logsumexp(s[:, live], -1)).abs().max() < 5e-3
        a, b = a + n, b + m
    assert E.read_and_clear_error() == 0


@pytest.mark.parametrize('dtype,hkv,d,e', [(torch.bfloat16, 8, 128, 128), (torch.bfloat16, 1, 24, 40), (torch.float32, 3, 64, 4), (torch.bfloat16, 1, 4, 3)])
@pytest.mark.parametrize('lens', [(1, ), (16, 1, 17), (300, 37, 111)])
def test_cache_write_places(E, dtype, hkv, d, e, lens):
    """Rows of prompts land where their block lists say and nowhere else: whole vectors, narrow rows (the general path), views with a pitch of their own."""
    from twinkle_b200 import ops
    bs, T = 16, sum(lens)
    need = [(n + bs - 1) // bs for n in lens]
    perm = (torch.randperm(sum(need)) + 1).tolist()
    blocks = [[perm.pop() for _ in range(n)] for n in need]
    rows = E.prompt_rows(blocks, list(lens), bs, True).cuda()
    kp, vp = (torch.zeros(sum(need) + 2, bs, hkv, w, device='cuda', dtype=dtype) for w in (d, e))
    both = torch.randn(T, hkv * (d + e) + 8, device='cuda').to(dtype)
    k, v = both[:, :hkv * d].view(T, hkv, d), both[:, hkv * d:hkv * (d + e)].view(T, hkv, e)
    ops.cache_write(kp, vp, rows, k, v)
    want_k, want_v, at = torch.zeros_like(kp), torch.zeros_like(vp), 0
    for n, b in zip(lens, blocks):
        for t in range(n):
            want_k[b[t // bs], t % bs], want_v[b[t // bs], t % bs] = k[at + t], v[at + t]
        at += n
    assert torch.equal(kp, want_k) and torch.equal(vp, want_v)
    out = torch.full((4 * (5 + 2), ), -1, dtype=torch.int32)
    E.pack_step(out, 4, 5, [[7, 8, 9], [3]], [40, 2], [1, 2])
    assert out.tolist() == [7, 8, 9, 0, 0, 3, 0, 0, 0, 0] + [0] * 10 + [40, 2, 0, 0] + [1, 2, 0, 0]


@pytest.mark.parametrize('H', [1024, 2048, 4096, 1032])
@pytest.mark.parametrize('rows', [1, 2, 147, 297, 1500])
def test_rmsnorm_rows_in_registers(E, H, rows):
    """Widths with and without a kernel that keeps its rows, few rows and many, with a residual and without."""
    x, r, w = torch.randn(rows, H, device='cuda').bfloat16(), torch.randn(rows, H, device='cuda').bfloat16(), torch.randn(H, device='cuda').bfloat16()
    for res in (None, r):
        got = E.rmsnorm_fwd(x, w, 1e-6, 0.5, res)
        h = x if res is None else (x.float() + r.float()).bfloat16()
        rstd = torch.rsqrt(h.double().pow(2).mean(-1) + 1e-6)
        assert rel(got[1], rstd) < 4e-6                       # fp32 sums
        assert rel(got[0], h.double() * rstd[:, None] * (w.double() + 0.5)) < 2.0 ** -8
        if res is not None:
            assert torch.equal(got[2], h)


@pytest.mark.parametrize('lens,klens', [((130, 300), (0, 40)), ((5, 400), (5, 100)), ((0, 200, 3), (300, 200, 0)), ((260, 129), (30, 0))])
@pytest.mark.parametrize('causal', [True, False])
@pytest.mark.parametrize('hq,hkv', [(8, 1), (64, 32)])
def test_flash_tiles_without_keys(E, lens, klens, causal, hq, hkv):
    """Query tiles that see no key and key tiles that no query sees: zeros, and −inf for the log-sum-exp, as for such rows of other tiles."""
    from twinkle_b200 import ops
    g = torch.Generator(device='cuda').manual_seed(sum(lens))
    q, k, v, do = (torch.randn(n, h, 128, device='cuda', generator=g).bfloat16() for n, h in ((sum(lens), hq), (sum(klens), hkv), (sum(klens), hkv), (sum(lens), hq)))
    cu, cuk = (torch.tensor([0] + list(x), device='cuda').cumsum(0).int() for x in (lens, klens))
    leaves = [t.clone().requires_grad_() for t in (q, k, v)]
    o, lse = ops.flash_attn_varlen(*leaves, cu, max(lens), causal=causal, cu_seqlens_k=cuk, max_seqlen_k=max(klens), return_lse=True)
    got = torch.autograd.grad(o, leaves, do)
    ref = [t.double().requires_grad_() for t in (q, k, v)]
    want, dead, a, b = torch.zeros_like(ref[0]), torch.ones(sum(lens), dtype=torch.bool, device='cuda'), 0, 0
    for n, m in zip(lens, klens):
        first = max(0, n - m) if causal else 0                # rows before it see nothing
        if m and first < n:
            kk, vv = (t[b:b + m].repeat_interleave(hq // hkv, 1) for t in ref[1:])
            s = torch.einsum('qhd,khd->hqk', ref[0][a + first:a + n], kk) * 128 ** -0.5
            if causal:
                s = s.masked_fill(torch.ones(n - first, m, dtype=torch.bool, device='cuda').triu(m - n + first + 1), float('-inf'))
            want = want.index_add(0, torch.arange(a + first, a + n, device='cuda'), torch.einsum('hqk,khd->qhd', torch.softmax(s, -1), vv))
            dead[a + first:a + n] = False
        a, b = a + n, b + m
    assert not o[dead].any() and (lse[:, dead] == float('-inf')).all() and lse[:, ~dead].isfinite().all()
    assert not got[0][dead].any()
    for x, y in zip((o, *got), (want, *torch.autograd.grad(want, ref, do.double()))):
        assert rel(x, y) < 8e-3        # P and dS rounded to bf16 (2^-9 each at most) and the result too
    # keys of three chunks: one query tile per CTA
    q, k, v = (torch.randn(n, h, w, device='cuda', generator=g).bfloat16() for n, h, w in ((sum(lens), hq, 192), (sum(klens), hkv, 192), (sum(klens), hkv, 64)))
    o, lse = E.flash_attn_fwd(q, k, v, cu, max(lens), causal, 192 ** -0.5, cuk)
    assert not o[dead].any() and (lse[:, dead] == float('-inf')).all() and o.isfinite().all() and o[~dead].any()
    sinks = torch.randn(hq, device='cuda', generator=g).bfloat16()
    for w in (128, 192):
        q, k, v = (torch.randn(n, h, w, device='cuda', generator=g).bfloat16() for n, h in ((sum(lens), hq), (sum(klens), hkv), (sum(klens), hkv)))
        o, lse = E.flash_attn_fwd(q, k, v[..., :128].contiguous(), cu, max(lens), causal, w ** -0.5, cuk, sinks)
        assert not o[dead].any() and torch.equal(lse[:, dead], sinks.float()[:, None].expand(-1, int(dead.sum())))
    assert E.read_and_clear_error() == 0


def test_cache_rows_outside_the_pool_are_an_error(E):
    """Rows outside the pools are not written, the others are, and generation raises instead of going on without those keys."""
    from twinkle_b200 import ops
    from twinkle_b200.data_format import SamplingParams
    from twinkle_b200.models import build_model
    from twinkle_b200.sampler.engine import NativeEngine
    assert E.read_and_clear_error() == 0
    k, v = (torch.randn(4, 2, 64, device='cuda').bfloat16() for _ in range(2))
    for bad in (-1, 48, 2**40):
        kp, vp = (torch.zeros(3, 16, 2, 64, device='cuda', dtype=torch.bfloat16) for _ in range(2))
        ops.cache_write(kp, vp, torch.tensor([5, bad, 0, 47], device='cuda'), k, v)
        assert E.read_and_clear_error() == 7
        for p, x in ((kp, k), (vp, v)):
            want = torch.zeros_like(p).view(48, 2, 64)
            want[[5, 0, 47]] = x[[0, 2, 3]]
            assert torch.equal(p.view(48, 2, 64), want)
    cfg = _tiny()
    eng = NativeEngine(build_model(cfg, device='cuda', dtype=torch.bfloat16, seed=0), cfg, num_blocks=64, block_size=16)
    places = eng._prompt_rows
    eng._prompt_rows = lambda seqs, lens: places(seqs, lens) + 64 * 16
    with pytest.raises(RuntimeError, match='error 7'):
        eng.generate([[1, 2, 3]], [SamplingParams(max_tokens=2, temperature=0.0)])
    eng._prompt_rows = places
    assert len(eng.generate([[1, 2, 3]], [SamplingParams(max_tokens=2, temperature=0.0)])[0].sequences[0].tokens) == 2
    assert E.read_and_clear_error() == 0


def _hashes(seed, n):
    """The 32-bit hash behind the Gumbel noise of tokens 0 … n of a row."""
    import numpy as np
    with np.errstate(over='ignore'):
        x = np.uint64(seed) * np.uint64(0x9E3779B97F4A7C15) + np.arange(n, dtype=np.uint64)
        for m in (0xff51afd7ed558ccd, 0xc4ceb9fe1a85ec53):
            x = (x ^ (x >> np.uint64(33))) * np.uint64(m)
        return (x ^ (x >> np.uint64(33))).astype(np.uint32)


def test_sampling_hash_that_rounds_to_one(E):
    """A token whose uniform number rounds to 1 gets a large but finite score: it loses to tokens of e^30 times its weight, and wins among equals."""
    from twinkle_b200 import ops
    V = 151936
    seed, at = next((s, int(h.argmax())) for s, h in ((s, _hashes(s, V)) for s in range(4000)) if h.max() >= 2**32 - 128)
    x = torch.zeros(1, V, device='cuda')
    seeds = torch.tensor([seed], device='cuda')
    assert int(ops.sample_tokens(x, 1.0, -1, 1.0, seeds=seeds)[0]) == at          # ln 2^26 = 18 of the others' 12 at most, as a rule
    x[0, at] = -30.0
    tok, lp = ops.sample_tokens(x, 1.0, -1, 1.0, seeds=seeds)
    assert int(tok) != at and abs(float(lp) + math.log(V)) < 1e-4


def test_sampling_leaves_out_no_winner_near_one(E):
    """Two tokens of one warp with u within 2^-17 of 1, where the error of the fast logarithm makes e / E larger than the exact bound e / (1 − u): the later one
    wins by a little, and must not be passed over because of the earlier one."""
    import numpy as np

    from twinkle_b200 import ops
    V, found = 8192, []
    for seed in range(60000):
        h = _hashes(seed, V)
        near = np.nonzero(h >= 2**32 - 200 * 256)[0]
        for a in near:
            for b in near:
                # steps of 2^-24 below 1; the same warp (512 threads per round), a later round
                ka, kb = (2**24 - int(np.float32(h[i]) / 256) for i in (a, b))
                if b // 512 > a // 512 and b % 512 // 32 == a % 512 // 32 and kb >= 2 * ka and ka >= 8:
                    found.append((seed, int(a), int(b), ka, kb))
        if len(found) >= 2:
            break
    assert len(found) >= 2
    for seed, a, b, ka, kb in found:
        # e_b / e_a between E_b / E_a as the exact logarithm has it and 0.999 (1 − u_b) / E_a with the fast one's E_a, about 0.8 steps less
        ratio = kb / (ka - 0.8) * (1 - 0.4 / kb)
        x = torch.full((1, V), -100.0, device='cuda')
        x[0, a], x[0, b] = 0.0, math.log(ratio)
        assert int(ops.sample_tokens(x, 1.0, -1, 1.0, seeds=torch.tensor([seed], device='cuda'))[0]) == b, (seed, a, b, ka, kb)


@pytest.mark.parametrize('V', [32, 1000, 8192, 20001, 60000, 151936, 400001])
@pytest.mark.parametrize('rows', [3, 300])
@pytest.mark.parametrize('how', [(1.0, -1, 1.0), (0.7, 50, 1.0), (1.0, -1, 0.9)])
def test_sampling_draws_the_largest_score(E, V, rows, how):
    """The drawn token has the largest of logit / T + Gumbel noise among those kept, recomputed in fp64 from the hash, for one to eight CTAs per row, in shared
    memory and beyond it.  Scores are uncertain by what __logf leaves: 2^-21 of E = −ln u."""
    import numpy as np

    from twinkle_b200 import ops
    if rows == 300 and V > 200000:
        rows = 40
    temp, k, p = how
    g = torch.Generator(device='cuda').manual_seed(V + rows)
    x = torch.randn(rows, V, device='cuda', generator=g) * 2
    seeds = torch.arange(rows, device='cuda') * 7919 + V
    tok, _ = ops.sample_tokens(x, temp, k, p, seeds=seeds)
    some = sorted(set(range(0, rows, max(1, rows // 12))))
    wins = 0
    for r in some:
        h = torch.from_numpy(_hashes(int(seeds[r]), V).astype(np.int64)).cuda()
        u = (h.float() + 0.5) * 2.0 ** -32
        en = torch.where(u < 1, -torch.log(u.double()), 2.0 ** -26)
        blur = torch.where(u < 1, -torch.log1p(-(2.0 ** -21 / en).clamp_max(1 - 1e-9)), 0) + 1e-4
        prob = torch.softmax(x[r].double() / temp, -1)
        top = prob.sort(descending=True)[0]
        tau = top[k - 1] if 0 < k < V else top[(top.cumsum(-1) < p).sum().clamp_max(V - 1)] if p < 1 else torch.zeros((), device='cuda', dtype=torch.float64)
        score = x[r].double() / temp - torch.log(en)
        sure = (prob >= tau * (1 + 1e-4) + top[0] * 2.0 ** -31) | (prob == top[0])
        t = int(tok[r])
        assert prob[t] >= tau * (1 - 1e-4) - top[0] * 2.0 ** -31
        assert float(score[t] + blur[t]) >= float((score - blur)[sure].max()), r
        wins += t == int(torch.where(sure, score, -torch.inf).argmax())
    assert wins >= len(some) - 1          # the blur decides next to nothing
    # a row is cut differently in a batch and alone
    one = torch.cat([ops.sample_tokens(x[r:r + 1], temp, -1, 1.0, seeds=seeds[r:r + 1])[0] for r in some])
    assert torch.equal(one, ops.sample_tokens(x, temp, -1, 1.0, seeds=seeds)[0][some])


def test_sampling_frequencies_over_a_wide_row(E):
    """Tokens in every CTA of a cluster and many per lane: drawn as often as their probabilities say."""
    from twinkle_b200 import ops
    V, n = 151936, 20000
    live = torch.linspace(3, V - 5, 24, device='cuda').long()
    weight = torch.arange(1, 25, device='cuda').double()
    x = torch.full((V, ), -60.0, device='cuda')
    x[live] = weight.log().float()
    got = torch.cat([ops.sample_tokens(x.expand(500, V).contiguous(), 1.0, -1, 0.999, seeds=torch.arange(i, i + 500, device='cuda'))[0] for i in range(0, n, 500)])
    count = (got[:, None] == live).sum(0).double()
    want = weight / weight.sum() * n
    assert int(count.sum()) == n
    assert float(((count - want) ** 2 / want).sum()) < 23 + 5 * (2 * 23) ** 0.5         # chi-squared of 23 degrees: mean 23, variance 46


@pytest.mark.parametrize('hq,hkv,d', [(32, 8, 128), (16, 4, 64), (16, 8, 128)])
@pytest.mark.parametrize('n', [5, 100, 1500])
def test_paged_decode_of_infinite_values(E, hq, hkv, d, n):
    """An infinite value among the visible ones is the result in its dimension, of either sign; two of opposite signs make NaN; other dimensions are as without it."""
    from twinkle_b200 import ops
    g = torch.Generator(device='cuda').manual_seed(n)
    blocks = (n + 15) // 16 + 1
    kc, vc = (torch.randn(blocks, 16, hkv, d, device='cuda', generator=g).bfloat16() for _ in range(2))
    q = torch.randn(1, hq, d, device='cuda', generator=g).bfloat16()
    table, lens = torch.arange(blocks, device='cuda').int()[None], torch.tensor([n], device='cuda').int()
    plain = ops.paged_attention_decode(q, kc, vc, table, lens)
    rows, last = vc.view(-1, hkv, d), blocks * 16 - 1
    rows[n // 2, :, 3], rows[n - 1, :, 10], rows[0, :, 20], rows[n - 1, :, 20], rows[last, :, 30] = math.inf, -math.inf, math.inf, -math.inf, math.nan
    o = ops.paged_attention_decode(q, kc, vc, table, lens)
    assert (o[..., 3] == math.inf).all() and (o[..., 10] == -math.inf).all() and o[..., 20].isnan().all()
    rest = [i for i in range(d) if i not in (3, 10, 20)]
    assert torch.equal(o[..., rest], plain[..., rest])


@pytest.mark.parametrize('window,chunk,at', [(70, 0, 200), (1, 0, 300), (0, 128, 300), (0, 384, 383), (130, 0, 120)])
@pytest.mark.parametrize('d,e', [(128, 128), (64, 40)])
@pytest.mark.parametrize('lens', [(512, ), (300, 509)])
def test_flash_forward_values_before_a_tile(E, window, chunk, at, d, e, lens):
    """Values that are not finite in a key block before everything that a query tile sees leave its rows as they are, also when the tile's neighbour sees the block."""
    g = torch.Generator(device='cuda').manual_seed(at)
    T, n = sum(lens), lens[-1]
    q, k, v = (torch.randn(T, h, w, device='cuda', generator=g).bfloat16() for h, w in ((6, d), (2, d), (2, e)))
    cu = torch.tensor([0] + list(lens), device='cuda').cumsum(0).int()
    run = lambda v: E.flash_attn_fwd(q, k, v, cu, max(lens), True, d ** -0.5, None, None, None, window, chunk)  # noqa: E731
    plain, lse = run(v)
    bad = v.clone()
    bad[T - n + at, :, 0], bad[T - n + at, :, 1] = math.inf, math.nan
    o, lse2 = run(bad)
    tile = next(t for t in range(0, n, 128) if (t - window + 1 if window else t // chunk * chunk) // 128 > at // 128)       # the first that sees later blocks only
    assert torch.equal(o[T - n + tile:], plain[T - n + tile:]) and torch.equal(lse, lse2)
    seen = slice(T - n + at, T - n + at + 1)
    assert (o[seen, :, 0] == math.inf).all() and o[seen, :, 1].isnan().all()
    assert E.read_and_clear_error() == 0


@pytest.mark.parametrize('H', [256, 768, 1536, 2560, 3072, 3584, 4864, 5120, 5376])
@pytest.mark.parametrize('rows', [1, 149, 2400])
def test_rmsnorm_of_any_multiple_of_256(E, H, rows):
    """Every width whose rows fit registers, and the first beyond them."""
    test_rmsnorm_rows_in_registers(E, H, rows)
