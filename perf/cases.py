"""Workloads of the framework's main path, small enough to be measured one pass at a time on one GPU.

A post-training job alternates between two things, and these cases follow them: training steps (packed rows of documents of uneven length,
forward and backward, full-parameter and LoRA on experts) and generation (prompts through the paged engine, one-token steps over a batch of
sequences, the choice of tokens).  Layers have the widths of the presets ``qwen3-0.6b``, ``qwen3-8b`` and ``qwen3-30b-a3b``; stacks are cut to a
few layers and the vocabulary with them, so that the output head keeps the share that it has in the whole model.

``attend``   packed causal attention with its gradients (``ops.flash_attn_varlen``), the part of a training step that grows with the documents
``sft``      forward and backward of a dense model through ``TransformersModel.forward_backward``: log-probs, loss and fp32 gradients
``experts``  the same for LoRA adapters on a mixture-of-experts model with the routing replayed from the sampler, as in policy training
``prefill``  prompts through ``NativeEngine.prefill`` into an empty paged cache, and the logits of their last tokens
``decode``   one token for every sequence through ``NativeEngine.decode_step``, contexts of uneven length in scattered pages
``sample``   tokens and their log-probs from a batch of logits (``ops.sample_tokens``)

``exact`` restates all but the last (whose draws come from the framework's own random stream) in plain fp64 torch.
"""
from __future__ import annotations

import math
import random
import zlib

import torch

EPS, THETA = 1e-6, 1e6
#: hidden, feed-forward, query heads, key heads (all 128 wide), tied output head; experts: number, chosen per token, width
MODELS = {
    'qwen3-0.6b': dict(h=1024, i=3072, hq=16, hkv=8, tied=True),
    'qwen3-8b': dict(h=4096, i=12288, hq=32, hkv=8, tied=False),
    'qwen3-30b-a3b': dict(h=2048, i=768, hq=32, hkv=4, tied=False, experts=128, top=8),
}
D, RANK, SCALE, AUX, BLOCK = 128, 16, 2.0, 1e-3, 16


def _documents(total, lo, hi, rng):
    """Lengths uniform in [lo, hi] that fill ``total`` tokens; the last one is cut."""
    out = []
    while sum(out) < total:
        out.append(min(rng.randint(lo, hi), total - sum(out)))
    return ','.join(map(str, out))


def listed():
    rng = random.Random(2024)
    return [
        # two short chat turns in one row: a handful of launches, none of which fills the chip
        {'name': 'attend-short', 'kind': 'attend', 'lengths': '700,324', 'heads': 32, 'kv_heads': 8},
        # one packed row of the long-document SFT configuration
        {'name': 'attend-documents', 'kind': 'attend', 'lengths': _documents(32768, 512, 8192, rng), 'heads': 32, 'kv_heads': 8},
        # the micro-batch of the expert LoRA configuration: full rows, groups of eight query heads
        {'name': 'attend-rows', 'kind': 'attend', 'lengths': ','.join(['4096'] * 8), 'heads': 32, 'kv_heads': 4},
        # full-parameter SFT on a packed row
        {'name': 'sft-documents', 'kind': 'sft', 'model': 'qwen3-8b', 'layers': 2, 'vocab': 8192, 'lengths': _documents(16384, 512, 8192, rng)},
        # expert LoRA on two rows with replayed routing
        {'name': 'experts-rows', 'kind': 'experts', 'model': 'qwen3-30b-a3b', 'layers': 2, 'vocab': 8192, 'lengths': '4096,4096'},
        # a few interactive prompts on a small model
        {'name': 'prefill-short', 'kind': 'prefill', 'model': 'qwen3-0.6b', 'layers': 28, 'vocab': 151936, 'lengths': '37,300,111'},
        # rollout prompts of one length in one go
        {'name': 'prefill-rows', 'kind': 'prefill', 'model': 'qwen3-8b', 'layers': 4, 'vocab': 8192, 'lengths': ','.join(['1024'] * 8)},
        # one user waiting for one token
        {'name': 'decode-one', 'kind': 'decode', 'model': 'qwen3-0.6b', 'layers': 28, 'vocab': 151936, 'sequences': 1, 'context': 1024},
        # an ordinary batch
        {'name': 'decode-batch', 'kind': 'decode', 'model': 'qwen3-8b', 'layers': 4, 'vocab': 8192, 'sequences': 64, 'context': 1024},
        # a few long contexts: the cache outweighs the weights
        {'name': 'decode-long', 'kind': 'decode', 'model': 'qwen3-8b', 'layers': 4, 'vocab': 8192, 'sequences': 16, 'context': 8192},
        # rollouts of a group-relative policy step: as many sequences as the engine takes
        {'name': 'decode-rollout', 'kind': 'decode', 'model': 'qwen3-8b', 'layers': 4, 'vocab': 8192, 'sequences': 256, 'context': 1280},
        # tokens of a batch under nucleus sampling
        {'name': 'sample-nucleus', 'kind': 'sample', 'rows': 64, 'vocab': 151936, 'temperature': 1.0, 'top_k': -1, 'top_p': 0.95},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['attend', 'sft', 'experts', 'prefill', 'decode', 'decode', 'sample'])
    if kind == 'attend':
        total = _log(rng, 256, 32768)
        heads = rng.choice([(32, 8), (32, 4), (16, 8), (64, 8)])
        if heads[0] == 64:
            total = min(total, 16384)
        hi = min(8192, max(64, total // rng.randint(1, 4)))
        return {'kind': kind, 'lengths': _documents(total, max(1, hi // 16), hi, rng), 'heads': heads[0], 'kv_heads': heads[1]}
    if kind == 'sft':
        model, total = rng.choice(['qwen3-0.6b', 'qwen3-8b']), _log(rng, 512, 16384)
        hi = min(8192, max(64, total // rng.randint(1, 4)))
        return {'kind': kind, 'model': model, 'layers': 2, 'vocab': 8192, 'lengths': _documents(total, max(8, hi // 16), hi, rng)}
    if kind == 'experts':
        total = _log(rng, 512, 8192)
        return {'kind': kind, 'model': 'qwen3-30b-a3b', 'layers': 2, 'vocab': 8192, 'lengths': _documents(total, max(8, total // 8), min(4096, total), rng)}
    if kind == 'prefill':
        if rng.random() < 0.4:
            model, layers, vocab, total = 'qwen3-0.6b', 28, 151936, _log(rng, 16, 2048)
        else:
            model, layers, vocab, total = 'qwen3-8b', 4, 8192, _log(rng, 64, 16384)
        hi = max(16, total // rng.randint(1, 6))
        return {'kind': kind, 'model': model, 'layers': layers, 'vocab': vocab, 'lengths': _documents(total, max(1, hi // 8), hi, rng)}
    if kind == 'decode':
        if rng.random() < 0.3:
            model, layers, vocab, n = 'qwen3-0.6b', 28, 151936, _log(rng, 1, 16)
            context = _log(rng, 32, 2048)
        else:
            model, layers, vocab, n = 'qwen3-8b', 4, 8192, _log(rng, 1, 256)
            context = _log(rng, 64, min(16384, 327680 // n))
        return {'kind': kind, 'model': model, 'layers': layers, 'vocab': vocab, 'sequences': n, 'context': context}
    return {'kind': kind, 'rows': _log(rng, 1, 256), 'vocab': rng.choice([32000, 151936, 128256]), 'temperature': rng.choice([0.7, 1.0]),
            'top_k': rng.choice([-1, -1, 20, 50]), 'top_p': rng.choice([0.8, 0.95, 1.0])}


# ------------------------------------------------------------------- inputs
def _lengths(case):
    if case['kind'] != 'decode':
        return [int(x) for x in case['lengths'].split(',')]
    rng = random.Random(case['sequences'] * 100003 + case['context'])        # contexts of uneven length, at most ``context`` tokens
    return [rng.randint(max(1, case['context'] // 2), case['context']) for _ in range(case['sequences'])]


def _gen(seed, name):
    return torch.Generator(device='cuda').manual_seed((zlib.crc32(name.encode()) << 20) + int(seed) % (1 << 20))


def _normal(shape, std, seed, name, mean=0.0):
    return torch.empty(shape, dtype=torch.bfloat16, device='cuda').normal_(mean, std, generator=_gen(seed, name))


def _weights(case, seed):
    """Weights by the names of the framework's modules, drawn one by one."""
    m, V = MODELS[case['model']], case['vocab']
    h, i, q, kv = m['h'], m['i'], m['hq'] * D, m['hkv'] * D
    yield 'embed_tokens.weight', _normal((V, h), 0.02, seed, 'embed')
    for n in range(case['layers']):
        at = f'layers.{n}.'
        for name, shape in (('input_layernorm', h), ('post_attention_layernorm', h), ('self_attn.q_norm', D), ('self_attn.k_norm', D)):
            yield at + name + '.weight', _normal((shape, ), 0.1, seed, at + name, 1.0)
        yield at + 'self_attn.qkv_proj.weight', _normal((q + 2 * kv, h), 0.02, seed, at + 'qkv')
        yield at + 'self_attn.o_proj.weight', _normal((h, q), 0.02, seed, at + 'o')
        if 'experts' in m:
            yield at + 'mlp.gate.weight', _normal((m['experts'], h), 0.02, seed, at + 'gate')
            yield at + 'mlp.experts.gate_up_proj', _normal((m['experts'], 2 * i, h), 0.02, seed, at + 'gu')
            yield at + 'mlp.experts.down_proj', _normal((m['experts'], h, i), 0.02, seed, at + 'down')
        else:
            yield at + 'mlp.gate_up_proj.weight', _normal((2 * i, h), 0.02, seed, at + 'gu')
            yield at + 'mlp.down_proj.weight', _normal((h, i), 0.02, seed, at + 'down')
    yield 'norm.weight', _normal((h, ), 0.1, seed, 'norm', 1.0)
    if not m['tied']:
        yield 'lm_head.weight', _normal((V, h), 0.02, seed, 'head')


def _adapters(case, seed):
    """The LoRA pool ``[1 adapter, …]`` of an adapter that has been trained for a while (B is not zero any more)."""
    m = MODELS[case['model']]
    h, i, E = m['h'], m['i'], m['experts']
    for n in range(case['layers']):
        at = f'layers.{n}.'
        for lin, inp, parts in (('self_attn.qkv_proj', h, (('q_proj', m['hq'] * D), ('k_proj', m['hkv'] * D), ('v_proj', m['hkv'] * D))),
                                ('self_attn.o_proj', m['hq'] * D, (('o_proj', h), ))):
            for p, out in parts:
                yield f'{at}{lin}.lora_A.{p}', _normal((1, RANK, inp), inp ** -0.5, seed, at + p + 'A')
                yield f'{at}{lin}.lora_B.{p}', _normal((1, out, RANK), 0.02, seed, at + p + 'B')
        for p, inp, out in (('gate_up', h, 2 * i), ('down', i, h)):
            yield f'{at}mlp.experts.lora.{p}_A', _normal((1, E, RANK, inp), inp ** -0.5, seed, at + p + 'A')
            yield f'{at}mlp.experts.lora.{p}_B', _normal((1, E, out, RANK), 0.02, seed, at + p + 'B')


def _rows(case, seed):
    """Token ids, positions and labels (the next token; none at the end of a document) of every document."""
    g, out = _gen(seed, 'ids'), []
    for n in _lengths(case):
        ids = torch.randint(0, case['vocab'], (n, ), device='cuda', generator=g)
        labels = torch.roll(ids, -1)
        labels[-1] = -100
        out.append({'input_ids': ids, 'labels': labels, 'position_ids': torch.arange(n, device='cuda')})
    return out


def _routes(case, seed):
    """Experts of every token, per layer ``[T, 8]``: near-uniform load, none twice."""
    m, T = MODELS[case['model']], sum(_lengths(case))
    return [torch.rand(T, m['experts'], device='cuda', generator=_gen(seed, f'routes{n}')).topk(m['top'], -1)[1] for n in range(case['layers'])]


def _qkv(case, seed):
    T, hq, hkv = sum(_lengths(case)), case['heads'], case['kv_heads']
    return [_normal((T, n, D), 1.0, seed, x) for n, x in ((hq, 'q'), (hkv, 'k'), (hkv, 'v'), (hq, 'do'))]


def _pages(case):
    """Block tables as continuous batching leaves them: pages of a sequence lie anywhere.  Block 0 belongs to nobody."""
    need = [(n + BLOCK) // BLOCK for n in _lengths(case)]      # the context and the token of this step
    free = list(range(1, sum(need) + 1))
    random.Random(sum(need)).shuffle(free)
    out, at = [], 0
    for n in need:
        out.append(free[at:at + n])
        at += n
    return out, len(free) + 1


def _caches(case, seed, blocks):
    hkv = MODELS[case['model']]['hkv']
    for n in range(case['layers']):
        yield _normal((blocks, BLOCK, hkv, D), 1.0, seed, f'k{n}'), _normal((blocks, BLOCK, hkv, D), 1.0, seed, f'v{n}')


def _logits(case, seed):
    """A broad background and a few tokens far above it."""
    shape, g = (case['rows'], case['vocab']), _gen(seed, 'logits')
    x = torch.empty(shape, device='cuda').normal_(0.0, 2.0, generator=g)
    return x + 10.0 * torch.rand(shape, device='cuda', generator=g).pow_(4000.0)


def _decoder(case, seed):
    from twinkle_b200.models.config import preset
    from twinkle_b200.models.decoder import build_model
    cfg = preset(case['model'], num_hidden_layers=case['layers'], vocab_size=case['vocab'])
    model = build_model(cfg, device='cuda', dtype=torch.bfloat16, init=False)
    model.requires_grad_(False)
    params = dict(model.named_parameters())
    for name, w in _weights(case, seed):
        params[name].copy_(w)
    return model, cfg


def prepare(case, seed):
    kind = case['kind']
    if kind == 'attend':
        q, k, v, do = _qkv(case, seed)
        lens = _lengths(case)
        cu = torch.tensor([0] + lens, device='cuda').cumsum(0).to(torch.int32)
        return {'kind': kind, 'q': q.requires_grad_(), 'k': k.requires_grad_(), 'v': v.requires_grad_(), 'do': do, 'cu': cu, 'longest': max(lens)}
    if kind == 'sample':
        seeds = torch.randint(0, 2**62, (case['rows'], ), device='cuda', generator=_gen(seed, 'seeds'))
        return {'kind': kind, 'logits': _logits(case, seed), 'seeds': seeds, 'how': (case['temperature'], case['top_k'], case['top_p'])}
    if kind in ('sft', 'experts'):
        from twinkle_b200.model import LoraConfig, TransformersModel
        from twinkle_b200.models.config import preset
        from twinkle_b200.utils.device_mesh import DeviceMesh
        cfg = preset(case['model'], num_hidden_layers=case['layers'], vocab_size=case['vocab'])
        lora = kind == 'experts'
        # the seed only feeds the start values, which are replaced below
        model = TransformersModel(config=cfg, device_mesh=DeviceMesh.from_sizes(dp_size=1), seed=0, grad_dtype='fp32', device='cuda:0',
                                  **({'max_loras': 1, 'max_r': RANK} if lora else {}))
        if lora:
            model.add_adapter_to_model('sft', LoraConfig(r=RANK, lora_alpha=int(SCALE * RANK), target_modules='all-linear'))
        params = dict(model.model.named_parameters())
        with torch.no_grad():
            for name, w in _weights(case, seed):
                params[name].copy_(w)
            for name, w in (_adapters(case, seed) if lora else ()):
                params[name].copy_(w)
        rows = _rows(case, seed)
        if lora:
            routes, at = _routes(case, seed), 0
            for r in rows:
                n = r['input_ids'].numel()
                r['routed_experts'] = [x[at:at + n] for x in routes]
                at += n
        return {'kind': kind, 'model': model, 'rows': rows, 'adapter': {'adapter_name': 'sft'} if lora else {}}
    from twinkle_b200.data_format import SamplingParams
    from twinkle_b200.sampler.engine import NativeEngine, _Seq
    model, cfg = _decoder(case, seed)
    lens = _lengths(case)
    ids = [t.tolist() for t in torch.randint(0, case['vocab'], (sum(lens), ), device='cuda', generator=_gen(seed, 'ids')).split(lens)]
    seqs = [_Seq(0, x, SamplingParams(max_tokens=0)) for x in ids]
    if kind == 'prefill':
        blocks = 1 + sum((n + BLOCK) // BLOCK for n in lens)
        engine = NativeEngine(model, cfg, torch.device('cuda'), num_blocks=blocks, block_size=BLOCK, max_batch=len(seqs))
        return {'kind': kind, 'engine': engine, 'seqs': seqs, 'ends': torch.tensor(lens, device='cuda').cumsum(0) - 1}
    tables, blocks = _pages(case)
    engine = NativeEngine(model, cfg, torch.device('cuda'), num_blocks=blocks, block_size=BLOCK, max_batch=len(seqs))
    for n, (k, v) in enumerate(_caches(case, seed, blocks)):
        engine.cache.k[n].copy_(k)
        engine.cache.v[n].copy_(v)
    last = torch.randint(0, case['vocab'], (len(seqs), ), device='cuda', generator=_gen(seed, 'last'))
    for s, t, token in zip(seqs, tables, last.tolist()):
        s.blocks = t
        s.tokens.append(token)
    engine.decode_step(seqs, last)          # a running engine has its step captured
    return {'kind': kind, 'engine': engine, 'seqs': seqs, 'last': last, 'k': [c[1:] for c in engine.cache.k], 'v': [c[1:] for c in engine.cache.v]}


def run(state):
    kind = state['kind']
    if kind == 'attend':
        from twinkle_b200 import ops
        q, k, v = state['q'], state['k'], state['v']
        o = ops.flash_attn_varlen(q, k, v, state['cu'], state['longest'])
        dq, dk, dv = torch.autograd.grad(o, (q, k, v), state['do'])
        return {'o': o.detach(), 'dq': dq, 'dk': dk, 'dv': dv}
    if kind == 'sample':
        from twinkle_b200 import ops
        tokens, logprobs = ops.sample_tokens(state['logits'], *state['how'], seeds=state['seeds'])
        return {'tokens': tokens, 'logprobs': logprobs}
    if kind in ('sft', 'experts'):
        model, extra = state['model'], state['adapter']
        model.zero_grad(**extra)
        out = model.forward_backward(inputs=state['rows'], **extra)
        got = {'loss': float(out['loss']), 'logps': out['logps'].detach()}
        if extra:
            got.update({n: p.grad for n, p in model.engine.replicated if p.grad is not None})
        else:
            for b in model.engine.trainable_buckets():
                got.update({n: b.grad_shard[o:o + math.prod(s)].view(s) for n, o, s in zip(b.names, b.offsets, b.shapes)})
        return got
    engine = state['engine']
    if kind == 'decode':        # block 0 belongs to nobody: what rows that fill up a batch write there is no result
        return {'logits': engine.decode_step(state['seqs'], state['last']), 'k': state['k'], 'v': state['v']}
    with torch.no_grad():
        hidden = engine.prefill(state['seqs'])
        logits = engine.model.logits(hidden[state['ends']]).float()
        engine.release(state['seqs'])
    return {'hidden': hidden, 'logits': logits, 'k': engine.cache.k, 'v': engine.cache.v}


# ------------------------------------------------------- what a pass cannot do without
def _layer_sizes(case):
    """(parameters that every token meets, those that lie in memory) of one layer."""
    m = MODELS[case['model']]
    attn = m['h'] * D * (2 * m['hq'] + 2 * m['hkv'])
    if 'experts' in m:
        return attn + m['h'] * m['experts'] + m['top'] * 3 * m['h'] * m['i'], attn + m['h'] * m['experts'] + m['experts'] * 3 * m['h'] * m['i']
    return attn + 3 * m['h'] * m['i'], attn + 3 * m['h'] * m['i']


def work(case):
    kind = case['kind']
    if kind == 'sample':
        return {'bytes': 4 * case['rows'] * case['vocab'] + 16 * case['rows'], 'flops': 5 * case['rows'] * case['vocab']}
    lens = _lengths(case)
    T, pairs = sum(lens), sum(n * (n + 1) // 2 for n in lens)
    if kind == 'attend':     # two products forward, five backward
        hq, hkv = case['heads'], case['kv_heads']
        return {'bytes': 2 * D * T * (4 * hq + 4 * hkv), 'flops': 14 * D * hq * pairs}
    m, L = MODELS[case['model']], case['layers']
    active, held = _layer_sizes(case)
    head = case['vocab'] * m['h']
    if kind == 'decode':
        B = case['sequences']
        cache = 4 * (T + B) * m['hkv'] * D
        return {'bytes': 2 * (L * held + head) + L * cache + 4 * B * case['vocab'], 'flops': 2 * B * (L * active + head) + 4 * L * m['hq'] * D * (T + B)}
    if kind == 'prefill':
        return {'bytes': 2 * (L * held + head) + 4 * L * T * m['hkv'] * D + 2 * T * m['h'] + 4 * len(lens) * case['vocab'],
                'flops': 2 * T * L * active + 2 * len(lens) * head + 4 * L * m['hq'] * D * pairs}
    attention = 14 * L * m['hq'] * D * pairs
    if kind == 'experts':    # gradients with respect to inputs and adapters
        adapters = sum(w.numel() for w in _adapter_sizes(case))
        return {'bytes': 2 * (L * held + head) + 4 * adapters + 24 * T, 'flops': 4 * T * (L * active + head) + attention}
    params = L * held + head * (1 if m['tied'] else 2)
    return {'bytes': 6 * params + 24 * T, 'flops': 6 * T * (L * active + head) + attention}


def _adapter_sizes(case):
    m = MODELS[case['model']]
    h, i, E, q, kv = m['h'], m['i'], m['experts'], m['hq'] * D, m['hkv'] * D
    per = RANK * ((h + q) + 2 * (h + kv) + (q + h) + E * (h + 2 * i) + E * (i + h))
    return [torch.empty(per, device='meta') for _ in range(case['layers'])]


def tolerance(case):
    """Measured as the distance from 64 bits, times about four; never over what 16-bit operands explain."""
    kind = case['kind']
    if kind == 'sample':
        return {'rel': 1e-5, 'max': 1e-4}        # fp32 sums; tokens stay the same
    if kind == 'attend':
        return {'rel': 0.015, 'max': 0.5}
    return {'rel': 0.03, 'max': 0.6}


# ----------------------------------------------------------------- 64 bits
def _rms(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w


def _rope(x, pos):
    f = THETA ** (-torch.arange(0, D, 2, device=x.device, dtype=torch.float64) / D)
    a = pos.double()[:, None, None] * f
    c, s, x1, x2 = a.cos(), a.sin(), x[..., :D // 2], x[..., D // 2:]
    return torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1)


def _causal(q, k, v):
    """One document, the query heads of one key head: ``q [G, L, D]``, ``k, v [L, D]``."""
    n = k.shape[0]
    s = (q @ k.t()) * D ** -0.5
    s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device=k.device).triu_(1), -math.inf)
    return torch.softmax(s, -1) @ v


def _attend(q, k, v, lens):
    """``q [T, Hq, D]``, ``k, v [T, Hkv, D]`` → ``[T, Hq, D]``; documents and key heads one at a time, recomputed for gradients."""
    from torch.utils.checkpoint import checkpoint
    G, rows, at = q.shape[1] // k.shape[1], [], 0
    for n in lens:
        heads = []
        for h in range(k.shape[1]):
            for g in range(0, G, 4):       # at most four query heads: a score matrix of 8192² fp64 is half a gigabyte
                a = q[at:at + n, h * G + g:h * G + min(g + 4, G)].transpose(0, 1), k[at:at + n, h], v[at:at + n, h]
                heads.append(checkpoint(_causal, *a, use_reentrant=False) if q.requires_grad else _causal(*a))
        rows.append(torch.cat(heads).transpose(0, 1))
        at += n
    return torch.cat(rows)


def _experts64(x, W, LP, at, w, idx):
    out = torch.zeros_like(x)
    gu, down = W[at + 'mlp.experts.gate_up_proj'], W[at + 'mlp.experts.down_proj']
    lo = [LP[f'{at}mlp.experts.lora.{p}'][0] for p in ('gate_up_A', 'gate_up_B', 'down_A', 'down_B')]
    for e in range(gu.shape[0]):
        t, j = (idx == e).nonzero(as_tuple=True)
        if not t.numel():
            continue
        u = x[t]
        y = u @ gu[e].double().t() + SCALE * (u @ lo[0][e].t()) @ lo[1][e].t()
        a, b = y.chunk(2, -1)
        a = torch.nn.functional.silu(a) * b
        y = a @ down[e].double().t() + SCALE * (a @ lo[2][e].t()) @ lo[3][e].t()
        out = out.index_add(0, t, y * w[t, j, None])
    return out


def _stack64(case, W, ids, pos, attend, routes=None, LP=None):
    """Embedding, layers and final norm.  ``attend(layer, q, k, v)`` gives the heads' outputs; returns hidden rows and the balance terms."""
    m, auxes = MODELS[case['model']], []
    hq, hkv, T = m['hq'], m['hkv'], ids.numel()

    def lin(x, at, name, parts):
        y = x @ W[f'{at}{name}.weight'].double().t()
        if LP is not None:
            y = y + SCALE * torch.cat([(x @ LP[f'{at}{name}.lora_A.{p}'][0].t()) @ LP[f'{at}{name}.lora_B.{p}'][0].t() for p in parts], -1)
        return y

    x = torch.nn.functional.embedding(ids, W['embed_tokens.weight'].double())
    for n in range(case['layers']):
        at = f'layers.{n}.'
        qkv = lin(_rms(x, W[at + 'input_layernorm.weight'].double()), at, 'self_attn.qkv_proj', ('q_proj', 'k_proj', 'v_proj')).view(T, hq + 2 * hkv, D)
        q = _rope(_rms(qkv[:, :hq], W[at + 'self_attn.q_norm.weight'].double()), pos)
        k = _rope(_rms(qkv[:, hq:hq + hkv], W[at + 'self_attn.k_norm.weight'].double()), pos)
        x = x + lin(attend(n, q, k, qkv[:, hq + hkv:]).reshape(T, hq * D), at, 'self_attn.o_proj', ('o_proj', ))
        y = _rms(x, W[at + 'post_attention_layernorm.weight'].double())
        if routes is None:
            a, b = (y @ W[at + 'mlp.gate_up_proj.weight'].double().t()).chunk(2, -1)
            x = x + (torch.nn.functional.silu(a) * b) @ W[at + 'mlp.down_proj.weight'].double().t()
        else:
            probs = torch.softmax(y @ W[at + 'mlp.gate.weight'].double().t(), -1)
            w = probs.gather(1, routes[n])
            share = torch.bincount(routes[n].reshape(-1), minlength=m['experts']).double() / routes[n].numel()
            auxes.append(m['experts'] * (share * probs.mean(0)).sum())
            x = x + _experts64(y, W, LP, at, w / w.sum(-1, keepdim=True), routes[n])
    return _rms(x, W['norm.weight'].double()), auxes


def exact(case, seed):
    kind = case['kind']
    if kind == 'sample':
        return None
    lens = _lengths(case)
    if kind == 'attend':
        q, k, v, do = (t.double() for t in _qkv(case, seed))
        for t in (q, k, v):
            t.requires_grad_()
        o = _attend(q, k, v, lens)
        dq, dk, dv = torch.autograd.grad(o, (q, k, v), do)
        return {'o': o.detach(), 'dq': dq, 'dk': dk, 'dv': dv}
    W = dict(_weights(case, seed))
    head = W['embed_tokens.weight' if MODELS[case['model']]['tied'] else 'lm_head.weight']
    if kind in ('sft', 'experts'):
        rows = _rows(case, seed)
        ids, pos, labels = (torch.cat([r[x] for r in rows]) for x in ('input_ids', 'position_ids', 'labels'))
        LP = routes = None
        if kind == 'experts':
            LP = {n: w.double().requires_grad_() for n, w in _adapters(case, seed)}
            routes, leaves = _routes(case, seed), LP
        else:
            leaves = W = {n: w.double().requires_grad_() for n, w in W.items()}
            head = W['embed_tokens.weight' if MODELS[case['model']]['tied'] else 'lm_head.weight']
        hidden, aux = _stack64(case, W, ids, pos, lambda n, q, k, v: _attend(q, k, v, lens), routes, LP)
        logps = torch.log_softmax(hidden @ head.double().t(), -1).gather(1, labels.clamp_min(0)[:, None])[:, 0]
        live = labels >= 0
        ce, n = -(logps * live).sum(), int(live.sum())
        loss = ce + (AUX * n * torch.stack(aux).mean() if aux else 0.0)
        grads = torch.autograd.grad(loss, list(leaves.values()))
        padded = torch.zeros(len(lens), max(lens), dtype=torch.float64, device='cuda')
        for i, x in enumerate(logps.detach().split(lens)):
            padded[i, :len(x)] = x
        return {'loss': float(loss) / n, 'logps': padded, **dict(zip(leaves, grads))}
    if kind == 'prefill':
        ids = torch.randint(0, case['vocab'], (sum(lens), ), device='cuda', generator=_gen(seed, 'ids'))
        pos = torch.cat([torch.arange(n, device='cuda') for n in lens])
        hkv, blocks = MODELS[case['model']]['hkv'], 1 + sum((n + BLOCK) // BLOCK for n in lens)
        first, starts = 1, []             # an empty cache hands its pages out in order
        for n in lens:
            starts.append(first * BLOCK)
            first += (n + BLOCK) // BLOCK
        rows = torch.cat([torch.arange(s, s + n, device='cuda') for s, n in zip(starts, lens)])
        ks, vs = [], []

        def attend(n, q, k, v):
            for out, x in ((ks, k), (vs, v)):
                pool = torch.zeros(blocks * BLOCK, hkv, D, device='cuda')
                pool[rows] = x.float()
                out.append(pool.view(blocks, BLOCK, hkv, D))
            return _attend(q, k, v, lens)

        hidden, _ = _stack64(case, W, ids, pos, attend)
        ends = torch.tensor(lens, device='cuda').cumsum(0) - 1
        return {'hidden': hidden, 'logits': hidden[ends] @ head.double().t(), 'k': ks, 'v': vs}
    tables, blocks = _pages(case)
    caches = [(k.double(), v.double()) for k, v in _caches(case, seed, blocks)]
    last = torch.randint(0, case['vocab'], (len(lens), ), device='cuda', generator=_gen(seed, 'last'))
    pos = torch.tensor(lens, device='cuda')

    def step(n, q, k, v):
        out = []
        for b, (t, length) in enumerate(zip(tables, lens)):
            at = torch.tensor(t, device='cuda')
            K, V = (c[at].flatten(0, 1) for c in caches[n])
            K[length], V[length] = k[b], v[b]
            for pool, x in zip(caches[n], (k[b], v[b])):
                pool[t[length // BLOCK], length % BLOCK] = x
            K, V = K[:length + 1].transpose(0, 1), V[:length + 1].transpose(0, 1)           # [Hkv, n, D]
            s = torch.softmax(q[b].view(K.shape[0], -1, D) @ K.transpose(1, 2) * D ** -0.5, -1)
            out.append((s @ V).reshape(-1, D))
        return torch.stack(out)

    hidden, _ = _stack64(case, W, last, pos, step)
    return {'logits': hidden @ head.double().t(), 'k': [k[1:] for k, _ in caches], 'v': [v[1:] for _, v in caches]}
