"""The work this package does for its callers, as a list of cases that a timing program can prepare, run and compare.

Every case goes through the public entry points in the order a caller uses them: ``cache.update`` -> attention ->
``cache.post_update`` for a prompt, a segment of a prompt or a token; the attention layer's ``forward``; the training
forward with its row statistics; the decode step with static launch parameters, recorded once and replayed.

Kinds of cases (``case["kind"]``):

* ``prefill``    a prompt: role-masked attention and the eviction that compacts its K/V into the cache
* ``forward``    ``nats_chunk_attention_fwd``: attention plus the two per-row statistics the training forward saves
* ``segments``   one prompt handed over in several calls, each over the compacted cache of the ones before
* ``layer``      ``LlamaNAtSChunkAttentionLayer.forward`` on a prompt: projections, role head, RoPE, attention, eviction
* ``layer_step`` the same layer on one new token per sequence, behind a prompt
* ``step``       one decode step on a layer cache: append + attention, and the placement of a completed chunk
* ``generate``   a prompt, then decode steps recorded in one CUDA graph and replayed

Roles are drawn independently per (sequence, kv-head, chunk); the first chunk is global, as the layers of this package
force it, and an unfinished last chunk is passed as global.
"""
import math

import numpy as np
import torch

from neuralattentionsearch_b200 import LlamaNAtSChunkAttentionLayer, NAtSCache, NAtSChunkLayerCache, prefill_attention
from neuralattentionsearch_b200.functional import nats_chunk_attention_fwd

DEVICE = 'cuda'
GLOBAL, LOCAL, SLIDING = 0, 1, 2


def _shape(kind, B, Hq, Hkv, D, N, C, SW, pg, pl, **more):
    return dict(kind=kind, B=B, Hq=Hq, Hkv=Hkv, D=D, N=N, C=C, SW=SW, p_global=pg, p_local=pl, **more)


def listed():
    return [
        # a short prompt of a small multi-head model in fp32: launches and host work count
        dict(_shape('prefill', 1, 8, 8, 64, 2048, 64, 256, 0.10, 0.30, dtype='float32'), name='prefill_2k_mha_fp32'),
        # a batch of prompts of a GQA 32/8 decoder whose length is no multiple of a chunk or of a tile
        dict(_shape('prefill', 8, 32, 8, 128, 15001, 128, 1024, 0.07, 0.20, dtype='bfloat16'), name='prefill_15001_batch8'),
        # the benchmark's prompt: 32k tokens, one sequence
        dict(_shape('prefill', 1, 32, 8, 128, 32768, 128, 1024, 0.05, 0.15, dtype='bfloat16'), name='prefill_32k'),
        # the long-context configuration: two sequences of 131k tokens with a wide window
        dict(_shape('prefill', 2, 32, 8, 128, 131072, 128, 4096, 0.02, 0.08, dtype='bfloat16'), name='prefill_131k_batch2'),
        # one role per token (the default granularity of NAtSCache)
        dict(_shape('prefill', 1, 32, 8, 128, 8192, 1, 256, 0.10, 0.30, dtype='bfloat16'), name='prefill_8k_token_roles'),
        # a training micro-batch with the chunk size of the layer cache's default
        dict(_shape('forward', 8, 16, 8, 64, 4096, 16, 256, 0.10, 0.30), name='forward_4k_batch8'),
        # a prompt that arrives in four segments (chunked prefill, turns of a conversation), three of them ragged
        dict(_shape('segments', 1, 32, 8, 128, 24576, 128, 1024, 0.05, 0.15, n_segments=4, ragged=True), name='segments_24k'),
        # the attention layer of a 4096-wide decoder on a prompt, and on one token behind a prompt (latency of one sequence)
        dict(_shape('layer', 1, 32, 8, 128, 16384, 128, 1024, 0.05, 0.15), name='layer_16k'),
        dict(_shape('layer_step', 1, 32, 8, 128, 8000, 128, 1024, 0.05, 0.15), name='layer_step_batch1'),
        # decode over the compacted cache of 32k tokens, 2k to 6k of them retained per (sequence, kv-head)
        dict(_shape('step', 64, 32, 8, 128, 32768 + 127, 128, 1024, 0.0625, 0.0, p_global_hi=0.1875), name='step_batch64'),
        # the same with one role per token: every step places its token
        dict(_shape('step', 16, 16, 4, 64, 16384, 1, 512, 0.0625, 0.15, p_global_hi=0.1875), name='step_batch16_token_roles'),
        # a reply of a small batch from a recorded step: latency of the decode kernels
        dict(_shape('generate', 2, 32, 8, 128, 6000, 128, 1024, 0.10, 0.20, n_replays=12), name='generate_batch2_graph'),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(case):
    """Seconds a pass takes at a large card's rates if every query looked at half of the keys of a fine-grained prompt (whole
    tiles are read there), plus what every pass costs; only compared with the largest listed case."""
    w = work(case)
    flops = w['flops']
    if case['kind'] in ('prefill', 'forward', 'segments', 'layer') and case['C'] < 128:
        flops = max(flops, 2.0 * case['B'] * case['Hq'] * float(case['N']) ** 2 * case['D'])
    return flops / 1e15 + w['bytes'] / 6e12


def draw(rng):
    largest = max(_cost(c) for c in listed())
    while True:
        case = _draw(rng)
        if _cost(case) <= 0.9 * largest:
            return case


def _draw(rng):
    kind = rng.choice(['prefill', 'prefill', 'prefill', 'forward', 'segments', 'layer', 'layer_step', 'step', 'step', 'generate'])
    D = rng.choice([64, 128, 128, 128])
    Hkv = rng.choice([2, 4, 8, 8])
    Hq = Hkv * rng.choice([2, 4, 4, 8])
    C = rng.choice([1, 16, 32, 64, 128, 128, 128])
    SW = C * max(1, _log_uniform(rng, 128, 4096) // C)
    pg, pl = rng.uniform(0.02, 0.12), rng.uniform(0.08, 0.30)
    long = {1: 16384, 16: 32768, 32: 49152}.get(C, 131072)
    if kind == 'prefill':
        dtype = rng.choice(['bfloat16', 'bfloat16', 'bfloat16', 'float32'])
        N = _log_uniform(rng, 300, long)
        B = min(16, max(1, _log_uniform(rng, 1, 131072) // N))
        if B * Hkv * N <= 128 * 128 and rng.random() < 0.5:
            Hq = Hkv                                                    # multi-head attention, in the small models that use it
        if B * Hq * N <= 128 * 128 and rng.random() < 0.5:
            D = 256
        return _shape(kind, B, Hq, Hkv, D, N, C, SW, pg, pl, dtype=dtype)
    if kind == 'forward':
        N = _log_uniform(rng, 500, 8192)
        return _shape(kind, rng.randint(1, 8), Hq, Hkv, D, N, C, min(SW, C * max(1, 1024 // C)), pg, pl)
    if kind == 'segments':
        N = _log_uniform(rng, 4096, min(long, 65536))
        return _shape(kind, rng.choice([1, 1, 2]), Hq, Hkv, D, N, C, SW, pg, pl, n_segments=rng.randint(2, 6), ragged=rng.random() < 0.7)
    if kind in ('layer', 'layer_step'):
        Hkv = rng.choice([4, 8])
        # a role per token needs a different scale of the role head than the pooled ones below
        C = rng.choice([32, 64, 128])
        SW = C * max(1, _log_uniform(rng, 256, 2048) // C)
        N = _log_uniform(rng, 600, 16384) if kind == 'layer' else _log_uniform(rng, 2 * C, 16384)
        B = rng.choice([1, 1, 2, 4]) if kind == 'layer' else rng.choice([1, 2, 4, 16])
        return _shape(kind, B, Hkv * rng.choice([2, 4]), Hkv, D, N, C, SW, pg, pl)
    if kind == 'step':
        N = _log_uniform(rng, 2000, 32768)
        B = min(96, _log_uniform(rng, 1, 96))
        return _shape(kind, B, Hq, Hkv, D, N, C, min(SW, C * max(1, 1024 // C)), pg, pl, p_global_hi=rng.uniform(0.12, 0.25))
    N = _log_uniform(rng, 1500, 16384)
    return _shape('generate', rng.choice([1, 2, 4, 8]), Hq, Hkv, D, N, C, min(SW, C * max(1, 1024 // C)), pg, pl, n_replays=rng.randint(4, 16))


# ---------------------------------------------------------------------------------------------------- preparation
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _randn(g, *shape, dtype=torch.bfloat16, sigma=0.5):
    return torch.randn(*shape, generator=g, device=DEVICE, dtype=dtype).mul_(sigma)


def _prompt_roles(g, case, last_is_global=True):
    """uint8 [B,Hkv,ceil(N/C)].  With p_global_hi the share of global chunks of a (sequence, kv-head) is uniform in
    [p_global, p_global_hi], which makes the compacted caches ragged.  How many tokens every head keeps is drawn once per
    case; the seed decides which (sequence, kv-head) it is and the order of its chunks up to its last global one, so that
    the compacted caches of all seeds have the same extent."""
    B, H, N, C = case['B'], case['Hkv'], case['N'], case['C']
    n = -(-N // C)
    once = _generator(7)
    u = torch.rand(B * H, n, generator=once, device=DEVICE)
    lo, hi = case['p_global'], case.get('p_global_hi', case['p_global'])
    pg = lo + (hi - lo) * torch.rand(B * H, 1, generator=once, device=DEVICE)
    roles = torch.where(u < pg, GLOBAL, torch.where(u < pg + case['p_local'], LOCAL, SLIDING)).to(torch.uint8)
    roles[:, 0] = GLOBAL
    index = torch.arange(n, device=DEVICE)
    last_global = torch.where((roles == GLOBAL) & (index < N // C), index, 0).amax(1, keepdim=True)
    key = torch.rand(B * H, n, generator=g, device=DEVICE)
    key = torch.where(index >= last_global, 1.0 + index, key)
    key[:, 0] = -1.0
    roles = roles.gather(1, key.argsort(1))[torch.randperm(B * H, generator=g, device=DEVICE)]
    if N % C and last_is_global:
        roles[:, -1] = GLOBAL
    return roles.view(B, H, n).contiguous()


def _token_roles(g, case, p_global, p_local):
    """uint8 [B,Hkv,1]: the role of a chunk that new tokens complete"""
    u = torch.rand(case['B'], case['Hkv'], 1, generator=g, device=DEVICE)
    return torch.where(u < p_global, GLOBAL, torch.where(u < p_global + p_local, LOCAL, SLIDING)).to(torch.uint8)


def _qkv(g, case, n, dtype=torch.bfloat16):
    B, D = case['B'], case['D']
    return tuple(_randn(g, B, h, n, D, dtype=dtype) for h in (case['Hq'], case['Hkv'], case['Hkv']))


def _segment_lengths(case):
    n, k, C = case['N'], case['n_segments'], case['C']
    if not case['ragged']:
        base = max(n // k // C * C, C)
        return [base] * (k - 1) + [n - base * (k - 1)]
    cuts = [0] + [int(n * (i + 0.37 * (-1) ** i) / k) for i in range(1, k)] + [n]
    return [b - a for a, b in zip(cuts, cuts[1:])]


def _rope(D, start, n):
    pos = torch.arange(start, start + n, device=DEVICE, dtype=torch.float32)
    inv = 500000.0 ** (-torch.arange(0, D, 2, device=DEVICE, dtype=torch.float32) / D)
    angle = (pos[:, None] * inv)[None].repeat(1, 1, 2)
    return angle.cos().to(torch.bfloat16), angle.sin().to(torch.bfloat16)


def _hidden(g, case, n):
    x = _randn(g, case['B'], n, case['Hq'] * case['D'], sigma=1.0)
    x[..., 0] = 1.0                              # carries the biases of the role head, see _layer
    return x


def _layer(case, seed):
    dim = case['Hq'] * case['D']
    torch.manual_seed(seed)
    with torch.device(DEVICE):
        layer = LlamaNAtSChunkAttentionLayer(dim=dim, n_heads=case['Hq'], n_kv_heads=case['Hkv'], chunk_size=case['C'],
                                             local_seq_max_length=case['SW']).to(torch.bfloat16).eval()
    with torch.no_grad():
        # role logits of roughly unit variance over pooled hidden states, with biases for the wanted mix (few global, some
        # local, most sliding); the role head has no bias term, so they ride on the constant feature 0
        layer.proj_layer.weight.normal_(0, math.sqrt(case['C'] / dim))
        w = layer.proj_layer.weight.view(case['Hkv'], 3, dim)
        w[:, 0, 0], w[:, 1, 0], w[:, 2, 0] = -2.0, -1.25, 0.0
    return layer


def _step_inputs(g, case, n):
    B, D = case['B'], case['D']
    return [(_randn(g, B, case['Hq'], 1, D), _randn(g, B, case['Hkv'], 1, D), _randn(g, B, case['Hkv'], 1, D)) for _ in range(n)]


@torch.no_grad()
def prepare(case, seed):
    g = _generator(seed)
    kind, C, N = case['kind'], case['C'], case['N']
    state = dict(case=case)
    if kind in ('prefill', 'forward'):
        state['q'], state['k'], state['v'] = _qkv(g, case, N, getattr(torch, case.get('dtype', 'bfloat16')))
        roles = _prompt_roles(g, case)
        if kind == 'forward':                    # what the training code has in hand: one-hot samples
            state['info'] = torch.nn.functional.one_hot(roles.long(), 3).to(torch.bfloat16)
        else:
            state['roles'] = roles
    elif kind == 'segments':
        roles = _prompt_roles(g, case, last_is_global=False)
        state['segments'], pos = [], 0
        for n in _segment_lengths(case):
            # a call describes its chunks from the unfinished one on; its own unfinished last chunk counts as global
            r = roles[..., pos // C:-(-(pos + n) // C)].clone()
            pos += n
            if pos % C:
                r[..., -1] = GLOBAL
            state['segments'].append((*_qkv(g, case, n), r))
    elif kind == 'layer':
        state['layer'] = _layer(case, seed)
        state['x'] = _hidden(g, case, N)
        state['rope'] = _rope(case['D'], 0, N)
    elif kind == 'layer_step':
        layer = state['layer'] = _layer(case, seed)
        state['cache'] = NAtSCache(case['SW'], C)
        n = N // C * C + C - 1                   # the first token completes a chunk
        layer(_hidden(g, case, n), _rope(case['D'], 0, n), None, 0, state['cache'])
        state['x'] = [_hidden(g, case, 1) for _ in range(4)]
        state['rope'] = _rope(case['D'], n, 1)
        state['pos'] = n
    elif kind == 'step':
        n = N // C * C + C - 1
        k, v = (_randn(g, case['B'], case['Hkv'], n, case['D']) for _ in range(2))
        roles = _prompt_roles(g, dict(case, N=n))
        cache = state['cache'] = NAtSChunkLayerCache(case['B'], case['Hkv'], case['SW'], chunk_size=C, device=torch.device(DEVICE))
        cache.update(k, v, roles)
        cache.post_update(n)
        state['tokens'] = _step_inputs(g, case, 4)
        # roles of the chunks the new tokens complete: few global ones, so that the cache keeps its size
        state['roles'] = [_token_roles(g, case, 0.02, 0.02) for _ in range(61)]
        state['count'] = state['done'] = 0
    elif kind == 'generate':
        state['q'], state['k'], state['v'] = _qkv(g, case, N)
        state['roles'] = _prompt_roles(g, case)
        state['tokens'] = _step_inputs(g, case, 16)
        state['token_roles'] = _token_roles(g, case, case['p_global'], case['p_local'])[..., 0].contiguous()
        state['out'] = [torch.empty_like(t[0]) for t in state['tokens']]
        state['side'] = torch.cuda.Stream()
    else:
        raise ValueError(kind)
    return state


# ---------------------------------------------------------------------------------------------------- one pass
def _new_cache(case):
    return NAtSChunkLayerCache(case['B'], case['Hkv'], case['SW'], chunk_size=case['C'], device=torch.device(DEVICE))


def _contents(cache):
    return [cache.cache_k, cache.cache_v, cache.valid_tokens, cache.size_global_kv, cache.size_local_kv]


def _run_prefill(s, case):
    cache = _new_cache(case)
    cache.update(s['k'], s['v'], s['roles'])
    o = prefill_attention(s['q'], s['k'], s['v'], s['roles'], case['C'], case['SW'])
    cache.post_update(case['N'])
    return o, cache


def _run_segments(s, case):
    cache = _new_cache(case)
    outs = []
    for i, (q, k, v, roles) in enumerate(s['segments']):
        cache.update(k, v, roles)
        outs.append(prefill_attention(q, k, v, roles, case['C'], case['SW']) if i == 0 else cache.prefill_attention(q))
        cache.post_update(q.shape[2])
    return outs + _contents(cache)


def _run_step(s, case):
    cache = s['cache']
    q, k, v = s['tokens'][s['count'] % len(s['tokens'])]
    s['count'] += 1
    roles = None
    if cache.get_chunk_fill_size() + 1 == case['C']:
        roles = s['roles'][s['done'] % len(s['roles'])]
        s['done'] += 1
    cache.update(k, v, roles, fused=True)
    o = cache.decode_attention(q)
    cache.post_update(1)
    return o, cache.size_global_kv, cache.size_local_kv


def _run_generate(s, case):
    o, cache = _run_prefill(s, case)
    n, tokens, outs = case['n_replays'], s['tokens'], s['out']
    cache.prepare_static_decode(1 + n * len(tokens), case['Hq'], case['D'])
    first = torch.empty_like(outs[0])
    cache.decode_step_static(*tokens[0], s['token_roles'], first)
    graph = torch.cuda.CUDAGraph()
    here = torch.cuda.current_stream()
    s['side'].wait_stream(here)
    with torch.cuda.stream(s['side']):
        graph.capture_begin()
        for (q, k, v), out in zip(tokens, outs):
            cache.decode_step_static(q, k, v, s['token_roles'], out, recording=True)
        graph.capture_end()
    here.wait_stream(s['side'])
    for _ in range(n):
        graph.replay()
    cache.note_static_steps(n * len(tokens))
    s['graph'], s['last'] = graph, cache         # the replays read the cache's buffers
    return [o, first, *outs, cache.size_global_kv, cache.size_local_kv]


@torch.no_grad()
def run(state):
    case = state['case']
    kind = case['kind']
    if kind == 'prefill':
        o, cache = _run_prefill(state, case)
        return [o, *_contents(cache)]
    if kind == 'forward':
        return nats_chunk_attention_fwd(state['q'], state['k'], state['v'], state['info'], None, True, case['D'] ** -0.5, case['C'],
                                        case['Hq'] // case['Hkv'], case['SW'])
    if kind == 'segments':
        return _run_segments(state, case)
    if kind == 'layer':
        cache = NAtSCache(case['SW'], case['C'])
        y = state['layer'](state['x'], state['rope'], None, 0, cache)
        lc = cache.cache_model[0]                # its extent depends on the roles the layer has chosen
        return [y, lc.size_global_kv, lc.size_local_kv]
    if kind == 'layer_step':
        cache, x = state['cache'], state['x'][state['pos'] % len(state['x'])]
        y = state['layer'](x, state['rope'], None, state['pos'], cache)
        state['pos'] += 1
        lc = cache.cache_model[0]
        return [y, lc.size_global_kv, lc.size_local_kv]
    if kind == 'step':
        return _run_step(state, case)
    return _run_generate(state, case)


# ---------------------------------------------------------------------------------------------------- work, tolerance
def _expected(case):
    """Per (sequence, kv-head), from a fixed sample of roles: visible (query, key) pairs of the prompt, tokens the eviction
    keeps behind the window, valid tokens of the window."""
    N, C, SW, heads = case['N'], case['C'], case['SW'], 4
    rng = np.random.default_rng(1)
    n_chunks, full = -(-N // C), N // C
    pairs = kept = ring = 0.0
    for _ in range(heads):
        pg = rng.uniform(case['p_global'], case.get('p_global_hi', case['p_global']))
        u = rng.random(n_chunks)
        roles = np.where(u < pg, GLOBAL, np.where(u < pg + case['p_local'], LOCAL, SLIDING))
        roles[0] = GLOBAL
        c = np.arange(n_chunks)
        fixed = (roles == GLOBAL) | (c == n_chunks - 1)
        nxt = np.minimum.accumulate(np.where(fixed, c, n_chunks - 1)[::-1])[::-1]      # next global (or last) chunk
        last = np.where(roles == SLIDING, c * C + SW + C - 1, np.where(fixed, N - 1, (nxt + 1) * C - 1))
        key = np.arange(N)
        pairs += float((np.minimum(last[key // C], N - 1) - key + 1).sum())
        done = roles[:full]
        last_global = np.flatnonzero(done == GLOBAL)[-1] if (done == GLOBAL).any() else -1
        kept += C * float(((done == GLOBAL) | ((done == LOCAL) & (np.arange(full) > last_global))).sum())
        ring += C * float((done[max(0, full - SW // C):] == SLIDING).sum())
    return pairs / heads, kept / heads, ring / heads


def work(case):
    """Bytes and flops of one pass: 4 * head_dim flops per visible (query, key) pair and query head, inputs and outputs once."""
    kind, B, Hq, Hkv, D, N = (case[k] for k in ('kind', 'B', 'Hq', 'Hkv', 'D', 'N'))
    size = 4 if case.get('dtype') == 'float32' else 2
    dim = Hq * D
    pairs, kept, ring = _expected(case)
    attention = 4.0 * D * B * Hq * pairs
    prompt = B * N * D * (2 * Hq + 2 * Hkv) * size                       # q, k, v in, o out
    cache = 2 * B * Hkv * D * 2 * (kept + case['SW'])                    # the compacted K and V
    decode = 2 * B * Hkv * D * 2 * (kept + ring) + 2 * B * D * (2 * Hq + 4 * Hkv)
    weights = 2 * dim * (2 * dim + 2 * Hkv * D)
    if kind in ('prefill', 'segments'):
        return dict(bytes=prompt + cache, flops=attention)
    if kind == 'forward':
        return dict(bytes=prompt + 8 * B * Hq * N, flops=attention)
    if kind == 'layer':
        return dict(bytes=weights + 4 * B * N * dim + cache, flops=attention + B * N * weights)
    if kind == 'layer_step':
        return dict(bytes=weights + decode, flops=4.0 * D * B * Hq * (kept + ring) + B * weights)
    if kind == 'step':
        return dict(bytes=decode, flops=4.0 * D * B * Hq * (kept + ring))
    steps = 1 + 16 * case['n_replays']
    return dict(bytes=prompt + cache + steps * decode, flops=attention + steps * 4.0 * D * B * Hq * (kept + ring))


def tolerance(case):
    """Four times what a pass differs from the same path in 64 bits: attention and decode outputs are bf16 roundings of fp32
    sums whose weights were rounded to bf16 (prompts: relative 0.0023, largest difference 0.059 of the root mean square, in rows
    that see many keys; single tokens: 0.0023 and 0.008); the layer adds bf16 projections on both sides (0.0037 and 0.107).
    Sizes, flags and counts are whole numbers and the same."""
    if case['kind'] in ('layer', 'layer_step'):
        return dict(rel=1.5e-2, max=0.43)
    return dict(rel=9e-3, max=0.04 if case['kind'] == 'step' else 0.24)
