"""The decode kernels against each other: which one runs depends on the number of (sequence, kv-head) pairs and segments."""
import pytest
import torch

from test_gpu_parity import assert_close_attn

pytestmark = pytest.mark.gpu

GLOBAL, LOCAL, SLIDING = 0, 1, 2


def dev():
    return torch.device('cuda', 0)


def make_cache(k, v, roles, C, SW):
    from neuralattentionsearch_b200 import NAtSChunkLayerCache
    cache = NAtSChunkLayerCache(k.shape[0], k.shape[1], SW, chunk_size=C, device=dev())
    cache.update(k, v, roles)
    cache.post_update(k.shape[2])
    return cache


def data(B, Hq, Hkv, N, D, C, seed):
    g = torch.Generator().manual_seed(seed)
    k, v = (torch.randn(B, Hkv, N, D, generator=g).mul_(0.5).to(dev()).bfloat16() for _ in range(2))
    roles = torch.randint(0, 3, (B, Hkv, -(-N // C)), generator=g).to(torch.uint8)
    roles[..., 0] = GLOBAL
    roles[0] = GLOBAL                                            # the first sequence keeps everything: its length is known
    if N % C:
        roles[..., -1] = GLOBAL
    toks = [tuple(torch.randn(B, h, 1, D, generator=g).mul_(0.5).to(dev()).bfloat16() for h in (Hq, Hkv, Hkv)) for _ in range(2 * C if C < 8 else 3)]
    return k, v, roles.to(dev()), toks


def kernel_of(cache, Hq, D, bound=None, fill=None):
    """Which kernel a step of this cache runs: the lines of use_strands and use_both in csrc/decode.cu."""
    splits = -(-((cache._t0_bound if bound is None else bound) + (cache.chunk_fill_size if fill is None else fill) + 1) // 1024)
    B, H = cache._buf_k.shape[:2]
    segments, nrep = B * H * splits, Hq // H
    if D == 64:
        if segments > (160 if splits <= 12 else 96) or splits > (16 if nrep < 8 else 48):
            return 'segments'
        return 'strands, V beside K' if segments <= 111 else 'strands, V in place of K'
    if segments > (72 if splits == 1 else 96) or splits > (16 if nrep == 1 else 24 if nrep < 4 else 96):
        return 'segments'
    return 'strands, V beside K' if segments <= 37 and splits <= 3 else 'strands, V in place of K'


def attend(cache, q, i, k, v, roles):
    """One step of sequences i of the inputs; returns the output and the kernel that ran."""
    full = cache.chunk_fill_size + 1 == cache.chunk_size
    cache.update(k[i].contiguous(), v[i].contiguous(), roles[i].contiguous() if full else None, fused=True)
    ran = kernel_of(cache, q.shape[1], q.shape[-1], fill=cache.chunk_fill_size - 1)
    o = cache.decode_attention(q[i].contiguous())
    cache.post_update(1)
    return o, ran


# cache lengths (window + tokens + the new one) around one, two and three segments of 1024 tokens, around tiles of 16, and short ones
@pytest.mark.parametrize('N,C,SW', [(1, 16, 64), (40, 16, 64), (959, 32, 64), (960, 32, 64), (991, 1, 32), (992, 1, 32), (1983, 64, 64), (2000, 8, 64),
                                    (3000, 128, 512)])
@pytest.mark.parametrize('D,Hq', [(64, 8), (64, 64), (128, 32), (128, 64)])
def test_a_head_decodes_the_same_whatever_the_batch(N, C, SW, D, Hq):
    """The same sequences in a large batch (a block per segment), in one of middle size (strands, V in the place of K) and alone
    (strands, with room for both where there are few segments per head): same bits, and those of a head are right."""
    Hkv = 8
    B = 26 if D == 64 else 13
    k, v, roles, toks = data(B, Hq, Hkv, N, D, C, seed=N + D)
    splits = -(-(SW + (N + len(toks)) // C * C + C) // 1024)     # of the longest sequence, at the last steps
    mid = -(-(112 if D == 64 else 38) // (Hkv * splits))
    batches = [slice(0, B), slice(0, mid), slice(0, 1), slice(mid - 1, mid)]
    caches = [make_cache(k[i].contiguous(), v[i].contiguous(), roles[i].contiguous(), C, SW) for i in batches]
    chunk_roles = torch.arange(B * Hkv, device=dev()).remainder(3).to(torch.uint8).view(B, Hkv, 1)
    ran = set()
    for step, (q, kn, vn) in enumerate(toks):
        (o, r0), (om, r1), (oa, r2), (ob, r3) = [attend(c, q, i, kn, vn, chunk_roles) for c, i in zip(caches, batches)]
        ran.update((('large', r0), ('middle', r1)))
        assert r2.startswith('strands') and r3.startswith('strands')
        assert torch.isfinite(o).all()
        assert torch.equal(om, o[:mid]) and torch.equal(oa, o[:1]) and torch.equal(ob, o[mid - 1:mid])
        if step == 0:                                            # the first sequence sees everything it has kept, which is everything
            keys, vals = (torch.cat([x[:1], y[:1]], 2).float() for x, y in ((k, kn), (v, vn)))
            s = torch.einsum('hrd,hnd->hrn', q[0].float().view(Hkv, Hq // Hkv, D), keys[0]) * D ** -0.5
            assert_close_attn(o[:1], torch.einsum('hrn,hnd->hrd', s.softmax(-1), vals[0]).reshape(1, Hq, 1, D))
    assert ran >= {('large', 'segments'), ('middle', 'strands, V in place of K')} and ('middle', 'segments') not in ran


@pytest.mark.parametrize('N,D,nrep,B', [(15500, 64, 2, 7), (15500, 128, 1, 7), (23900, 128, 2, 5), (47500, 64, 8, 3), (64000, 128, 4, 2), (97000, 128, 8, 2)])
def test_heads_of_many_segments(N, D, nrep, B):
    """The longest heads that run as strands: one head alone, and in a batch that runs in blocks of a segment."""
    C, SW = 128, 512
    k, v, roles, toks = data(B, nrep, 1, N, D, C, seed=N)
    both = [make_cache(k[:b].contiguous(), v[:b].contiguous(), roles[:b].contiguous(), C, SW) for b in (B, 1)]
    for q, kn, vn in toks:
        (o, r0), (oa, r1) = [attend(c, q, slice(0, b), kn, vn, roles[:, :, :1]) for c, b in zip(both, (B, 1))]
        assert r0 == 'segments' and r1.startswith('strands')
        assert torch.isfinite(o).all() and torch.equal(oa, o[:1])


@pytest.mark.parametrize('B,nrep,D,L', [(2, 8, 64, 10000), (1, 8, 128, 12000), (1, 1, 64, 900), (9, 4, 128, 900), (12, 8, 128, 900), (20, 2, 64, 5000)])
def test_a_launch_stays_inside_its_workspace(B, nrep, D, L):
    """A workspace of the size asked for, bytes behind it: the largest launches of strands and ones of whole segments."""
    from neuralattentionsearch_b200 import functional as F_
    H, C, SW = 8, 128, 512
    g = torch.Generator(device=dev()).manual_seed(L)
    k, v = (torch.randn(B, H, L + C, D, generator=g, device=dev()).bfloat16() for _ in range(2))
    valid = torch.ones(B, H, L + C, dtype=torch.uint8, device=dev())
    sg, sl = torch.full((B, H), L, dtype=torch.long, device=dev()), torch.zeros(B, H, dtype=torch.long, device=dev())
    state = torch.zeros(8, dtype=torch.int32, device=dev())
    state[0] = L
    q, kn = (torch.randn(B, h, 1, D, generator=g, device=dev()).bfloat16() for h in (H * nrep, H))
    need = F_.decode_workspace_bytes(B, H * nrep, H, D, L + C)
    ws = torch.full((need + 65536,), 0x5a, dtype=torch.uint8, device=dev())
    ws[:need] = 0
    o = torch.empty_like(q)
    F_.decode_fwd(q, kn, kn, o, k, v, valid, sg, sl, state, 3, L, C, SW, D ** -0.5, ws[:need])
    assert (ws[need:] == 0x5a).all()
    keys, vals = (torch.cat([x[:1, :, :L + 3], kn[:1]], 2)[0].float() for x in (k, v))
    s = torch.einsum('hrd,hnd->hrn', q[0].float().view(H, nrep, D), keys) * D ** -0.5
    assert_close_attn(o[:1], torch.einsum('hrn,hnd->hrd', s.softmax(-1), vals).reshape(1, H * nrep, 1, D))


STEP_SHAPES = [(1, 1, 32, 700, 64, 'strands'), (2, 16, 64, 1010, 128, 'strands'), (12, 4, 64, 900, 128, 'segments'), (9, 1, 16, 300, 64, 'strands'),
               (1, 128, 256, 1100, 128, 'strands'), (12, 1, 16, 300, 64, 'segments'), (26, 1, 32, 1500, 64, 'segments'), (26, 16, 64, 2100, 64, 'segments'),
               (14, 4, 64, 2100, 128, 'segments')]


@pytest.mark.parametrize('B,C,SW,N,D,kernel', STEP_SHAPES)
def test_one_launch_per_step_equals_the_two_it_replaces(B, C, SW, N, D, kernel):
    """Outputs, cache bytes, flags, sizes and step counters over steps that complete chunks of every role; the shapes for blocks of a
    segment have heads of one, two and three segments in launches of room for more."""
    from neuralattentionsearch_b200 import functional as F_
    Hkv, Hq, steps = 8, 16, max(10, C + 3)
    k, v, roles, _ = data(B, Hq, Hkv, N, D, C, seed=N)
    a, b = (make_cache(k, v, roles, C, SW) for _ in range(2))
    g = torch.Generator().manual_seed(1)
    for c in (a, b):
        c.prepare_static_decode(steps, Hq, D)
    assert kernel_of(a, Hq, D, bound=a._static_bound, fill=C - 1).startswith(kernel)
    for _ in range(steps):
        q, kn, vn = (torch.randn(B, h, 1, D, generator=g).mul_(0.5).to(dev()).bfloat16() for h in (Hq, Hkv, Hkv))
        r = torch.randint(0, 3, (B, Hkv), generator=g).to(torch.uint8).to(dev())
        oa, ob = torch.empty_like(q), torch.empty_like(q)
        a.decode_step_static(q, kn, vn, r, oa)
        F_.decode_step_fwd(q, kn, vn, ob, b._buf_k, b._buf_v, b._buf_valid, b.size_global_kv, b.size_local_kv, b._state, b._static_bound, C, SW,
                           D ** -0.5, b._dec_ws)
        F_.decode_step_place(r, b._buf_k, b._buf_v, b._buf_valid, b.size_global_kv, b.size_local_kv, b._state, C, SW)
        b.note_static_steps(1)
        for x, y in ((oa, ob), (a._buf_k, b._buf_k), (a._buf_v, b._buf_v), (a._buf_valid, b._buf_valid), (a.size_global_kv, b.size_global_kv),
                     (a.size_local_kv, b.size_local_kv), (a._state, b._state)):
            assert torch.equal(x, y)


@pytest.mark.parametrize('B,C,SW,N,D', [(26, 2, 32, 1500, 64), (14, 4, 64, 2100, 128)])
def test_large_recorded_steps_replay(B, C, SW, N, D):
    """A step in blocks of a segment, recorded once and replayed: outputs, cache bytes and counters of the steps called one by one."""
    Hkv, Hq, steps = 8, 16, 9
    k, v, roles, _ = data(B, Hq, Hkv, N, D, C, seed=N + 1)
    a, b = (make_cache(k, v, roles, C, SW) for _ in range(2))
    g = torch.Generator().manual_seed(2)
    ins = [tuple(torch.randn(B, h, 1, D, generator=g).mul_(0.5).to(dev()).bfloat16() for h in (Hq, Hkv, Hkv)) for _ in range(steps)]
    rs = [torch.randint(0, 3, (B, Hkv), generator=g).to(torch.uint8).to(dev()) for _ in range(steps)]
    for c in (a, b):
        c.prepare_static_decode(steps, Hq, D)
        assert kernel_of(c, Hq, D, bound=c._static_bound, fill=C - 1) == 'segments'
    outs = [torch.empty_like(q) for q, _, _ in ins]
    for (q, kn, vn), r, o in zip(ins, rs, outs):
        a.decode_step_static(q, kn, vn, r, o)
    held, hr, out = [t.clone() for t in ins[0]], rs[0].clone(), torch.empty_like(outs[0])
    b.decode_step_static(*held, hr, out)                         # one step outside of the graph first
    assert torch.equal(out, outs[0])
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        graph.capture_begin()
        b.decode_step_static(*held, hr, out, recording=True)
        graph.capture_end()
    torch.cuda.current_stream().wait_stream(side)
    for i in range(1, steps):
        for t, x in zip(held, ins[i]):
            t.copy_(x)
        hr.copy_(rs[i])
        graph.replay()
        assert torch.equal(out, outs[i]), i
    b.note_static_steps(steps - 1)
    for x, y in ((a._buf_k, b._buf_k), (a._buf_v, b._buf_v), (a._buf_valid, b._buf_valid), (a.size_global_kv, b.size_global_kv),
                 (a.size_local_kv, b.size_local_kv), (a._state, b._state)):
        assert torch.equal(x, y)


@pytest.mark.parametrize('B,C,SW,N,D,kernel', [(1, 1, 32, 700, 64, 'strands'), (2, 4, 64, 1010, 128, 'strands'), (2, 64, 128, 1142, 128, 'strands'),
                                               (12, 4, 64, 900, 128, 'segments'), (26, 1, 32, 1500, 64, 'segments')])
def test_steps_recorded_back_to_back(B, C, SW, N, D, kernel):
    """Steps whose launches overlap (nothing between them in the graph): outputs, cache bytes and counters of steps that are waited for
    one by one, over steps that complete chunks and steps that do not."""
    Hkv, Hq, steps = 8, 16, 11
    k, v, roles, _ = data(B, Hq, Hkv, N, D, C, seed=N + 2)
    a, b = (make_cache(k, v, roles, C, SW) for _ in range(2))
    g = torch.Generator().manual_seed(3)
    ins = [tuple(torch.randn(B, h, 1, D, generator=g).mul_(0.5).to(dev()).bfloat16() for h in (Hq, Hkv, Hkv)) for _ in range(steps)]
    rs = [torch.randint(0, 3, (B, Hkv), generator=g).to(torch.uint8).to(dev()) for _ in range(steps)]
    for c in (a, b):
        c.prepare_static_decode(2 * steps, Hq, D)
        assert kernel_of(c, Hq, D, bound=c._static_bound, fill=C - 1).startswith(kernel)
    want, got = ([torch.empty_like(q) for q, _, _ in ins] for _ in range(2))
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    assert N % C + steps >= C                                     # the first replay completes a chunk
    for again in range(2):
        for (q, kn, vn), r, o in zip(ins, rs, want):
            a.decode_step_static(q, kn, vn, r, o)
            torch.cuda.synchronize()
        if not again:
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                graph.capture_begin()
                for (q, kn, vn), r, o in zip(ins, rs, got):
                    b.decode_step_static(q, kn, vn, r, o, recording=True)
                graph.capture_end()
            torch.cuda.current_stream().wait_stream(side)
        graph.replay()
        b.note_static_steps(steps)
        for x, y in zip(want + [a._buf_k, a._buf_v, a._buf_valid, a.size_global_kv, a.size_local_kv, a._state],
                        got + [b._buf_k, b._buf_v, b._buf_valid, b.size_global_kv, b.size_local_kv, b._state]):
            assert torch.equal(x, y)
        assert a.chunk_fill_size == b.chunk_fill_size == (N + (again + 1) * steps) % C == int(b._state[4])


@pytest.mark.parametrize('B,rows,D,blocks,overlap', [(2, 1900, 64, 256, False), (2, 3900, 64, 384, True), (1, 3900, 64, 192, True), (4, 1900, 64, 512, False),
                                                     (8, 1900, 64, 256, True), (8, 3900, 64, 384, False), (16, 1900, 64, 512, True),
                                                     (2, 1100, 128, 192, True), (2, 1900, 128, 256, False), (2, 3900, 128, 384, True), (4, 1900, 128, 128, True),
                                                     (8, 1100, 128, 192, True), (16, 1900, 128, 512, True)])
def test_which_recorded_steps_overlap(B, rows, D, blocks, overlap):
    """The edge between two recorded steps: programmatic where the launches overlap, full where the second starts behind the first (the
    rule of csrc/decode.cu, for 148 SMs).  Outputs, cache and counters equal those of steps that are waited for either way."""
    import ctypes
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip('the numbers of blocks are for 148 SMs')
    Hkv, C, SW, steps = 8, 128, 512, 6
    Hq = 4 * Hkv
    g = torch.Generator(device=dev()).manual_seed(rows)
    k, v = (torch.randn(B, Hkv, rows, D, generator=g, device=dev()).bfloat16() for _ in range(2))
    roles = torch.full((B, Hkv, -(-rows // C)), GLOBAL, dtype=torch.uint8, device=dev())
    a, b = (make_cache(k, v, roles, C, SW) for _ in range(2))
    ins = [tuple(torch.randn(B, h, 1, D, generator=g, device=dev()).bfloat16() for h in (Hq, Hkv, Hkv)) for _ in range(steps)]
    r = torch.randint(0, 3, (B, Hkv), generator=g, device=dev()).to(torch.uint8)
    want, got = ([torch.empty_like(q) for q, _, _ in ins] for _ in range(2))
    for c in (a, b):
        c.prepare_static_decode(22, Hq, D)
    splits = -(-(a._static_bound + C) // 1024)
    assert B * Hkv * splits * (1 if kernel_of(a, Hq, D, bound=a._static_bound, fill=C - 1) == 'segments' else 4) == blocks
    for (q, kn, vn), o in zip(ins, want):
        a.decode_step_static(q, kn, vn, r, o)
        torch.cuda.synchronize()
    graph, side = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        graph.capture_begin()
        for (q, kn, vn), o in zip(ins, got):
            b.decode_step_static(q, kn, vn, r, o, recording=True)
        graph.capture_end()
    # an edge's data: from_port, to_port, type (1: programmatic), five reserved bytes
    n, nodes, data8 = ctypes.c_size_t(steps), [(ctypes.c_void_p * steps)() for _ in range(2)], (ctypes.c_uint8 * (8 * steps))()
    assert ctypes.CDLL('libcuda.so.1').cuGraphGetEdges_v2(ctypes.c_void_p(graph.raw_cuda_graph()), *nodes, data8, ctypes.byref(n)) == 0
    assert [data8[8 * i + 2] for i in range(n.value)] == [int(overlap)] * (steps - 1)
    graph.instantiate()
    graph.replay()
    torch.cuda.synchronize()
    for x, y in zip(want + [a._buf_k, a._buf_v, a._buf_valid, a.size_global_kv, a.size_local_kv, a._state],
                    got + [b._buf_k, b._buf_v, b._buf_valid, b.size_global_kv, b.size_local_kv, b._state]):
        assert torch.equal(x, y)
