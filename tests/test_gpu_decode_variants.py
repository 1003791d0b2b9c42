"""The decode kernels against each other: which one runs depends on the number of (sequence, kv-head) pairs and segments."""
import pytest
import torch

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


# cache lengths (window + tokens + the new one) around one and two segments of 1024 tokens, around tiles of 16, and short ones
@pytest.mark.parametrize('N,C,SW', [(1, 16, 64), (40, 16, 64), (959, 32, 64), (960, 32, 64), (991, 1, 32), (992, 1, 32), (1983, 64, 64), (2000, 8, 64),
                                    (3000, 128, 512)])
@pytest.mark.parametrize('D,Hq', [(64, 8), (128, 32), (128, 64)])
def test_a_head_decodes_the_same_whatever_the_batch(N, C, SW, D, Hq):
    """Ten sequences of 8 kv-heads run in blocks of a whole segment, one sequence in a block per strand: same bits."""
    B, Hkv = 10, 8
    k, v, roles, toks = data(B, Hq, Hkv, N, D, C, seed=N + D)
    every = make_cache(k, v, roles, C, SW)
    single = [make_cache(k[i:i + 1].contiguous(), v[i:i + 1].contiguous(), roles[i:i + 1].contiguous(), C, SW) for i in (0, 7)]
    chunk_roles = torch.arange(B * Hkv, device=dev()).remainder(3).to(torch.uint8).view(B, Hkv, 1)
    for q, kn, vn in toks:
        full = every.chunk_fill_size + 1 == C
        every.update(kn, vn, chunk_roles if full else None, fused=True)
        o = every.decode_attention(q)
        every.post_update(1)
        assert torch.isfinite(o).all()
        for i, c in zip((0, 7), single):
            s = slice(i, i + 1)
            c.update(kn[s].contiguous(), vn[s].contiguous(), chunk_roles[s].contiguous() if full else None, fused=True)
            oi = c.decode_attention(q[s].contiguous())
            c.post_update(1)
            assert torch.equal(oi, o[s])


@pytest.mark.parametrize('B,C,SW,N,D', [(1, 1, 32, 700, 64), (2, 16, 64, 1010, 128), (12, 4, 64, 900, 128), (12, 1, 16, 300, 64), (1, 128, 256, 1100, 128)])
def test_one_launch_per_step_equals_the_two_it_replaces(B, C, SW, N, D):
    """Outputs, cache bytes, flags, sizes and step counters over steps that complete chunks of every role."""
    from neuralattentionsearch_b200 import functional as F_
    Hkv, Hq, steps = 8, 16, max(10, C + 3)
    k, v, roles, _ = data(B, Hq, Hkv, N, D, C, seed=N)
    a, b = (make_cache(k, v, roles, C, SW) for _ in range(2))
    g = torch.Generator().manual_seed(1)
    for c in (a, b):
        c.prepare_static_decode(steps, Hq, D)
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
