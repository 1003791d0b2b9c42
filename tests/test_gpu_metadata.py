"""Role metadata kernels whose blocks go over the chunks in several steps: sizes around the step and the block."""
import numpy as np
import pytest
import torch

from oracle import nats_oracle as orc

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 4), (1023, 1, 4), (1024, 1, 4), (1025, 1, 64), (5000, 1, 256), (3001, 2, 64), (4097, 16, 64), (9000, 48, 96), (70000, 32, 128), (9000, 5000, 5000)]


def dev():
    return torch.device('cuda', 0)


def draw_roles(B, H, Nc, seed):
    roles = orc.make_roles(B, H, Nc, 0.05, 0.3, seed=seed)
    roles[0, 0] = orc.ROLE_LOCAL                                # a head without a global chunk
    roles[-1, -1, Nc // 2:] = orc.ROLE_SLIDING
    return roles


@pytest.mark.parametrize('N,C,SW', SHAPES)
def test_row_limits_and_visible_counts(N, C, SW):
    from neuralattentionsearch_b200 import _lib
    B, H, rep = 2, 2, 3
    Nc, Nt = -(-N // C), -(-N // 128)
    roles = draw_roles(B, H, Nc, N)
    r = torch.from_numpy(roles).to(dev())
    lim = torch.empty(B, H, Nc, dtype=torch.int32, device=dev())
    tmax, tmin = (torch.empty(B, H, Nt, dtype=torch.int32, device=dev()) for _ in range(2))
    n_vis = torch.empty(B, H * rep, N, dtype=torch.int32, device=dev())
    _lib.call('nats_b200_role_prep', r.data_ptr(), B, H, N, C, SW, lim.data_ptr(), tmax.data_ptr(), tmin.data_ptr(), None, None)
    _lib.call('nats_b200_visible_counts', lim.data_ptr(), B, H * rep, H, N, C, n_vis.data_ptr(), None)
    ref = np.minimum(orc.row_limit(roles, C, SW), orc.NO_LIMIT).astype(np.int64)
    assert np.array_equal(lim.cpu().numpy(), ref)
    for b in range(B):
        for h in range(H):
            d = np.ones(N + 1, np.int64)                         # key q appears at row q, key k leaves behind row lim
            size = np.minimum(np.arange(1, Nc + 1) * C, N) - np.arange(Nc) * C
            np.subtract.at(d, np.minimum(ref[b, h] + 1, N), size)
            want = np.cumsum(d[:N])
            got = n_vis.cpu().numpy()[b, h * rep:(h + 1) * rep]
            assert (got == want).all()


@pytest.mark.parametrize('N,C,SW', SHAPES)
def test_eviction_plan(N, C, SW):
    from neuralattentionsearch_b200 import functional as F_
    B, H = 2, 2
    Nc, full = -(-N // C), N // C
    roles = draw_roles(B, H, Nc, N + 1)
    r = torch.from_numpy(roles).to(dev())
    rank = torch.empty(B, H, Nc, dtype=torch.int32, device=dev())
    sg, sl = (torch.empty(B, H, dtype=torch.long, device=dev()) for _ in range(2))
    state = torch.zeros(8, dtype=torch.int32, device=dev())
    F_.evict_plan(r, N, C, SW, rank, sg, sl, state)
    lens = []
    for b in range(B):
        for h in range(H):
            x = roles[b, h, :full]
            g = x == orc.ROLE_GLOBAL
            last = np.flatnonzero(g)[-1] if g.any() else -1
            keep = np.zeros(Nc, bool)
            keep[:full] = g | ((x == orc.ROLE_LOCAL) & (np.arange(full) > last))
            before = np.cumsum(keep) - keep
            assert np.array_equal(rank[b, h].cpu().numpy(), np.where(keep, before, -1 - before))
            assert sg[b, h].item() == SW + C * g.sum() and sl[b, h].item() == C * (keep.sum() - g.sum())
            lens.append(SW + C * keep.sum())
    assert state.cpu().tolist() == [max(lens), 0, 0, 0, 0, 0, 0, 0]


def test_output_in_token_order_holds_the_same_bits():
    from neuralattentionsearch_b200 import prefill_attention
    g = torch.Generator().manual_seed(0)
    for B, Hq, Hkv, N, D, C in ((2, 6, 2, 700, 64, 32), (1, 8, 4, 513, 128, 32), (2, 2, 2, 200, 256, 32), (1, 4, 2, 150, 32, 32), (1, 4, 2, 1700, 64, 16),
                                (1, 4, 2, 1500, 128, 1)):        # the last two with gathered tiles
        q, k, v = (torch.randn(B, h, N, D, generator=g).mul_(0.5).to(dev()).bfloat16() for h in (Hq, Hkv, Hkv))
        roles = torch.from_numpy(orc.make_roles(B, Hkv, -(-N // C), 0.1, 0.3, seed=N)).to(dev())
        a = prefill_attention(q, k, v, roles, C, 128)
        b = prefill_attention(q, k, v, roles, C, 128, token_major=True)
        assert b.shape == a.shape and torch.equal(a, b)
        assert D == 32 or b.transpose(1, 2).is_contiguous()


@pytest.mark.parametrize('B,Hq,Hkv,N,D,C,SW', [(1, 4, 4, 1000, 64, 16, 64), (2, 8, 2, 513, 128, 1, 32), (1, 2, 2, 300, 256, 64, 128), (1, 2, 1, 9, 64, 8, 8),
                                               (1, 4, 2, 1700, 64, 16, 64), (1, 4, 2, 1500, 128, 1, 64)])
def test_fp32_prompts_are_rounded_by_the_kernels(B, Hq, Hkv, N, D, C, SW):
    """q, k, v in fp32: the output before its rounding to bf16, the cache bytes of a prompt given in bf16; also for tensors the
    rounding kernels do not take (not contiguous)."""
    from neuralattentionsearch_b200 import NAtSChunkLayerCache, prefill_attention
    g = torch.Generator().manual_seed(N)
    q, k, v = (torch.randn(B, h, N, D, generator=g).mul_(0.5).to(dev()) for h in (Hq, Hkv, Hkv))
    roles = torch.from_numpy(orc.make_roles(B, Hkv, -(-N // C), 0.2, 0.3, seed=N)).to(dev())
    outs, caches = [], []
    strided = [t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v)]
    for qq, kk, vv in ((q, k, v), strided, [t.bfloat16() for t in (q, k, v)]):
        cache = NAtSChunkLayerCache(B, Hkv, SW, chunk_size=C, device=dev())
        cache.update(kk, vv, roles)
        outs.append(prefill_attention(qq, kk, vv, roles, C, SW))
        cache.post_update(N)
        caches.append(cache)
    assert outs[0].dtype == outs[1].dtype == torch.float32 and outs[2].dtype == torch.bfloat16
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0].bfloat16(), outs[2])
    for c in caches[:2]:
        assert torch.equal(c.cache_k, caches[2].cache_k) and torch.equal(c.cache_v, caches[2].cache_v) and torch.equal(c.valid_tokens, caches[2].valid_tokens)


@pytest.mark.parametrize('B,H,N,C,SW', [(1, 1, 64, 64, 64), (2, 3, 700, 16, 64), (3, 5, 5001, 1, 32)])
@pytest.mark.parametrize('past', [False, True])
def test_planned_size_reaches_the_host(B, H, N, C, SW, past):
    """The plan that reports the new extent to pinned host memory: sizes, ranks and state of the plain one, the same number on the host, for
    several reports under way at once; a raised status word comes along."""
    from neuralattentionsearch_b200 import _lib, functional as F_
    dev = torch.device('cuda', 0)
    g = torch.Generator(device=dev).manual_seed(N)
    outs, reports = [], []
    roles = [torch.randint(0, 3, (B, H, -(-N // C)), generator=g, device=dev).to(torch.uint8) for _ in range(3)]

    def buffers():
        sizes = [torch.full((B, H), x, dtype=torch.long, device=dev) for x in (SW + 3 * C, 2 * C)]
        return [torch.empty(B, H, roles[0].shape[-1], dtype=torch.int32, device=dev), torch.empty(B, H, dtype=torch.int32, device=dev) if past else None,
                *sizes, torch.zeros(8, dtype=torch.int32, device=dev)]

    for r in roles:
        outs.append(buffers())
        reports.append(F_.evict_plan_report(r, N, C, SW, *outs[-1]))
    for r, out, report in zip(roles, outs, reports):
        want = buffers()
        if past:
            F_.evict_plan_past(r, N, C, SW, *want)
        else:
            F_.evict_plan(r, N, C, SW, want[0], *want[2:])
        for x, y in zip(want, out):
            assert x is None or torch.equal(x, y)
        assert report() == int(want[-1][0]) == int((want[2] + want[3]).max())
    F_.status_word(dev).fill_(5)
    with pytest.raises(_lib.NatsB200Error, match='code 5'):
        F_.evict_plan_report(roles[0], N, C, SW, *buffers())()
    F_.check_status(dev)


def test_scalars_are_read_back_behind_the_callers_stream():
    """``read_word_async``: the value that the caller's stream has written when the call is made, several at once and dropped unread ones among
    them; a raised status word comes along."""
    from neuralattentionsearch_b200 import _lib, functional as F_
    dev = torch.device('cuda', 0)
    x = torch.randn(2048, 2048, device=dev)
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            words, reads = torch.zeros(6, 4, dtype=torch.int32, device=dev), []
            for i, w in enumerate(words):
                x = (x @ x).clamp_(-1, 1)                         # the copy has something to wait for
                w.fill_(100 + i)
                reads.append(F_.read_word_async(w))
                words[i, 1:].fill_(-1)
            del reads[2]
            assert [r() for r in reads] == [100, 101, 103, 104, 105]
    F_.status_word(dev).fill_(5)
    with pytest.raises(_lib.NatsB200Error, match='code 5'):
        F_.read_word_async(words[0])()
    F_.check_status(dev)


def test_a_refused_cuda_call_does_not_fail_the_next_one():
    """A report that is to go to memory the device cannot be given an address of is refused (by the runtime, before any launch), and the
    same call with pinned memory right behind it succeeds."""
    import numpy as np
    from neuralattentionsearch_b200 import _lib, functional as F_
    rt = pytest.importorskip('cuda.bindings.runtime')
    dev = torch.device('cuda', 0)
    B, H, N, C, SW = 1, 2, 300, 16, 64
    roles = torch.zeros(B, H, -(-N // C), dtype=torch.uint8, device=dev)
    rank = torch.empty(B, H, roles.shape[-1], dtype=torch.int32, device=dev)
    sg, sl, state = torch.empty(B, H, dtype=torch.long, device=dev), torch.empty(B, H, dtype=torch.long, device=dev), torch.zeros(8, dtype=torch.int32, device=dev)
    pageable, pinned = np.zeros(1 << 12, dtype=np.int32), torch.zeros(2, dtype=torch.int32, pin_memory=True)
    err, _ = rt.cudaHostGetDevicePointer(pageable.ctypes.data, 0)
    rt.cudaGetLastError()
    if err == rt.cudaError_t.cudaSuccess:
        pytest.skip('this system gives out device addresses of pageable memory')

    def report(host):
        _lib.call('nats_b200_evict_plan_report', roles.data_ptr(), B, H, N, C, SW, rank.data_ptr(), None, sg.data_ptr(), sl.data_ptr(), state.data_ptr(),
                  F_.status_word(dev).data_ptr(), host, torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        with pytest.raises(_lib.NatsB200Error, match='cudaHostGetDevicePointer'):
            report(pageable.ctypes.data)
        report(pinned.data_ptr())
        torch.cuda.synchronize()
        assert int(pinned[0]) == int((sg + sl).max())
