"""Prefill shapes at which the work distribution or a variant of the kernel can go wrong, against the fp32 oracle."""
import pytest
import torch

from oracle import nats_oracle as orc
from test_gpu_parity import assert_close_attn, dev, inputs

pytestmark = pytest.mark.gpu


def run_prefill(q, k, v, roles, C, SW):
    from neuralattentionsearch_b200 import check_status, prefill_attention
    o = prefill_attention(q.to(dev()).bfloat16(), k.to(dev()).bfloat16(), v.to(dev()).bfloat16(), torch.from_numpy(roles).to(dev()), C, SW)
    check_status(dev())
    return o


@pytest.mark.parametrize('B,Hq,Hkv,N,D,C,SW', [(8, 16, 16, 700, 64, 16, 64), (6, 12, 4, 600, 128, 32, 128), (6, 12, 12, 500, 128, 128, 128),
                                               (8, 16, 16, 330, 256, 64, 64)])
def test_items_with_an_empty_head_slot(B, Hq, Hkv, N, D, C, SW):
    """More work items than SMs, items of one head (group sizes 1 and 3, head_dim 256) and of few KV tiles: the issuer of the
    empty slot runs ahead of the other one by more than an item."""
    roles = orc.make_roles(B, Hkv, -(-N // C), 0.1, 0.3, seed=N)
    q, k, v = inputs(B, Hq, Hkv, N, D, seed=N + D, sigma=0.5)
    assert_close_attn(run_prefill(q, k, v, roles, C, SW), orc.prefill_attention(q, k, v, roles, C, SW))


@pytest.mark.parametrize('C', [1, 3, 8, 24, 32, 40, 64, 96])
def test_mask_bits_of_every_chunk_granularity(C):
    """Row masks from transposed column bits (chunks finer than 32 keys or no power of two) and from one compare per 32 columns
    (the others): tiles cut by the causal edge, by window and local limits and by the end of the sequence."""
    B, Hq, Hkv, N, D = 1, 4, 2, 777, 64
    SW = C * max(1, 150 // C)
    roles = orc.make_roles(B, Hkv, -(-N // C), 0.1, 0.4, seed=C)
    q, k, v = inputs(B, Hq, Hkv, N, D, seed=C, sigma=0.5)
    assert_close_attn(run_prefill(q, k, v, roles, C, SW), orc.prefill_attention(q, k, v, roles, C, SW))


@pytest.mark.parametrize('C,N,p_global,p_local', [(1, 2048, 0.1, 0.3), (2, 2500, 0.05, 0.3), (4, 2177, 0.2, 0.1), (8, 2300, 0.1, 0.3),
                                                  (16, 3001, 0.03, 0.1), (32, 2600, 0.3, 0.0), (64, 4000, 0.1, 0.6), (16, 2304, 1.0, 0.0),
                                                  (1, 2304, 0.0, 1.0), (32, 2304, 0.0, 0.0),
                                                  (1, 2304, 1.0, 0.0), (2, 3000, 0.6, 0.2), (1, 1024, 0.1, 0.3), (16, 1500, 0.1, 0.2),
                                                  (8, 2500, 0.5, 0.2), (16, 2500, 0.85, 0.1), (64, 4000, 0.9, 0.1)])
@pytest.mark.parametrize('D', [64, 128, 256])
def test_far_chunks_are_gathered(C, N, p_global, p_local, D):
    """Prompts long enough for the gathered tiles: every way of gathering (copied rows, boxes of 8 to 64 rows), a last gathered
    tile that is full, part empty or missing (no global chunk but the first), all chunks global (more rows than are copied), all local, and so many global ones
    that some or all items leave their tiles in place."""
    B, Hq, Hkv = (2, 4, 2) if D == 64 else (1, 3, 1)
    SW = C * max(1, 200 // C)
    roles = orc.make_roles(B, Hkv, -(-N // C), p_global, p_local, seed=N + C)
    q, k, v = inputs(B, Hq, Hkv, N, D, seed=N, sigma=0.5)
    assert_close_attn(run_prefill(q, k, v, roles, C, SW), orc.prefill_attention(q, k, v, roles, C, SW))


@pytest.mark.parametrize('C', [1, 4])
def test_workspace_without_room_for_copied_rows(C):
    """A C caller who asks for the workspace without the head_dim (no room for copies of rows) gets the tiles computed in place; one byte
    less than the full size does the same."""
    from neuralattentionsearch_b200 import _lib, check_status
    from neuralattentionsearch_b200.functional import status_word
    B, Hq, Hkv, N, D, SW = 1, 4, 2, 2000, 64, 64
    roles = orc.make_roles(B, Hkv, -(-N // C), 0.1, 0.3, seed=C)
    q, k, v = inputs(B, Hq, Hkv, N, D, seed=C, sigma=0.5)
    ref = orc.prefill_attention(q, k, v, roles, C, SW)
    qd, kd, vd, r = *(t.to(dev()).bfloat16() for t in (q, k, v)), torch.from_numpy(roles).to(dev())
    lib, outs = _lib.lib(), []
    small, full = lib.nats_b200_prefill_workspace_bytes(B, Hkv, N, C), lib.nats_b200_prefill_workspace_bytes_for(B, Hkv, N, D, C)
    assert small < full
    for nbytes in (small, full - 1, full):
        ws, o = torch.full((nbytes + 4096,), 0x5a, dtype=torch.uint8, device=dev()), torch.empty_like(qd)
        _lib.call('nats_b200_prefill_fwd', qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), o.data_ptr(), r.data_ptr(), B, Hq, Hkv, N, D, C, SW, D ** -0.5,
                  ws.data_ptr(), nbytes, None, status_word(dev()).data_ptr(), torch.cuda.current_stream().cuda_stream)
        check_status(dev())
        assert (ws[nbytes:] == 0x5a).all()
        assert_close_attn(o, ref)
        outs.append(o)
    assert torch.equal(outs[0], outs[1]) and not torch.equal(outs[1], outs[2])


@pytest.mark.parametrize('C', [1, 2, 4, 8, 16, 32, 64])
@pytest.mark.parametrize('D', [64, 128, 256])
def test_gathered_tiles_hold_no_key_of_the_future(C, D):
    """K and V that are not finite from some position on (what stands behind the end of a prompt, or one bad token) leave every
    row in front of the tile of that position as it is: a masked key is multiplied by an exact zero, which needs a finite V."""
    from neuralattentionsearch_b200 import check_status, prefill_attention
    B, Hq, Hkv, N = 1, 2, 1, 2700
    SW = C * max(1, 200 // C)
    roles = orc.make_roles(B, Hkv, -(-N // C), 0.1, 0.3, seed=C)
    roles[..., -(-N // C) // 2:][..., ::7] = orc.ROLE_GLOBAL
    q, k, v = (t.to(dev()).bfloat16() for t in inputs(B, Hq, Hkv, N, D, seed=C + D, sigma=0.5))
    r = torch.from_numpy(roles).to(dev())
    clean = prefill_attention(q, k, v, r, C, SW)
    assert torch.isfinite(clean).all()
    for first, last in ((2300, N), (1800, 1801), (1999, N)):
        at = first // C * C                                      # from a chunk's first token on, and that chunk is a global one
        rr = r.clone()
        rr[..., first // C] = orc.ROLE_GLOBAL
        want = prefill_attention(q, k, v, rr, C, SW)
        for bad in (float('inf'), float('nan')):
            kk, vv = k.clone(), v.clone()
            kk[:, :, at:last], vv[:, :, at:last] = bad, bad
            got = prefill_attention(q, kk, vv, rr, C, SW)
            assert torch.equal(got[:, :, :at // 128 * 128], want[:, :, :at // 128 * 128])
            assert not torch.isfinite(got[:, :, last - 1]).any()
    check_status(dev())


@pytest.mark.parametrize('C', [1, 16, 64])
def test_far_chunks_of_a_call_over_a_cache(C):
    """Segments over the compacted cache (ragged, the second one starting inside a chunk) equal one call over the sequence."""
    from neuralattentionsearch_b200 import NAtSChunkLayerCache, check_status, prefill_attention
    B, Hq, Hkv, D, SW = 2, 4, 2, 128, 256
    lens = [1500, 1301, 900]
    N = sum(lens)
    roles = torch.from_numpy(orc.make_roles(B, Hkv, -(-N // C), 0.08, 0.25, seed=C)).to(dev())
    q, k, v = (t.to(dev()).bfloat16() for t in inputs(B, Hq, Hkv, N, D, seed=C, sigma=0.5))
    whole = orc.prefill_attention(q.float().cpu(), k.float().cpu(), v.float().cpu(), roles.cpu().numpy(), C, SW)
    cache = NAtSChunkLayerCache(B, Hkv, SW, chunk_size=C, device=dev())
    pos = 0
    for n in lens:
        s = slice(pos, pos + n)
        r = roles[..., pos // C:-(-(pos + n) // C)].clone()
        last = (pos + n) // C if (pos + n) % C else -1           # an unfinished last chunk counts as global
        if last >= 0:
            r[..., -1] = 0
        cache.update(k[:, :, s], v[:, :, s], r.contiguous())
        o = prefill_attention(q[:, :, s].contiguous(), k[:, :, s].contiguous(), v[:, :, s].contiguous(), r.contiguous(), C, SW) if pos == 0 \
            else cache.prefill_attention(q[:, :, s].contiguous())
        cache.post_update(n)
        check_status(dev())
        assert_close_attn(o, whole[:, :, s])
        pos += n


@pytest.mark.parametrize('D', [64, 128, 256])
@pytest.mark.parametrize('Hq,Hkv', [(4, 2), (3, 1)])
@pytest.mark.parametrize('C,N,p_global', [(128, 1100, 1.0), (32, 900, 1.0), (24, 900, 1.0), (16, 1500, 0.4), (1, 2048, 0.2)])
def test_rows_whose_maximum_grows_in_every_tile(D, Hq, Hkv, C, N, p_global):
    """Keys that grow along the sequence: the reference maximum of a row moves in every tile for one query head of a pair, in every second
    one for the other, so that O is rescaled again and again behind the P.V of the tile in front (chunks of a multiple of 32 tokens and
    others, gathered tiles, items of one and of two heads)."""
    SW = C * max(1, 200 // C)
    q, k, v = inputs(1, Hq, Hkv, N, D, seed=N + D, sigma=0.5)
    per_tile = 12.0                                               # growth of the scores, in powers of two
    slope = torch.where(torch.arange(Hq) % 2 == 0, 1.0, 0.45).view(1, -1, 1, 1)
    q = (q + slope).bfloat16().float()
    k = (k + (torch.arange(N) * (per_tile / 128 * 0.6931 / D ** 0.5)).view(1, 1, -1, 1)).bfloat16().float()
    roles = orc.make_roles(1, Hkv, -(-N // C), p_global, 0.0, seed=C)
    if p_global == 1.0:
        # how often the kernel's rule (a growth of more than 8) moves the reference of a row that sees all keys up to its own
        s = torch.einsum('hqd,hkd->hqk', q[0], k[0].repeat_interleave(Hq // Hkv, 0)) * (D ** -0.5 * 1.4427)
        s.masked_fill_(torch.ones(N, N, dtype=torch.bool).triu(1), float('-inf'))
        tops = torch.stack([t.amax(-1) for t in s.split(128, -1)], -1)
        ref, moves = tops[..., 0], torch.zeros(Hq, N)
        for j in range(1, tops.shape[-1]):
            move = tops[..., j] > ref + 8
            ref, moves = torch.where(move, tops[..., j], ref), moves + move
        tiles = torch.arange(N) // 128
        assert (moves[0] >= tiles - 1).float().mean() > 0.9 and (moves[1] >= tiles // 2 - 1).float().mean() > 0.9 and (moves[1] < tiles).float().mean() > 0.5
    assert_close_attn(run_prefill(q, k, v, roles, C, SW), orc.prefill_attention(q, k, v, roles, C, SW))
