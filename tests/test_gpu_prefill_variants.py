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
