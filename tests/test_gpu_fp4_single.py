"""The fast kernel with one query tile per block (calls that would leave SMs idle) against the one with two: bit for bit."""

import math

import pytest
import torch

from gpu_common import randn_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq, nk, smooth", [(129, 64, 512), (300, 77, 512), (256, 1000, 0), (640, 300, 512), (1100, 1100, 256)])
def test_one_tile_is_a_pair(nq, nk, smooth):
    import unicaattention_b200 as unica

    sms = unica.sm_count(torch.device("cuda", torch.cuda.current_device()))
    tiles, pairs = math.ceil(nq / 128), math.ceil(nq / 256)
    many = sms // pairs  # one round of pairs, two of single tiles
    assert 2 * math.ceil(tiles * many / sms) >= 3 > 2 * math.ceil(tiles * 2 / sms)
    q = randn_bf16((1, many, nq, 128), 1).cuda()
    k, v = (randn_bf16((1, many, nk, 128), i).cuda() for i in (2, 3))
    q += torch.linspace(0, 1, nq, device="cuda")[:, None].bfloat16()
    whole = unica.attention(q, k, v, kernel="attention_fp4", SMOOTH_Q=smooth)
    for first, last in ((0, 1), (many - 2, many)):
        part = [t[:, first:last] for t in (q, k, v)]
        assert torch.equal(unica.attention(*part, kernel="attention_fp4", SMOOTH_Q=smooth), whole[:, first:last])
    unica.check_status()


def test_heads_of_one_tile():
    """Up to 128 queries a pair's second tile would be empty: one tile per block whatever the number of heads."""
    import unicaattention_b200 as unica

    q, k, v = (randn_bf16((2, 100, n, 128), i).cuda() for i, n in enumerate((100, 130, 130)))
    whole = unica.attention(q, k, v, **unica.PRESETS["fast"])
    for b, h in ((0, 0), (1, 99), (1, 47)):
        one = [t[b : b + 1, h : h + 1] for t in (q, k, v)]
        assert torch.equal(unica.attention(*one, **unica.PRESETS["fast"]), whole[b : b + 1, h : h + 1])
    unica.check_status()


@pytest.mark.parametrize("keys", [1, 64, 65, 190, 256, 300, 513])
def test_blocks_of_several_one_tile_items(keys):
    """Four items for most blocks, at key counts around the rings' lengths: from the third on the two query slots are taken again."""
    import unicaattention_b200 as unica

    q, k, v = (randn_bf16((1, 500, n, 128), i).cuda() for i, n in enumerate((100, keys, keys)))
    whole = unica.attention(q, k, v, **unica.PRESETS["fast"])
    for head in (0, 147, 148, 295, 296, 320, 443, 444, 499):  # a block's first, second, third and fourth item
        one = [t[:, head : head + 1] for t in (q, k, v)]
        assert torch.equal(unica.attention(*one, **unica.PRESETS["fast"]), whole[:, head : head + 1]), head
    unica.check_status()
