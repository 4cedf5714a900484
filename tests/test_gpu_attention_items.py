"""The accurate kernel's blocks take several tiles of 128 queries one after the other, with every ring running on from one to
the next: more such items than the GPU has SMs, at key counts around the lengths of those rings, against the oracle."""

import pytest
import torch

import oracle
from gpu_common import out_heads, qkv, rel_l2

pytestmark = pytest.mark.gpu
MODES = {"per_channel": oracle.V_CHANNEL, "per_token": oracle.V_TOKEN, "outliers": oracle.V_OUTLIERS}


@pytest.mark.parametrize("preset", list(MODES))
@pytest.mark.parametrize("keys", [1, 64, 65, 190, 256, 449, 512, 513, 640, 1100])
def test_items_share_a_block(keys, preset):
    import unicaattention_b200 as unica

    q, k, v = qkv(1, 70, 700, keys, seed=keys)  # 70 heads x 6 tiles: three items for most blocks, the last tile ragged
    out = unica.attention(q.cuda(), k.cuda(), v.cuda(), **unica.PRESETS[preset])
    unica.check_status()
    k_mean = unica.quantize_k(k.cuda())[2].cpu()
    heads = [0, 1, 31, 48, 69]
    part = [x[:, heads] for x in (q, k, v)]
    want = oracle.attention_accurate(*part, MODES[preset], recip=True, k_mean=k_mean[:, heads])
    got = out_heads(out)[heads]
    assert rel_l2(got, want) < 2e-3, (keys, preset, rel_l2(got, want))
    for head in heads:  # and the same bits as alone, where a block has one item
        alone = unica.attention(*(x[:, head:head + 1].cuda() for x in (q, k, v)), **unica.PRESETS[preset])
        assert torch.equal(alone[:, 0], out[:, head]), (keys, preset, head)
