"""The one-launch quantizers with four blocks per head (many heads of up to 2048 tokens) against eight (the same heads, few at a time):
bit for bit, at the edges of a block's 256-token statistics."""

import pytest
import torch

from gpu_common import randn_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset, heads", [("per_channel", 38), ("per_token", 38), ("fast", 19)])
@pytest.mark.parametrize("tokens", [1025, 1400, 2047, 2048])
def test_four_blocks_are_eight(preset, heads, tokens):
    import unicaattention_b200 as unica

    q, k, v = (randn_bf16((1, heads, tokens, 128), i).cuda() for i in range(3))
    q += torch.linspace(0, 1, tokens, device="cuda")[:, None].bfloat16()
    k += 0.5
    v[:, :, tokens // 3] *= 30
    whole = unica.attention(q, k, v, **unica.PRESETS[preset])
    for first in (0, heads - 2):
        part = [t[:, first : first + 2] for t in (q, k, v)]
        assert torch.equal(unica.attention(*part, **unica.PRESETS[preset]), whole[:, first : first + 2])
    unica.check_status()
