"""The forms of the one-launch quantizers (four or eight blocks per head; tiles loaded ahead or not), at both sides of the lines between
them on a device of 148 SMs, against the separate statistics and quantizer passes: bit for bit."""

import pytest
import torch

from gpu_common import qkv
from test_gpu_call import rope

pytestmark = pytest.mark.gpu

INT8 = [(18, 513), (19, 513),                        # ahead up to 37 clusters of eight, with more than a tile to a block
        (18, 512), (3, 255), (3, 256), (3, 257),     # ... and a tile at most; four blocks per head up to 256 keys
        (34, 300), (35, 300), (29, 1024), (30, 1024), (31, 1025), (37, 2048), (38, 2048)]  # four where eight would crowd the SMs
OUTLIERS = [(3, 77), (16, 1024), (17, 1024), (24, 600), (25, 600), (8, 4128)]  # ahead: room for K and V, but not for Q with them
FAST = [(3, 511), (3, 512), (3, 513), (16, 1000), (17, 1000), (17, 2049), (2, 4096), (2, 4097)]
FAST_ROTATED = [(3, 511), (3, 513), (11, 700), (12, 700), (16, 1024), (17, 1024), (17, 1025), (23, 512), (24, 512), (38, 300), (39, 300), (48, 300)]


def by_separate_passes(unica, q, k, v, preset, table):
    settings = unica.PRESETS[preset]
    if preset == "fast":  # statistics, codes and table by kernels of their own
        return unica.kernel_inputs(q, k, v, rope=table, **settings)
    q_tiles = 2 * -(-q.shape[2] // 256)
    q8, q_scale = unica.quantize_int8(q, None, 128, table, tiles=q_tiles)
    k8, k_scale = unica.quantize_int8(k, unica.rope_stats(k, table)[0], 64, table)
    if preset == "per_token":
        v8, v_scale, v_token = unica.quantize_v(v, per_token=True)
        return q8, q_scale, k8, k_scale, v8, v_scale, v_token, unica.lib.V_TOKEN
    if preset == "outliers":  # head by head, which is never the form with tiles loaded ahead
        v8, v_scale, keys, rows = (torch.cat(parts, 1) for parts in zip(*(unica.quantize_v(v[:, h : h + 1], outliers=8) for h in range(v.shape[1]))))
        return q8, q_scale, k8, k_scale, v8, v_scale, (keys, rows), unica.lib.V_OUTLIERS
    return q8, q_scale, k8, k_scale, *unica.quantize_v(v), None, unica.lib.V_CHANNEL


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("preset, rotated, heads, tokens", [(preset, rotated, *shape) for preset, rotated, shapes in (
    ("per_channel", False, INT8), ("per_token", False, INT8), ("per_channel", True, [(3, 257), (28, 600), (27, 600)]), ("outliers", False, OUTLIERS),
    ("outliers", True, [(17, 600)]), ("fast", False, FAST), ("fast", True, FAST_ROTATED)) for shape in shapes])
def test_every_form_equals_the_separate_passes(preset, rotated, heads, tokens, dtype):
    import unicaattention_b200 as unica

    q, k, v = (x.to(dtype).cuda() for x in qkv(1, heads, tokens, tokens, seed=heads, channel_scale=True))
    q += torch.linspace(0, 1, tokens, device="cuda")[:, None].to(dtype)
    v[:, :, tokens // 3] *= 30
    settings, table = unica.PRESETS[preset], rope(tokens) if rotated else None
    want = unica.attention(q, k, v, inputs=by_separate_passes(unica, q, k, v, preset, table), rope=table, **settings)
    assert torch.equal(unica.attention(q, k, v, rope=table, **settings), want)
    unica.check_status()
