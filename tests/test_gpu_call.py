"""A whole call through the one entry point (and, up to 8192 tokens, the one-launch quantizers) against the single steps, bit
for bit: kernel_inputs() and the kernel on its operands, at sizes around the statistics' 256-token blocks, the 64-key tiles and
the line between the short and the long quantizers."""

import pytest
import torch

from gpu_common import qkv

pytestmark = pytest.mark.gpu
PRESETS = ["per_channel", "per_token", "outliers", "fast"]


def rope(tokens, batch=1):
    angle = torch.rand((batch, tokens, 1, 64), generator=torch.Generator().manual_seed(7)) * 6
    cos, sin = angle.cos(), angle.sin()
    return torch.stack([torch.stack([cos, -sin], -1), torch.stack([sin, cos], -1)], -2).cuda()


@pytest.mark.parametrize("preset", PRESETS)
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 3, 300, 77), (1, 2, 1000, 1000), (1, 2, 129, 5), (1, 2, 2050, 8192), (1, 1, 8192, 8193), (1, 2, 8300, 700)])
def test_one_entry_point_equals_the_steps(shape, preset):
    import unicaattention_b200 as unica

    q, k, v = (x.cuda() for x in qkv(*shape, seed=shape[3], channel_scale=True))
    settings = unica.PRESETS[preset]
    inputs = unica.kernel_inputs(q, k, v, **settings)
    if preset == "outliers" and shape[3] >= 8:
        v8, scale, keys, rows = inputs[4], inputs[5], *inputs[6]
        order = unica.v_outliers(v, 8).sort(-1).values  # found by torch
        assert torch.equal(keys.long().sort(-1).values, order)
    steps = unica.attention(q, k, v, inputs=inputs, **settings)
    assert torch.equal(unica.attention(q, k, v, **settings), steps)
    half = [x.transpose(1, 2).contiguous().transpose(1, 2).half() for x in (q, k, v)]
    steps = unica.attention(*(x.half().bfloat16() for x in (q, k, v)), **settings).half()
    assert torch.equal(unica.attention(*half, **settings), steps)
    unica.check_status()


@pytest.mark.parametrize("preset", PRESETS)
@pytest.mark.parametrize("tokens", [65, 513, 4100, 8200])
def test_with_rope(tokens, preset):
    import unicaattention_b200 as unica

    q, k, v = (x.cuda() for x in qkv(2, 2, tokens, tokens, seed=tokens))
    table, settings = rope(tokens), unica.PRESETS[preset]
    steps = unica.attention(q, k, v, inputs=unica.kernel_inputs(q, k, v, rope=table, **settings), rope=table, **settings)
    assert torch.equal(unica.attention(q, k, v, rope=table, **settings), steps)
    unica.check_status()


@pytest.mark.parametrize("tokens", [1, 255, 257, 2048, 8192])
def test_short_operands_equal_the_separate_passes(tokens):
    """quantize_k and quantize_v_channel of short heads, whose means are summed as rope_stats sums them."""
    import unicaattention_b200 as unica

    _, k, v = (x.cuda() for x in qkv(1, 3, 1, tokens, seed=tokens, channel_scale=True))
    k8, scale, mean = unica.quantize_k(k)
    assert torch.equal(mean, unica.rope_stats(k)[0])
    want8, want_scale = unica.quantize_int8(k, mean, 64)
    assert torch.equal(k8, want8) and torch.equal(scale, want_scale)
    assert all(torch.equal(a, b) for a, b in zip(unica.quantize_v_channel(v), unica.quantize_v(v)))
    unica.check_status()


@pytest.mark.parametrize("heads", [8, 9, 55, 60, 112])
@pytest.mark.parametrize("tokens", [1024, 1025, 2048, 2049, 4128, 8192])
def test_short_operands_alone(tokens, heads):
    """K alone and V alone: few heads, which go through the single steps above 2048 tokens, and with and without enough heads for
    clusters of four blocks, which have room for 4096 tokens."""
    import unicaattention_b200 as unica

    x = (torch.randn(1, heads, tokens, 128, generator=torch.Generator("cuda").manual_seed(tokens), device="cuda") + 0.5).bfloat16()
    k8, scale, mean = unica.quantize_k(x)
    assert torch.equal(mean, unica.rope_stats(x)[0])
    want8, want_scale = unica.quantize_int8(x, mean, 64)
    assert torch.equal(k8, want8) and torch.equal(scale, want_scale)
    assert all(torch.equal(a, b) for a, b in zip(unica.quantize_v_channel(x), unica.quantize_v(x)))
    unica.check_status()


@pytest.mark.parametrize("rotated", [False, True])
@pytest.mark.parametrize("preset", PRESETS)
@pytest.mark.parametrize("keys", [255, 1024, 1025])
def test_many_short_heads_equal_the_same_heads_alone(keys, preset, rotated):
    """Enough heads for the one-launch quantizers to take clusters of four blocks (up to 2048 tokens, rotated 1024), against one head at a time, which
    takes clusters of eight above 256 keys (NVFP4: 512 tokens); test_gpu_call_lines.py has the lines themselves."""
    import unicaattention_b200 as unica

    q, k, v = (x.cuda() for x in qkv(1, 48, keys, keys, seed=keys, channel_scale=True))
    settings = dict(unica.PRESETS[preset], **({"rope": rope(keys)} if rotated else {}))
    out = unica.attention(q, k, v, **settings)
    unica.check_status()
    for head in (0, 17, 47):
        alone = unica.attention(*(x[:, head:head + 1] for x in (q, k, v)), **settings)
        assert torch.equal(alone, out[:, head:head + 1]), (keys, preset, head)


@pytest.mark.parametrize("preset", PRESETS)
@pytest.mark.parametrize("halves", ["k", "v", "qv", "k out"])
@pytest.mark.parametrize("keys", [300, 8192])
def test_each_tensor_by_its_own_element_type(keys, halves, preset):
    """The C entry point with float16 and bfloat16 mixed: a float16 tensor counts as its rounding to bfloat16."""
    import ctypes

    import unicaattention_b200 as unica

    q, k, v = (x.cuda() for x in qkv(1, 2, 300, keys, seed=keys))
    q, k, v = (x.half() if name in halves.split()[0] else x for name, x in zip("qkv", (q, k, v)))
    want = unica.attention(*(x.bfloat16() for x in (q, k, v)), **unica.PRESETS[preset])
    out = torch.empty_like(want, dtype=torch.float16 if "out" in halves else torch.bfloat16)
    settings = unica.TILE | unica.PRESETS[preset]
    mode = 1 if settings["V_TOKEN"] else 2 if settings["V_OUTLIERS"] else 0
    layouts = [n for x in (q, k, v, out) for n in (*x.stride()[:3], 2, int(x.dtype == torch.float16))]
    where = (0, 0, 0, unica.status_word(q.device).data_ptr(), torch.cuda.current_stream().cuda_stream)
    sizes = (2, 300, keys, int(preset == "fast"), mode, settings["V_OUTLIERS"], settings["SMOOTH_Q"], 0, unica.SCALE_LOG2)
    size = unica.lib.attention_workspace(unica.lib.pack_call(0, 0, 0, 0, 0, 0, *where, *layouts, *sizes))
    workspace, queued = torch.empty(size, dtype=torch.uint8, device="cuda"), ctypes.c_int()
    pointers = [x.data_ptr() for x in (q, k, v, out, workspace)]
    assert unica.lib.library().unica_b200_attention_call(unica.lib.pack_call(*pointers, size, *where, *layouts, *sizes), ctypes.byref(queued)) == 0
    unica.check_status()
    assert out.equal(want.to(out.dtype)) and queued.value >= 2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("tokens", [100, 8192, 8200])
def test_outlier_keys_that_are_not_numbers(tokens, value, dtype):
    """A key with a NaN or an infinity is an outlier before every finite one, at any length, and shows in the output."""
    import unicaattention_b200 as unica

    q, k, v = (x.to(dtype).cuda() for x in qkv(1, 2, 64, tokens, seed=tokens))
    bad, large = tokens // 3, tokens - 1
    v[:, :, large] *= 50
    v[:, 1, bad, 77] = value
    _, _, keys, rows = unica.quantize_v(v, outliers=8)
    assert torch.equal(keys.long().sort(-1).values, unica.v_outliers(v, 8).sort(-1).values)
    assert bad in keys[0, 1] and large in keys[0, 1] and bad not in keys[0, 0]
    out = unica.attention(q, k, v, **unica.PRESETS["outliers"])
    unica.check_status()
    assert not out[:, 1, :, 77].isfinite().any() and out[:, 1, :, :77].isfinite().all() and out[:, 0].isfinite().all()
