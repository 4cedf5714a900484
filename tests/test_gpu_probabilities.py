"""How often a byte P^ of the accurate kernel misses the rounding of its exact probability.

One key tile whose V is a unit matrix makes the output P^ / sum: a byte of 1 .. 64 that is one off shows as a change of at least
1/64, four times what the bfloat16 output rounds away."""

import pytest
import torch

import unicaattention_b200 as unica

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset", ["per_channel", "per_token"])
def test_bytes_of_p_round_as_the_exact_probabilities_do(preset):
    heads, n = 37, 8192
    gen = torch.Generator("cuda").manual_seed(5)
    q = torch.randn(1, heads, n, 128, device="cuda", generator=gen).bfloat16()
    k = torch.randn(1, heads, 64, 128, device="cuda", generator=gen).bfloat16()
    v = torch.cat([torch.eye(64)] * 2, 1).bfloat16().cuda().expand(1, heads, 64, 128).contiguous()
    inputs = unica.kernel_inputs(q, k, v, **unica.PRESETS[preset])
    out = unica.attention(q, k, v, inputs=inputs, **unica.PRESETS[preset])
    unica.check_status()
    q8, q_scale, k8, k_scale = inputs[:4]
    q_codes, k_codes = unica.decode_int8(q8, n), unica.decode_int8(k8, 64)
    missed = total = 0
    for h in range(heads):
        factor = (q_scale[0, h] * k_scale[0, h, 0]) * torch.tensor(unica.SCALE_LOG2, dtype=torch.float32, device="cuda")  # as the kernel forms it
        x = (q_codes[0, h].double() @ k_codes[0, h].double().T) * factor.double().repeat_interleave(128)[:n, None]
        p = 255 * torch.exp2(x - x.amax(1, keepdim=True))
        want = p.round()
        share = want / (want if preset == "per_channel" else p).sum(1, keepdim=True)  # per token the denominator sums p before rounding
        small = (want >= 1) & (want <= 64)
        missed += int((((out[0, h, :, :64].double() - share).abs() * want > 0.5 * share) & small).sum())
        total += int(small.sum())
    # A byte misses where p is within its error of a half: 2 |error| p of them, p some 20 on average here.  The exponent's argument
    # is rounded twice at values of 4 .. 8 (a quarter of the step 2^-21 on average each) and the exponential errs by some 1e-7:
    # 1.6e-7 of p, 6e-6 of the bytes (measured 2.7e-6 and 4.5e-6).  With the argument another 23 below, 1.3e-5 and 9.8e-6.
    assert missed < 7e-6 * total, (missed, total)


@pytest.mark.parametrize("preset", ["per_channel", "per_token"])
def test_sums_over_the_key_tiles(preset):
    """A tile's 64 keys are one key here, so that every byte of P^ is 255 and only the sums over the tiles are left to err: how many
    outputs are not the bfloat16 of what 64-bit sums of the same operands give."""
    heads, n, tiles = 4, 4096, 65
    gen = torch.Generator("cuda").manual_seed(8)
    q = torch.randn(1, heads, n, 128, device="cuda", generator=gen).bfloat16()
    k = (0.2 * torch.randn(1, heads, tiles, 128, device="cuda", generator=gen)).bfloat16().repeat_interleave(64, 2)
    v = torch.randn(1, heads, tiles * 64, 128, device="cuda", generator=gen).bfloat16()
    if preset == "per_token":  # one value of each size in every token: all keys have the scale 4 / 127
        v = v.clamp(-4, 4)
        v[..., 0] = 4
    inputs = unica.kernel_inputs(q, k, v, **unica.PRESETS[preset])
    out = unica.attention(q, k, v, inputs=inputs, **unica.PRESETS[preset])
    unica.check_status()
    q8, q_scale, k8, k_scale, v8, v_scale = inputs[:6]
    scores = unica.decode_int8(q8, n)[0].float() @ unica.decode_int8(k8, tiles * 64)[0, :, ::64].float().transpose(1, 2)  # exact: below 2^24
    factor = q_scale[0].repeat_interleave(128, 1)[:, :n, None] * k_scale[0][:, None, :] * torch.tensor(unica.SCALE_LOG2, dtype=torch.float32, device="cuda")
    top = (scores * factor).double()  # a tile's maximum as the kernel has it
    weight = torch.exp2(top - top[..., :1])
    sums = unica.decode_v8(v8, tiles * 64)[0].double().view(heads, tiles, 64, 128).sum(2)
    want = (weight @ sums) / (64 * weight.sum(-1, keepdim=True)) * (v_scale[0].double()[:, None, :] if preset == "per_channel" else 4 / 127)
    missed = (out[0].double() != want.float().bfloat16().double()).double().mean()
    # What V's bias adds to a tile's sums is 128 * 64 * 255 = 2^21 here, the most there is.  With one tile's share of it in a sum, an
    # addition rounds to 2^-2 (0.07 rms), 65 of them err by 0.6 at random; the sums themselves are 28 * 8 * 255 * 8 = 460000 in size:
    # 1.3e-6.  The same sums in numpy with an error of 8.3e-7 miss the bfloat16 of the exact ones in 8.9e-4 of the outputs, with
    # 1.4e-7 (no bias) in 2.1e-4, with 4.8e-6 (eight tiles' shares) in 4.1e-3: in proportion, so that 1.3e-6 is 1.4e-3 at most.  The
    # tiles' factors (an exponential each) add some 2e-7.
    assert missed < 1.6e-3, float(missed)
