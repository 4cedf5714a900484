"""Calls in a loop, on buffers that the kernel before has just written and the kernel after writes again: the first kernel of a call is
launched to overlap the end of the kernel before it, and must neither read nor write anything early."""

import pytest
import torch

from gpu_common import qkv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset", ["per_channel", "per_token", "outliers", "fast"])
@pytest.mark.parametrize("shape", [(2, 3, 300, 77), (1, 4, 1024, 1024)])
def test_inputs_just_written(preset, shape):
    import unicaattention_b200 as unica

    settings, calls = unica.PRESETS[preset], 24
    base = [t.cuda() for t in qkv(*shape, seed=12)]
    given = [t.clone() for t in base]
    factor = torch.linspace(0.5, 2.0, calls, device="cuda").bfloat16()
    ballast = torch.zeros(64 << 20, device="cuda")  # a kernel long enough for everything behind it to be queued

    def write(i):
        for x, t in zip(given, base):
            torch.mul(t.roll(i, 2), factor[i], out=x)

    want = []
    for i in range(calls):
        write(i)
        torch.cuda.synchronize()
        want.append(unica.attention(*given, **settings))
        torch.cuda.synchronize()
    for _ in range(2):
        ballast.add_(1)
        got = []
        for i in range(calls):
            write(i)
            got.append(unica.attention(*given, **settings))
        got += [unica.attention(*given, **settings) for _ in range(3)]  # and straight after one another, on the last inputs
        for x in given:
            x.zero_()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want + [want[-1]] * 3))
    unica.check_status()
