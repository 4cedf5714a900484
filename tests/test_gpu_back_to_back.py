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
    ballast = torch.zeros(64 << 20, device="cuda")  # 0.1 ms: the first calls or so are queued behind it (for all of them see below)

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


def written_and_read(unica, preset, rotated, shape=(1, 4, 1000, 1000), calls=18):
    """A function that queues `calls` calls, each behind kernels that write its q, k, v and, rotated, the angle table that the kernels read, a
    different one of them last each time; and the outputs that it must give."""
    settings = dict(unica.PRESETS[preset])
    base = [t.cuda() for t in qkv(*shape, seed=13)]
    given = [t.clone() for t in base]
    factor = torch.linspace(0.5, 2.0, calls, device="cuda").bfloat16()
    writes = [lambda i, x=x, t=t: torch.mul(t, factor[i], out=x) for x, t in zip(given, base)]
    if rotated:
        angle = torch.rand(1, shape[2], 1, 64, device="cuda") * 6
        cos, sin = angle.cos(), angle.sin()
        settings["rope"] = torch.stack([torch.stack([cos, -sin], -1), torch.stack([sin, cos], -1)], -2)
        compact = unica.compact_rope(settings["rope"])  # kept while the table is this one
        tables = [compact.clone(), compact.flip(1).contiguous(), compact.roll(7, 1)]
        writes.append(lambda i: compact.copy_(tables[i % 3]))
    given[2][:, :, shape[3] // 2] = 0  # (outputs of an early read differ by far)

    def run(between=lambda: None):
        outputs = []
        for i in range(calls):
            for j in range(len(writes)):
                writes[(i + j) % len(writes)](i)
            between()
            outputs.append(unica.attention(*given, **settings))
            between()
        for x in given:
            x.zero_()
        return outputs

    return run, run(torch.cuda.synchronize)


@pytest.mark.parametrize("rotated", [False, True])
@pytest.mark.parametrize("preset", ["per_channel", "per_token", "outliers", "fast"])
def test_calls_queued_behind_work_that_outlasts_the_loop(preset, rotated):
    import unicaattention_b200 as unica

    run, want = written_and_read(unica, preset, rotated)
    x = torch.randn(8192, 8192, device="cuda").bfloat16()
    y, done = torch.empty_like(x), torch.cuda.Event()
    for _ in range(30):  # some 20 ms
        torch.mm(x, x, out=y)
    done.record()
    got = run()
    assert not done.query()  # every call was queued before the first one's turn came
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    unica.check_status()


@pytest.mark.parametrize("rotated", [False, True])
@pytest.mark.parametrize("preset", ["per_channel", "per_token", "outliers", "fast"])
def test_captured_calls(preset, rotated):
    import unicaattention_b200 as unica

    run, want = written_and_read(unica, preset, rotated)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run()
    for _ in range(3):
        for out in got:
            out.zero_()
        graph.replay()
        graph.replay()  # straight after the first
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    unica.check_status()
