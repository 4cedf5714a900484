"""attention() by a plan (a call whose shapes, strides, types and settings came before) against the call without one, bit for bit."""

import pytest
import torch

from gpu_common import qkv

pytestmark = pytest.mark.gpu


def without_plans(unica, *args, **settings):
    unica._PLANS.clear()
    return unica.attention(*args, **settings)


@pytest.mark.parametrize("preset", ["per_channel", "per_token", "outliers", "fast"])
def test_planned_calls(preset):
    import unicaattention_b200 as unica

    settings = unica.PRESETS[preset]
    base = qkv(2, 3, 300, 300, seed=5) + qkv(2, 3, 300, 300, seed=6)
    first, second = ([t.cuda() for t in base[i : i + 3]] for i in (0, 3))
    odd = [torch.cat([t.flatten(), t.flatten()[:8]])[1 : 1 + t.numel()].view(t.shape) for t in second]  # the strides of `second`, two bytes off
    views = [t.transpose(1, 2).contiguous().transpose(1, 2) for t in second]  # the shapes, other strides
    half = [t.half() for t in second]
    for tensors in (second, odd, views, half):
        want = without_plans(unica, *tensors, **settings)
        unica._PLANS.clear()
        unica.attention(*first, **settings)
        assert len(unica._PLANS) == 1
        for _ in range(2):
            got = unica.attention(*tensors, **settings)
            assert torch.equal(got, want) and got.stride() == want.stride() and got.dtype == want.dtype
    unica.check_status()


def test_what_a_plan_looks_at_in_every_call(monkeypatch):
    import unicaattention_b200 as unica

    q, k, v = (t.cuda() for t in qkv(1, 4, 260, 77, seed=8))
    want = without_plans(unica, q, k, v)
    asked = []
    with monkeypatch.context() as patch:  # another planner takes over at once
        patch.setattr(unica, "heads_per_call", lambda *args: asked.append(1) or 3)
        assert torch.equal(unica.attention(q, k, v), want) and asked
    with monkeypatch.context() as patch:  # memory has become short
        patch.setattr(unica, "free_vram", lambda device, fresh=False: 1)
        patch.setattr(unica, "_attention_call", lambda *args: asked.append(2) and False)
        assert torch.equal(unica.attention(q, k, v), want) and 2 in asked
    stream = torch.cuda.Stream()  # the stream is the call's, not the plan's
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        got = unica.attention(q, k, v)
    stream.synchronize()
    assert torch.equal(got, want)
    for bad in ((q, k[:, :, :0], v[:, :, :0]), (q.float(), k, v), (q, k, v[:, :, :70]), (q.cpu(), k, v)):
        with pytest.raises((ValueError, TypeError)):
            unica.attention(*bad)
    with pytest.raises(ValueError):
        unica.attention(q, k, v, NOPE=1)


def test_a_changed_default(monkeypatch):
    import unicaattention_b200 as unica

    q, k, v = (t.cuda() for t in qkv(1, 4, 260, 77, seed=9))
    per_channel, per_token = unica.attention(q, k, v), unica.attention(q, k, v, V_TOKEN=1)
    assert not torch.equal(per_channel, per_token)
    with monkeypatch.context() as patch:
        patch.setitem(unica.TILE, "V_TOKEN", 1)
        for _ in range(2):
            assert torch.equal(unica.attention(q, k, v), per_token)
            assert torch.equal(unica.attention(q, k, v, V_TOKEN=0), per_channel)
    assert torch.equal(unica.attention(q, k, v), per_channel)


def test_only_plain_calls_leave_a_plan():
    """A call with out= in another layout, or on tensors that are copied first, takes no plan: it must not leave one that plain calls cannot use either."""
    import unicaattention_b200 as unica

    q, k, v = (t.cuda() for t in qkv(1, 4, 260, 77, seed=10))
    want = without_plans(unica, q, k, v)
    (plan,) = unica._PLANS.values()
    out = torch.empty(1, 260, 4, 128, dtype=q.dtype, device="cuda").transpose(1, 2)
    assert torch.equal(unica.attention(q, k, v, out=out), want) and list(unica._PLANS.values()) == [plan]
    assert plan.run(q, k, v) is not None
    unica._PLANS.clear()
    unica.attention(q, k, v, out=out)
    odd = torch.cat([q.flatten(), q.flatten()[:8]])[1 : 1 + q.numel()].view(q.shape)  # two bytes off a 16-byte boundary
    assert torch.equal(unica.attention(odd, k, v), without_plans(unica, odd.clone(), k, v))
    unica._PLANS.clear()
    unica.attention(odd, k, v)
    assert not unica._PLANS
