"""What attention() looks at before it takes a plan: everything that a call's outcome follows from, and nothing that the checks refuse."""

import pytest
import torch

import unicaattention_b200 as unica


def qkv():
    return [torch.zeros(1, 2, 64, 128, dtype=torch.bfloat16) for _ in range(3)]


def key(q, k, v, kernel=unica.DEFAULT_KERNEL, **tile):
    return unica._plan_key(kernel, q, k, v, tile)


def test_settings_that_are_equal_but_not_the_same():
    q, k, v = qkv()
    assert key(q, k, v, SMOOTH_Q=512) == key(q, k, v, SMOOTH_Q=512)
    for other in (512.0, True, 256):
        assert key(q, k, v, SMOOTH_Q=512) != key(q, k, v, SMOOTH_Q=other)
    assert key(q, k, v, V_TOKEN=1) != key(q, k, v, PRODUCER=1)
    assert key(q, k, v, NOPE=0) != key(q, k, v)


def test_a_changed_default_is_another_call(monkeypatch):
    q, k, v = qkv()
    before = key(q, k, v)
    monkeypatch.setitem(unica.TILE, "V_TOKEN", 1)
    assert key(q, k, v) != before and key(q, k, v, V_TOKEN=0) != before


def test_arguments_without_a_key_are_refused_as_ever():
    q, k, v = qkv()
    attention = unica.attention.__wrapped__  # (the wrapper asks for a GPU first)
    with pytest.raises(ValueError, match="KEYS_PER_TILE"):
        attention(q, k, v, KEYS_PER_TILE=[64])
    with pytest.raises(ValueError, match="unknown kernel"):
        attention(q, k, v, kernel=["attention_fp4"])
    with pytest.raises(ValueError, match="on the GPU"):  # an unused setting may hold anything
        attention(q, k, v, WAVE_DISPATCH=[])
    with pytest.raises(TypeError, match="all be bfloat16 or all float16"):
        attention(q, k.float().numpy(), v)
