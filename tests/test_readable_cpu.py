"""What the kernels read in place, and what they are given a copy of: tokens must start on 16-byte boundaries."""

import pytest
import torch

import unicaattention_b200 as unica


@pytest.mark.parametrize("offset, in_place", [(0, True), (8, True), (1, False), (4, False)])
def test_tokens_between_boundaries_are_copied(offset, in_place):
    flat = torch.randn(2 * 3 * 5 * 128 + 8).bfloat16()
    x = flat[offset:][: 2 * 3 * 5 * 128].view(2, 3, 5, 128)  # contiguous, wherever it starts
    got = unica.readable(x)
    assert (got is x) == in_place and got.data_ptr() % 16 == 0
    assert got.is_contiguous() and torch.equal(got, x)


def test_strides():
    x = torch.randn(2, 5, 3, 128).bfloat16().transpose(1, 2)
    assert unica.readable(x) is x
    for odd in (torch.randn(2, 3, 5, 129).bfloat16()[..., :128], torch.randn(2, 3, 128, 5).bfloat16().transpose(2, 3)):
        got = unica.readable(odd)
        assert got is not odd and got.is_contiguous() and torch.equal(got, odd)
