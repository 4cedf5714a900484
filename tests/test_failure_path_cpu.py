"""What the kernels' source must hold to for a wait that gives up: seen without a GPU, since no test may make one fail there."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "unicaattention_b200" / "csrc"


@pytest.mark.parametrize("name, warps", [("attention_int8.cu", 2), ("attention_fp4.cu", 3)])
def test_no_two_warps_drain_on_one_word(name, warps):
    """A wait that gives up sets its word, and ends every other wait on it at once.  What a warp waits for at the block's end, when
    tensor memory and shared memory go away, no other warp's wait may cut short."""
    roles = re.split(r"__device__ __forceinline__ void (\w+_warp)\(", (CSRC / name).read_text())
    words = {}
    for role, body in zip(roles[1::2], roles[2::2]):
        if used := set(re.findall(r"mbar_wait_line\(.*, &(sm\.[^,]+), nullptr, 0\)", body)):  # the waits that report no status
            words[role] = used
    assert len(words) == warps and all(len(used) == 1 for used in words.values()), words
    assert len(set.union(*words.values())) == warps and not any("abort_flag" in word for used in words.values() for word in used), words


@pytest.mark.parametrize("name", ["attention_int8.cu", "attention_fp4.cu"])
def test_rows_are_sent_only_if_no_warp_gave_up(name):
    """The warps that store rows see their own waits only: another's, which went on with whatever lay in its buffers, is in the word
    that all share."""
    source = (CSRC / name).read_text()
    before, _, _ = source.partition("send_staged_rows(")
    last = before[before.rindex("ok = __all_sync("):].partition(";")[0]
    assert "gave_up(sm.abort_flag)" in last, last


def test_the_smoothing_kernel_has_its_tensor_memory_before_the_next_kernel_comes():
    """An attention block takes all tensor memory of its SM and then waits for the kernel before it."""
    body = (CSRC / "quantize_fp4.cu").read_text().partition("smooth_bias_kernel(")[2]
    assert body.index("tmem_alloc(") < body.index("__syncthreads();") < body.index("let_next_kernel_start();") < body.index("wait_for_previous_kernel();")
