"""wave_plan() and the group sizes of attention_host() by the items that the kernels' launches really take."""

import math

import pytest
import torch

import unicaattention_b200 as unica


@pytest.fixture(autouse=True)
def a_b200(monkeypatch):
    monkeypatch.setattr(unica, "sm_count", lambda device: 148)


def plan(heads, n_queries, kernel="attention_fp4"):
    return unica.wave_plan(heads, n_queries, kernel, "cuda:0")


@pytest.mark.parametrize("heads, n_queries, rows, blocks, waves", [
    (1, 8192, 128, 64, 1), (18, 1024, 128, 144, 1), (19, 1024, 256, 76, 1), (100, 128, 128, 100, 1), (400, 100, 128, 400, 3), (400, 129, 256, 400, 3),
    (30, 4128, 256, 510, 4), (40, 32760, 256, 5120, 35)])
def test_items_of_the_fast_kernel(heads, n_queries, rows, blocks, waves):
    got = plan(heads, n_queries)
    assert (got["rows"], got["blocks"], got["waves"], got["per_wave"]) == (rows, blocks, waves, 148)
    assert got["efficiency"] == blocks / (waves * 148)


def test_the_form_that_takes_less_time():
    for heads in (1, 3, 18, 19, 37, 40, 74, 75, 148, 149, 300):
        for n_queries in (1, 128, 129, 256, 257, 777, 1024, 4128):
            one, two = (math.ceil(heads * math.ceil(n_queries / rows) / 148) for rows in (128, 256))
            assert plan(heads, n_queries)["rows"] == (128 if 2 * one < 3 * two else 256)
    assert unica.lib.library().unica_b200_fast_item_rows(0, 1, 148) == 0


def test_accurate_items_are_tiles():
    assert plan(30, 4128, unica.DEFAULT_KERNEL) == {"blocks": 990, "per_wave": 148, "waves": 7, "efficiency": 990 / 1036, "rows": 128}


def test_host_groups_weigh_both_forms(monkeypatch):
    """40 heads x 512 tokens: groups of 4 .. 7 heads, all of single tiles; where one size takes pairs its efficiency counts whole."""
    asked = []

    class NoGpu(Exception):
        pass

    def no_gpu(device):  # the sizes have been chosen
        raise NoGpu

    def wave_plan(heads, n_queries, kernel, device):
        asked.append(heads)
        return {"efficiency": 0.9 if heads == 5 else 0.7 if heads == 6 else 0.1, "rows": 128 if heads == 5 else 256}  # 0.675 against 0.7

    sizes = []
    monkeypatch.setattr(unica, "wave_plan", wave_plan)
    monkeypatch.setattr("unicaattention_b200.host.group_sizes", lambda heads, largest=None: sizes.append(largest) or [])
    monkeypatch.setattr(torch.cuda, "device", no_gpu)
    q, k, v = (torch.zeros(1, 40, 512, 128, dtype=torch.bfloat16) for _ in range(3))
    with pytest.raises(NoGpu):
        unica.attention_host(q, k, v, out=torch.empty_like(q), device=torch.device("cuda:0"), **unica.PRESETS["fast"])
    assert asked == [4, 5, 6, 7] and sizes == [6]
