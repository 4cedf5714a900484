"""The calls whose speed matters, as a user of this framework makes them: `attention()` in its four presets on tensors in
GPU memory (contiguous, or the transposed [batch, tokens, heads, 128] view the ComfyUI nodes hand over; bfloat16 or
float16; RoPE left to the quantizers or not), and `attention_host()` on pinned host memory.

A case is a dict: batch, heads, queries, keys, preset, dtype, layout ("bhnd" contiguous, "bnhd" transposed view), rope,
host, values ("plain": N(0,1) with a mean in K; "uneven": channels of Q and K of uneven size, a drifting mean in Q and two
V tokens far above the rest, as image and video models have them)."""

import functools
import math

import torch

import unicaattention_b200 as unica

HEAD_DIM = 128
LONGEST = 118320  # tokens of the longest call the benchmark has (the high-resolution pass)
PRESETS = ("per_token", "per_channel", "outliers", "fast")


def case(name, batch, heads, queries, keys, preset, dtype="bfloat16", layout="bhnd", rope=False, host=False, values="plain"):
    return {"name": name, "batch": batch, "heads": heads, "queries": queries, "keys": keys, "preset": preset, "dtype": dtype,
            "layout": layout, "rope": rope, "host": host, "values": values}


def listed():
    return [
        # the smallest calls, where launches and host time count: the reference emulator's own example ...
        case("example", 1, 4, 1024, 1024, "per_channel"),
        # ... cross-attention from an image to a short prompt, both lengths ragged ...
        case("cross", 2, 8, 1000, 77, "per_token", dtype="float16", layout="bnhd"),
        # ... and a preview-sized latent with RoPE in the quantizers, two prompts in a batch
        case("preview_fast", 2, 16, 777, 777, "fast", layout="bnhd", rope=True, values="uneven"),
        # an image model's self-attention (30 heads x 4128 tokens) as the ComfyUI node calls it by default ...
        case("image", 1, 30, 4128, 4128, "per_token", layout="bnhd", values="uneven"),
        # ... with V's largest keys kept exact, in float16 ...
        case("image_outliers", 1, 30, 4128, 4128, "outliers", dtype="float16", values="uneven"),
        # ... and in the fast mode
        case("image_fast", 1, 30, 4128, 4128, "fast", values="uneven"),
        # a video model's self-attention (40 heads x 32760 tokens): the benchmark's headline ...
        case("video", 1, 40, 32760, 32760, "per_channel"),
        # ... the node's default with fused RoPE ...
        case("video_rope", 1, 40, 32760, 32760, "per_token", layout="bnhd", rope=True, values="uneven"),
        # ... the fast mode ...
        case("video_fast", 1, 40, 32760, 32760, "fast", values="uneven"),
        # ... and the same call for tensors that live in host memory
        case("video_host", 1, 40, 32760, 32760, "per_channel", host=True),
        # the largest: the high-resolution pass of that model
        case("hires", 1, 40, LONGEST, LONGEST, "per_channel", values="uneven"),
    ]


def _log_uniform(rng, low, high):
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    batch, heads = rng.choice((1, 1, 2)), _log_uniform(rng, 1, 40)
    host = rng.random() < 0.1
    queries = _log_uniform(rng, 64, 32760 if host else LONGEST)
    cross = rng.random() < 0.2
    keys = _log_uniform(rng, 16, 4096) if cross else queries
    most = 20 * LONGEST * LONGEST  # half of the largest listed call: the dearest preset stays below that one
    heads = max(1, min(heads, most // (batch * queries * keys)))
    c = case("", batch, heads, queries, keys, rng.choice(PRESETS), rng.choice(("bfloat16", "bfloat16", "float16")),
             "bhnd" if host else rng.choice(("bhnd", "bnhd")), not cross and not host and rng.random() < 0.3, host, rng.choice(("plain", "uneven")))
    del c["name"]
    return c


@functools.lru_cache(maxsize=1)
def _rope_table(tokens):
    """A rotation per token and pair of channels, float32 [1, tokens, 1, 64, 2, 2]: one table serves every layer and step
    of a model, so a program makes it once per latent size and keeps it."""
    pair = torch.arange(HEAD_DIM // 2, device="cuda", dtype=torch.float64) / (HEAD_DIM // 2)
    angle = torch.arange(tokens, device="cuda", dtype=torch.float64)[:, None] * 10000.0**-pair
    cos, sin = angle.cos().float(), angle.sin().float()
    return torch.stack([torch.stack([cos, -sin], -1), torch.stack([sin, cos], -1)], -2)[None, :, None].contiguous()


def _tensor(c, kind, tokens, gen):
    """q (0), k (1) or v (2) of a case."""
    batch, heads = c["batch"], c["heads"]
    bnhd = c["layout"] == "bnhd"
    shape = (batch, tokens, heads, HEAD_DIM) if bnhd else (batch, heads, tokens, HEAD_DIM)
    x = torch.randn(shape, device="cuda", dtype=getattr(torch, c["dtype"]), generator=gen)
    x = x.transpose(1, 2) if bnhd else x  # [batch, heads, tokens, 128] either way
    per_head = (1, heads, 1, HEAD_DIM)
    if kind == 1:
        x += 0.5 * torch.randn(per_head, device="cuda", generator=gen)
    if c["values"] == "uneven":
        if kind < 2:
            x *= torch.exp(0.4 * torch.randn(per_head, device="cuda", generator=gen))
        if kind == 0:
            drift = torch.linspace(0, 1, tokens, device="cuda")[:, None]
            x += drift * torch.randn(per_head, device="cuda", generator=gen)
        if kind == 2:
            first, last = tokens // 2, tokens - tokens // 2  # one token in either half: two different ones
            x[:, :, torch.randint(first, (1,), device="cuda", generator=gen)] *= 65.0
            x[:, :, first + torch.randint(last, (1,), device="cuda", generator=gen)] *= 250.0
    return x


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v = (_tensor(case, kind, case["keys"] if kind else case["queries"], gen) for kind in range(3))
    settings = dict(unica.PRESETS[case["preset"]])
    if case["host"]:
        pinned = []
        for x in (q, k, v, q):
            pinned.append(torch.empty(x.shape, dtype=x.dtype, pin_memory=True))
            pinned[-1].copy_(x)
        return {"host": True, "tensors": pinned[:3], "out": pinned[3], "settings": settings}
    if case["rope"]:
        settings["rope"] = _rope_table(case["keys"])
    return {"host": False, "tensors": [q, k, v], "settings": settings}


def run(state):
    if state["host"]:
        return unica.attention_host(*state["tensors"], out=state["out"], **state["settings"])
    return unica.attention(*state["tensors"], **state["settings"])


def work(case):
    rows = case["batch"] * case["heads"]
    # q, k and v read, the output written, two bytes an element; a cosine and a sine in half precision per pair for RoPE
    read_write = 2 * rows * HEAD_DIM * (2 * case["queries"] + 2 * case["keys"]) + (2 * HEAD_DIM * case["keys"] if case["rope"] else 0)
    return {"bytes": read_write, "flops": 4 * rows * case["queries"] * case["keys"] * HEAD_DIM}


def tolerance(case):
    # 16-bit results.  Accurate: probabilities and V in 8 bits, a code at a rounding boundary may fall either way.  Fast:
    # probabilities in 4 bits, where such a code is a step of a fifth to a third and a row's few largest weights carry it.
    return {"rel": 1e-2, "max": 0.6} if case["preset"] == "fast" else {"rel": 5e-3, "max": 0.2}
