"""Performance cases of the attention path: what a user's program has it do, through the public entry points.

A case is a dict of plain values whose ``kind`` names the call; ``listed()`` gives fixed ones, ``draw(rng)``
one more of the same ranges.  ``prepare`` makes the inputs of a case, ``run`` is one pass, ``work`` the bytes
and operations one pass cannot do without, ``tolerance`` how far another correct implementation may be.

Kinds
  prefill       ops.sdpa_prefill: no mask / causal / causal window, optional fused output gate
  canvas        ops.gqa_attention_sdpa: canvas queries over cached prompt + canvas, no mask, scale 1
  masked        ops.fill_causal_mask + ops.gqa_attention_sdpa with the mask buffer: sliding encoder layers
  vision        ops.batched_attention with vision-block ids
  decode        ops.sdpa_decode over a batch of sequences of different length
  decode_one    ops.qwen35_xmx_attention_decode_gqa: one token of one sequence, gated
  decode_slide  ops.gemma4_sliding_decode_attention: one token over a slice of the cache
  prepare       ops.qkv_prepare: norms, rotation and cache append of a prompt chunk
  prepare_qwen  ops.qkv_prepare, multi-axis rotation on part of the head, V appended as it is
"""
import math
import random

import torch

from arcaine_b200 import ops

DEVICE = "cuda"


def listed():
    return [
        # The smallest attention call of the benchmark's configurations: one short bidirectional sequence.
        dict(name="single_op", kind="prefill", batch=1, seq=512, kv=512, nq=8, nkv=4, hd=128, causal=False, window=0,
             gate=False),
        # One denoising step of block diffusion: a 256-token canvas over a 2048-token cached prompt; a
        # generation runs it tens of times per layer and block.
        dict(name="canvas_step", kind="canvas", seq=256, prompt=2048, nq=16, nkv=8, hd=256),
        # Prompt processing of sliding-window layers, a full batch: the largest contraction.
        dict(name="window_prefill", kind="prefill", batch=4, seq=8192, kv=8192, nq=32, nkv=16, hd=128, causal=True,
             window=1024, gate=False),
        # A chunk of a long prompt at head dim 256 behind a ragged past, with the fused sigmoid output gate.
        dict(name="gated_chunk", kind="prefill", batch=1, seq=2048, kv=5049, nq=24, nkv=4, hd=256, causal=True, window=0,
             gate=True),
        # A sliding encoder layer that goes through the additive mask buffer, as the two calls a layer makes.
        dict(name="masked_encoder", kind="masked", seq=1000, past=300, nq=16, nkv=8, hd=256, window=1024),
        # A prompt with images: bidirectional inside each image's tokens, causal with a window elsewhere.
        dict(name="vision_prompt", kind="vision", seq=1531, past=0, nq=16, nkv=8, hd=256, window=1024, images=3, image=256),
        # One user's chat at a small depth: the latency of a token's attention, gate fused.
        dict(name="decode_one", kind="decode_one", past=512, nq=24, nkv=4, hd=256),
        # A handful of requests of different length in one cache block each.
        dict(name="decode_few", kind="decode", batch=12, lo=200, hi=6000, lengths=7, packed=False, nq=16, nkv=2, hd=128,
             gate=False),
        # A serving batch: 64 sequences of 1 K to 32 K keys in one packed cache, gated.
        dict(name="decode_batch", kind="decode", batch=64, lo=1024, hi=32768, lengths=4, packed=True, nq=24, nkv=4, hd=256,
             gate=True),
        # Long context: four sequences of half a million keys.
        dict(name="decode_long", kind="decode", batch=4, lo=524288, hi=524288, lengths=0, packed=False, nq=16, nkv=2, hd=128,
             gate=False),
        # What comes before the attention of window_prefill: norms, rotation, cache append.
        dict(name="prepare_prompt", kind="prepare", batch=4, seq=8192, past=0, nq=32, nkv=16, hd=128, partial=1.0, tables=False),
        # The same for one new token of each sequence of a serving batch, multi-axis rotation.
        dict(name="prepare_tokens", kind="prepare_qwen", batch=64, seq=1, past=777, nq=24, nkv=4, hd=256, rotary=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


#: (query heads, KV heads, head dim) of the configurations, the tests and the bench program
HEADS = [(8, 4, 128), (16, 8, 256), (32, 16, 128), (24, 4, 256), (16, 2, 128), (28, 4, 128), (16, 8, 128), (8, 2, 256)]
#: most operations of a drawn prefill, most bytes of a drawn decode: under what the largest listed cases take
MOST_FLOPS = 1.2e11
MOST_BYTES = 3.0e9


def draw(rng: random.Random):
    kind = rng.choice(["prefill", "prefill", "prefill", "canvas", "masked", "vision", "decode", "decode", "decode",
                       "decode_one", "decode_slide", "prepare", "prepare_qwen"])
    if kind == "prefill":
        nq, nkv, hd = rng.choice(HEADS)
        causal = rng.random() < 0.7
        c = dict(kind=kind, batch=rng.choice([1, 1, 2, 4]), seq=_log(rng, 32, 8192), kv=0, nq=nq, nkv=nkv, hd=hd, causal=causal,
                 window=_log(rng, 128, 4096) if causal and rng.random() < 0.5 else 0, gate=hd == 256 and rng.random() < 0.5)
        c["kv"] = c["seq"] + (_log(rng, 1, 8192) if rng.random() < 0.5 else 0)
        while work(c)["flops"] > MOST_FLOPS:  # fewer queries, the rest of the call as it is
            past = c["kv"] - c["seq"]
            c["seq"] = max(32, int(c["seq"] * 0.8))
            c["kv"] = c["seq"] + past
        return c
    if kind == "canvas":
        nq, nkv = rng.choice([(16, 8), (8, 4), (16, 2)])
        return dict(kind=kind, seq=rng.choice([64, 128, 256, 256, 512]), prompt=_log(rng, 64, 8192), nq=nq, nkv=nkv, hd=256)
    if kind == "masked":
        return dict(kind=kind, seq=_log(rng, 64, 2048), past=rng.choice([0, _log(rng, 16, 2048)]), nq=16, nkv=8, hd=256,
                    window=rng.choice([512, 1024]))
    if kind == "vision":
        images, image = rng.randint(1, 4), rng.choice([64, 196, 256])
        return dict(kind=kind, seq=images * image + _log(rng, 64, 2048), past=rng.choice([0, _log(rng, 16, 1024)]), nq=16, nkv=8,
                    hd=rng.choice([128, 256]), window=rng.choice([512, 1024]), images=images, image=image)
    if kind == "decode":
        nq, nkv, hd = rng.choice(HEADS)
        c = dict(kind=kind, batch=_log(rng, 1, 64), lo=0, hi=_log(rng, 128, 131072), lengths=rng.randrange(1 << 20),
                 packed=rng.random() < 0.5, nq=nq, nkv=nkv, hd=hd, gate=rng.random() < 0.5)
        row = 4 * nkv * hd
        c["hi"] = max(64, min(c["hi"], int(MOST_BYTES / (row * c["batch"]))))
        c["lo"] = max(1, int(c["hi"] * rng.choice([0.05, 0.3, 1.0])))
        return c
    if kind == "decode_one":
        return dict(kind=kind, past=_log(rng, 16, 32768), nq=24, nkv=4, hd=256)
    if kind == "decode_slide":
        return dict(kind=kind, start=_log(rng, 1, 8192), kv=_log(rng, 32, 1024), nq=16, nkv=8, hd=256)
    if kind == "prepare":
        nq, nkv, hd = rng.choice(HEADS)
        return dict(kind=kind, batch=rng.choice([1, 1, 2, 4]), seq=_log(rng, 1, 4096), past=rng.choice([0, _log(rng, 1, 4096)]),
                    nq=nq, nkv=nkv, hd=hd, partial=rng.choice([1.0, 1.0, 0.25]), tables=rng.random() < 0.5)
    batch, seq = rng.choice([(1, _log(rng, 1, 4096)), (_log(rng, 1, 64), 1)])
    return dict(kind=kind, batch=batch, seq=seq, past=_log(rng, 1, 4096), nq=24, nkv=4, hd=256, rotary=64)


# ---------------------------------------------------------------------------
# Shapes that follow from a case
# ---------------------------------------------------------------------------
def _lengths(c):
    """Keys of every sequence of a decode batch, uniform in [lo, hi]."""
    r = random.Random(c["lengths"])
    return [r.randint(c["lo"], c["hi"]) for _ in range(c["batch"])]


def _block_ids(c):
    """Ids by absolute position: images of `image` tokens, spread evenly over the chunk, text (-1) between."""
    ids = [-1] * (c["past"] + c["seq"])
    gap = (c["seq"] - c["images"] * c["image"]) // (c["images"] + 1)
    for i in range(c["images"]):
        at = c["past"] + gap + i * (gap + c["image"])
        ids[at:at + c["image"]] = [i] * c["image"]
    return ids


def _pairs(seq, kv, causal, window, ids=None):
    """(query, key) pairs of one head that are not masked out; query i sits at position kv - seq + i."""
    if not causal:
        return seq * kv
    n, end = 0, {}
    for j, b in enumerate(ids or ()):
        if b >= 0:
            end[b] = j + 1
    for i in range(seq):
        at = kv - seq + i
        hi = end.get(ids[at], at + 1) if ids else at + 1
        n += max(0, hi - (max(0, at + 1 - window) if window else 0))
    return n


def work(case):
    c, kind = case, case["kind"]
    nq, nkv, hd = c["nq"], c["nkv"], c["hd"]
    if kind in ("prefill", "canvas", "masked", "vision"):
        batch, seq = c.get("batch", 1), c["seq"]
        kv = c["kv"] if kind == "prefill" else seq + c["prompt" if kind == "canvas" else "past"]
        causal, window = kind in ("masked", "vision") or c.get("causal", False), c.get("window", 0)
        ids = _block_ids(c) if kind == "vision" else None
        seen = min(kv, seq + window - 1) if causal and window else kv
        nbytes = batch * 2 * hd * (seq * nq * (3 if c.get("gate") else 2) + 2 * seen * nkv)
        if kind == "masked":
            nbytes += 2 * 4 * seq * kv  # the buffer: written by one call, read by the other
        return {"bytes": nbytes, "flops": 4.0 * hd * nq * batch * _pairs(seq, kv, causal, window, ids)}
    if kind in ("decode", "decode_one", "decode_slide"):
        keys = sum(_lengths(c)) if kind == "decode" else c["past"] + 1 if kind == "decode_one" else c["kv"]
        gate = kind == "decode_one" or c.get("gate", False)
        return {"bytes": 4 * keys * nkv * hd + c.get("batch", 1) * nq * hd * 2 * (3 if gate else 2), "flops": 4.0 * hd * nq * keys}
    rows = c["batch"] * c["seq"]
    tables = 8 * c["seq"] * int(c["partial"] * hd / 2) if c.get("tables") else 0
    return {"bytes": 2 * 2 * rows * (nq + 2 * nkv) * hd + tables, "flops": 8.0 * rows * (nq + nkv) * hd}


def tolerance(case):
    return {"rel": 1e-2}  # bf16 results; probabilities in bf16


# ---------------------------------------------------------------------------
# Inputs: N(0, 1) bf16 drawn on the device, norm weights near one
# ---------------------------------------------------------------------------
def prepare(case, seed):
    g = torch.Generator(device=DEVICE).manual_seed(seed)

    def rnd(*shape, by=1.0):
        t = torch.randn(*shape, generator=g, device=DEVICE, dtype=torch.bfloat16)
        return t if by == 1.0 else t.mul_(by)

    s = dict(case)
    kind, nq, nkv, hd = case["kind"], case["nq"], case["nkv"], case["hd"]
    if kind == "prefill":
        s["q"] = rnd(case["batch"], case["seq"], nq, hd)
        s["k"], s["v"] = rnd(case["batch"], case["kv"], nkv, hd), rnd(case["batch"], case["kv"], nkv, hd)
        s["g"] = rnd(case["batch"], case["seq"], nq, hd) if case["gate"] else None
        s["out"] = torch.empty_like(s["q"])
    elif kind in ("canvas", "masked", "vision"):
        kv = case["seq"] + case["prompt" if kind == "canvas" else "past"]
        s["kv"] = kv
        # these layers use no scale: their Q comes out of a norm whose weight is what keeps the scores small
        s["q"], s["k"], s["v"] = rnd(case["seq"], nq, hd, by=hd ** -0.5), rnd(kv, nkv, hd), rnd(kv, nkv, hd)
        if kind == "masked":
            s["mask"] = torch.empty(case["seq"], kv, device=DEVICE, dtype=torch.float32)
        if kind == "vision":
            s["ids"] = torch.tensor(_block_ids(case), dtype=torch.int32, device=DEVICE)
    elif kind == "decode":
        lens = _lengths(case)
        s["q"], s["out"] = rnd(case["batch"], nq, hd), torch.empty(case["batch"], nq, hd, device=DEVICE, dtype=torch.bfloat16)
        s["g"] = rnd(case["batch"], nq, hd) if case["gate"] else None
        shape = (sum(lens),) if case["packed"] else (case["batch"], max(lens))
        s["k"], s["v"] = rnd(*shape, nkv, hd), rnd(*shape, nkv, hd)
        s["lens"] = torch.tensor(lens, dtype=torch.int32, device=DEVICE)
        s["rows"] = torch.tensor([sum(lens[:b]) for b in range(len(lens))], dtype=torch.int64, device=DEVICE) \
            if case["packed"] else None
    elif kind == "decode_one":
        s["q"], s["g"] = rnd(nq, hd), rnd(nq, hd)
        s["k"], s["v"] = rnd(case["past"] + 64, nkv, hd), rnd(case["past"] + 64, nkv, hd)
        s["out"] = torch.empty_like(s["q"])
    elif kind == "decode_slide":
        rows = case["start"] + case["kv"]
        s["q"], s["k"], s["v"] = rnd(nq, hd, by=hd ** -0.5), rnd(rows, nkv, hd), rnd(rows, nkv, hd)
    else:
        rows = (case["batch"], case["seq"])
        s["q"], s["k"], s["v"] = rnd(*rows, nq, hd), rnd(*rows, nkv, hd), rnd(*rows, nkv, hd)
        capacity = case["past"] + case["seq"] + 16
        s["kc"], s["vc"] = (torch.zeros(case["batch"], capacity, nkv, hd, device=DEVICE, dtype=torch.bfloat16) for _ in range(2))
        s["qw"], s["kw"] = rnd(hd, by=0.1).add_(1.0), rnd(hd, by=0.1).add_(1.0)
        if case.get("tables"):
            pairs = int(case["partial"] * hd / 2)
            inv = 10000.0 ** (-2.0 * torch.arange(pairs, device=DEVICE, dtype=torch.float32) / hd)
            at = torch.arange(case["past"], case["past"] + case["seq"], device=DEVICE, dtype=torch.float32)
            angle = at[:, None] * inv[None]
            s["cos"], s["sin"] = angle.cos().contiguous(), angle.sin().contiguous()
        if kind == "prepare_qwen":
            at = torch.arange(case["past"], case["past"] + case["seq"], dtype=torch.int32, device=DEVICE)
            s["positions"] = at.expand(case["batch"], 3, case["seq"]).contiguous()
    return s


def run(state):
    s, kind = state, state["kind"]
    if kind == "prefill":
        return ops.sdpa_prefill(s["q"], s["k"], s["v"], scale=s["hd"] ** -0.5,
                                mask_type=ops.MASK_CAUSAL if s["causal"] else ops.MASK_NONE,
                                window=s["window"] or ops.NO_WINDOW, gate=s["g"], out=s["out"])
    if kind == "canvas":
        return ops.gqa_attention_sdpa(s["q"], s["seq"], s["nq"], s["hd"], s["k"], s["v"], s["kv"], s["nkv"])
    if kind == "masked":
        mask = ops.fill_causal_mask(s["seq"], s["kv"], s["past"], s["window"], out=s["mask"])
        return mask, ops.gqa_attention_sdpa(s["q"], s["seq"], s["nq"], s["hd"], s["k"], s["v"], s["kv"], s["nkv"], mask,
                                            ops.MASK_EXPLICIT)
    if kind == "vision":
        return ops.batched_attention(s["q"], s["seq"], s["nq"], s["hd"], s["k"], s["v"], s["kv"], s["nkv"], s["hd"], s["past"],
                                     s["window"], block_ids=s["ids"])
    if kind == "decode":
        return ops.sdpa_decode(s["q"], s["k"], s["v"], scale=s["hd"] ** -0.5, kv_len=s["lens"], kv_row_offset=s["rows"],
                               gate=s["g"], out=s["out"])
    if kind == "decode_one":
        return ops.qwen35_xmx_attention_decode_gqa(s["q"], s["k"], s["v"], s["out"], s["past"], s["nq"], s["nkv"], s["hd"],
                                                   s["hd"] ** -0.5, gate=s["g"])
    if kind == "decode_slide":
        return ops.gemma4_sliding_decode_attention(s["q"], s["k"], s["v"], s["kv"], s["start"], s["nq"], s["nkv"], s["hd"])
    end = s["past"] + s["seq"]
    if kind == "prepare":
        ops.qkv_prepare(s["q"], s["k"], s["v"], k_cache=s["kc"], v_cache=s["vc"], past_len=s["past"], q_weight=s["qw"],
                        k_weight=s["kw"], eps=1e-6, partial_rotary_factor=s["partial"], rope_cos=s.get("cos"),
                        rope_sin=s.get("sin"))
    else:
        ops.qkv_prepare(s["q"], s["k"], s["v"], k_cache=s["kc"], v_cache=s["vc"], past_len=s["past"], q_weight=s["qw"],
                        k_weight=s["kw"], eps=1e-6, theta=1e6, rotary_dim=s["rotary"], mrope_positions=s["positions"],
                        mrope_section=(11, 11, 10), v_copy=True)
    return s["q"], s["kc"][:, s["past"]:end], s["vc"][:, s["past"]:end]
