"""Parity of the sm_100a prefill / canvas kernel with the CPU oracle, through the C ABI."""
import ctypes as C

import pytest
import torch

from helpers import assert_close, seeded_bf16
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from arcaine_b200 import ops as o
    o.clear_device_status()
    yield o
    assert o.device_status() == (0, 0), "a bounded device-side wait gave up during the prefill tests"


def run_case(ops, seq, kv_len, nq, nkv, hd, scale, mask_type, window, seed, num_splits=0, gate=False, lse=False):
    q, k, v = seeded_bf16(seq, nq, hd, seed=seed), seeded_bf16(kv_len, nkv, hd, seed=seed + 1), \
        seeded_bf16(kv_len, nkv, hd, seed=seed + 2)
    g = seeded_bf16(seq, nq, hd, seed=seed + 3) if gate else None
    res = ops.sdpa_prefill(q.cuda(), k.cuda(), v.cuda(), scale=scale, mask_type=mask_type, window=window,
                           num_splits=num_splits, gate=g.cuda() if gate else None, return_lse=lse)
    want = oracle.sdpa_f32(q, k, v, scale=scale, mask_type=mask_type, window=window, gate=g, want_lse=lse)
    if lse:
        assert_close(res[0], want[0], "out")
        finite = torch.isfinite(want[2])
        assert torch.equal(torch.isfinite(res[1].cpu()), finite)
        assert torch.allclose(res[1].cpu()[finite], want[2][finite], atol=2e-3)
    else:
        assert_close(res, want[0], f"S{seq} L{kv_len} nq{nq}/{nkv} hd{hd} mask{mask_type} w{window}")


@pytest.mark.parametrize("hd", [128, 256])
@pytest.mark.parametrize("mask_type,window", [(0, oracle.INT_MAX), (3, oracle.INT_MAX), (3, 100), (3, 1)])
def test_single_sequence(ops, hd, mask_type, window):
    run_case(ops, 300, 300, 8, 4, hd, hd ** -0.5, mask_type, window, seed=100 + hd)


@pytest.mark.parametrize("seq,kv_len", [(1, 1), (1, 129), (77, 300), (128, 128), (129, 127), (130, 1000), (200, 517)])
@pytest.mark.parametrize("mask_type,window", [(0, oracle.INT_MAX), (3, oracle.INT_MAX), (3, 64)])
def test_ragged_shapes(ops, seq, kv_len, mask_type, window):
    # includes kv_len < seq with bottom-right causal: leading queries see no key and must be zero
    run_case(ops, seq, kv_len, 4, 2, 128, 0.09, mask_type, window, seed=seq * 7 + kv_len, lse=True)


def test_config1_cpu_runnable_case(ops):
    """B1, 8Q/4KV, hd128, seq 512, non-causal, scale 1/sqrt(128)."""
    run_case(ops, 512, 512, 8, 4, 128, 128 ** -0.5, 0, oracle.INT_MAX, seed=1)


@pytest.mark.parametrize("scale", [1.0, 256 ** -0.5])
def test_config2_canvas_over_prompt_steps(ops, scale):
    """DiffusionGemma denoising steps: 2048 cached prompt rows + a 256-row canvas written at the cache
    tail each step (src/modeling/diffusion_gemma/attention.cpp:1079-1103), all 32 steps
    (src/modeling/diffusion_gemma/generate.cpp:123): every output row of the first and the last step,
    every fifth row of the others.  Scale 1.0 is what the reference runs, 1/sqrt(256) the conditioned
    variant."""
    nq, nkv, hd, prompt, canvas, steps = 16, 8, 256, 2048, 256, 32
    kc = torch.empty(prompt + canvas, nkv, hd, dtype=torch.bfloat16)
    vc = torch.empty_like(kc)
    kc[:prompt], vc[:prompt] = seeded_bf16(prompt, nkv, hd, seed=2000), seeded_bf16(prompt, nkv, hd, seed=2001)
    kd, vd = kc.cuda(), vc.cuda()
    prompt_k, prompt_v = kd[:prompt].clone(), vd[:prompt].clone()
    worst = 0.0
    for step in range(steps):
        q = seeded_bf16(canvas, nq, hd, seed=2100 + step)
        kc[prompt:], vc[prompt:] = seeded_bf16(canvas, nkv, hd, seed=2200 + step), seeded_bf16(canvas, nkv, hd, seed=2300 + step)
        kd[prompt:].copy_(kc[prompt:])
        vd[prompt:].copy_(vc[prompt:])
        got = ops.gqa_attention_sdpa(q.cuda(), canvas, nq, hd, kd, vd, prompt + canvas, nkv) if scale == 1.0 else \
            ops.sdpa_prefill(q.cuda(), kd, vd, scale=scale)
        rows = list(range(canvas * nq)) if step in (0, steps - 1) else list(range(step % 5, canvas * nq, 5))
        want, _ = oracle.sdpa_f32(q, kc, vc, scale=scale, rows=rows)
        rel, _ = assert_close(got.reshape(-1, hd)[rows], want, f"step {step}")
        worst = max(worst, rel)
    assert worst < 5e-3  # the tolerance is 1e-2; the steps sit well inside it
    # the prompt rows of the cache are read, never written
    assert torch.equal(kd[:prompt], prompt_k) and torch.equal(vd[:prompt], prompt_v)


@pytest.mark.parametrize("splits", [1, 2, 3, 5, 0])
def test_key_range_splits_agree(ops, splits):
    run_case(ops, 256, 1100, 4, 2, 256, 0.0625, 3, 700, seed=31, num_splits=splits, lse=True)


@pytest.mark.parametrize("hd", [128, 256])
@pytest.mark.parametrize("seq,kv_len,nq,nkv,mask_type,window,parts", [
    # (parts: what head dim 128 takes; 256 chooses by units of two tiles)
    (256, 1300, 28, 4, 0, oracle.INT_MAX, 2),   # 56 tiles on 148 SMs, 11 key blocks: two parts
    (200, 1300, 28, 4, 3, 300, 2),              # the same ragged and windowed: parts without keys
    (256, 2100, 16, 8, 0, oracle.INT_MAX, 4),   # 32 tiles, 17 key blocks (the last one ragged): four parts
    (130, 2100, 16, 2, 3, 100, 4),              # 32 tiles, a window: most parts see no key
    (130, 2100, 4, 2, 0, oracle.INT_MAX, 8),    # 8 tiles: eight parts, always two launches
    (256, 1200, 8, 4, 3, oracle.INT_MAX, 5),    # 16 tiles, 10 key blocks: five parts, two launches
])
def test_key_range_splits_the_library_chooses(ops, hd, seq, kv_len, nq, nkv, mask_type, window, parts):
    """Splits the library chooses itself: at head dim 256 few parts run as one thread-block cluster per unit that folds
    them itself (one launch), or none at all; everything else as partial records and a merge launch.  With the gate
    and the log-sum-exp output."""
    before = ops.launch_count()
    run_case(ops, seq, kv_len, nq, nkv, hd, hd ** -0.5, mask_type, window, seed=500 + hd + seq, gate=True, lse=True)
    torch.cuda.synchronize()
    assert ops.launch_count() - before == (1 if hd == 256 and parts in (2, 4) else 2)
    run_case(ops, seq, kv_len, nq, nkv, hd, hd ** -0.5, mask_type, window, seed=600 + hd + seq)


@pytest.mark.parametrize("case", ["hd128", "single", "cluster", "two_launch", "nothing_visible"])
def test_output_copies_are_written_by_every_epilogue(ops, case):
    """out_copies: further buffers that receive the same rows at the same offsets (other GPUs' buffers when
    a head-sharded output is gathered; here two more buffers on the same device), through every kernel
    that writes output."""
    seq, kv, nq, nkv, hd, mask, win, splits = {
        "hd128": (1024, 1024, 8, 4, 128, 3, 256, 0),         # (the two-tile kernel's copies: test_prefill_pair_gpu.py)
        "single": (300, 300, 4, 2, 256, 3, oracle.INT_MAX, 1),
        "cluster": (256, 2100, 16, 8, 256, 0, oracle.INT_MAX, 0),    # 16 units, 17 key blocks: three parts, folded in a cluster
        "two_launch": (256, 1200, 4, 2, 128, 0, oracle.INT_MAX, 3),
        "nothing_visible": (200, 100, 4, 2, 128, 3, oracle.INT_MAX, 0),  # the first 100 queries see no key
    }[case]
    q, k, v = seeded_bf16(seq, nq, hd, seed=700), seeded_bf16(kv, nkv, hd, seed=701), seeded_bf16(kv, nkv, hd, seed=702)
    g = seeded_bf16(seq, nq, hd, seed=703)
    plain = ops.sdpa_prefill(q.cuda(), k.cuda(), v.cuda(), scale=hd ** -0.5, mask_type=mask, window=win,
                             num_splits=splits, gate=g.cuda())
    # the copies sit inside a wider buffer (a head slice of a full-width output), like the gathered layout
    wide = [torch.full((seq, 2 * nq, hd), 9.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    out = torch.empty(seq, 2 * nq, hd, dtype=torch.bfloat16, device="cuda")[:, nq:]
    copies = torch.tensor([w[:, nq:].data_ptr() for w in wide], dtype=torch.int64, device="cuda")
    gate_wide = torch.empty(seq, 2 * nq, hd, dtype=torch.bfloat16, device="cuda")[:, nq:]  # laid out like out
    gate_wide.copy_(g)
    got = ops.sdpa_prefill(q.cuda(), k.cuda(), v.cuda(), scale=hd ** -0.5, mask_type=mask, window=win,
                           num_splits=splits, gate=gate_wide, out=out, out_copies=copies)
    torch.cuda.synchronize()
    assert torch.equal(got, plain)
    for w in wide:
        assert torch.equal(w[:, nq:], plain) and (w[:, :nq].float() == 9.0).all()


@pytest.mark.parametrize("gate", [False, True])
def test_windowed_pairs_worth_of_tiles_in_one_launch(ops, gate):
    """13 token tiles of 32 heads: 208 pairs of tiles on 148 SMs, but so few key blocks in each that one launch of single
    tiles, dealt longest first, is judged faster than pairs with or without a tail."""
    before = ops.launch_count()
    run_case(ops, 1664, 1664, 32, 16, 128, 128 ** -0.5, 3, 300, seed=800, gate=gate, lse=True)
    assert ops.launch_count() - before == 1


# Calls that are cut by a clear margin (5 % and more) into whole waves of two-tile CTAs and a second launch for the pairs left
# over, one CTA for each of their tiles: batch, queries, keys, heads, KV heads, causal, vision blocks.
CUT = [
    (3, 1590, 1700, 32, 16, False, False),  # 624 pairs in plain order: the last 32, heads 26 to 31 of the last sequence
    (4, 1650, 4700, 24, 4, True, False),    # 624 longest first: the first token tile of all sequences but the first
    (4, 1650, 4700, 24, 4, True, True),
]


def cut_call(B, seq, kv, nq, nkv, causal, vision, seed):
    g = torch.Generator().manual_seed(seed)
    q, k, v, gate = (torch.randn(B, n, h, 128, generator=g).bfloat16() for n, h in ((seq, nq), (kv, nkv), (kv, nkv), (seq, nq)))
    ids = None
    if vision:  # one that starts in the past, one across the first two tiles, one up to the last key
        ids = torch.full((kv,), -1, dtype=torch.int32)
        for i, (a, b) in enumerate([(kv - seq - 50, kv - seq + 30), (kv - seq + 100, kv - seq + 300), (kv - 90, kv)]):
            ids[a:b] = i
    return q, k, v, gate, ids


@pytest.mark.parametrize("with_gate", [False, True])
@pytest.mark.parametrize("B,seq,kv,nq,nkv,causal,vision", CUT)
def test_two_tile_launch_with_a_single_head_tail(ops, B, seq, kv, nq, nkv, causal, vision, with_gate):
    """Every row must come out exactly once, from either launch: all rows against the same call in parts of the key range
    (single tiles and a merge), one in 61 — all heads, all tiles — against the oracle; with the log-sum-exp and an output copy."""
    q, k, v, gate, ids = cut_call(B, seq, kv, nq, nkv, causal, vision, seed=820)
    dev = [t.cuda() for t in (q, k, v)]
    args = dict(scale=128 ** -0.5, mask_type=3 if causal else 0, gate=gate.cuda() if with_gate else None, block_ids=ids.cuda() if vision else None,
                return_lse=True)
    copy = torch.zeros(B, seq, nq, 128, dtype=torch.bfloat16, device="cuda")
    before = ops.launch_count()
    out, lse = ops.sdpa_prefill(*dev, out_copies=torch.tensor([copy.data_ptr()], dtype=torch.int64, device="cuda"), **args)
    assert ops.launch_count() - before == 2
    assert torch.equal(copy, out)
    parts, parts_lse = ops.sdpa_prefill(*dev, num_splits=2, **args)
    # (both within half a rounding of bf16 of their own result, as in the comparison of vision blocks below)
    assert_close(out, parts.float(), "parts", rel_tol=4e-3, abs_tol=1.6e-2)
    assert torch.allclose(lse, parts_lse, atol=2e-3)
    mask = oracle.fill_causal_mask_with_block_ids(ids.numpy(), seq, kv, kv - seq, oracle.INT_MAX) if vision else None
    rows = list(range(0, seq * nq, 61))
    for b in range(B):
        want = oracle.sdpa_f32(q[b], k[b], v[b], scale=128 ** -0.5, mask_type=1 if vision else args["mask_type"], mask=mask,
                               gate=gate[b] if with_gate else None, rows=rows, want_lse=True)
        assert_close(out[b].reshape(-1, 128)[rows], want[1].float() if with_gate else want[0], f"sequence {b}")
        assert torch.allclose(lse[b].cpu().reshape(-1)[rows], want[2], atol=2e-3)


@pytest.mark.parametrize("with_gate", [False, True])
@pytest.mark.parametrize("B,seq,kv,nq,nkv,causal,vision", CUT)
def test_consumer_right_behind_the_two_launch_form_sees_finished_rows(ops, B, seq, kv, nq, nkv, causal, vision, with_gate):
    """The single-head tail runs beside the two-tile launch in front of it; what follows in the stream waits for
    the tail launch only, so the tail must not complete first.  A copy enqueued right behind the call, with no
    host synchronisation in between, has to see every row."""
    q, k, v, gate, ids = cut_call(B, seq, kv, nq, nkv, causal, vision, seed=810)
    q, k, v = (t.cuda() for t in (q, k, v))
    args = dict(scale=128 ** -0.5, mask_type=3 if causal else 0, gate=gate.cuda() if with_gate else None, block_ids=ids.cuda() if vision else None)
    ref = ops.sdpa_prefill(q, k, v, **args).clone()
    torch.cuda.synchronize()
    for _ in range(20):
        out = torch.zeros_like(ref)
        before = ops.launch_count()
        ops.sdpa_prefill(q, k, v, out=out, **args)
        snap = out.clone()
        assert ops.launch_count() - before == 2
        torch.cuda.synchronize()
        assert torch.equal(snap, ref)


def test_gate_epilogue_and_split_gate(ops):
    run_case(ops, 150, 400, 6, 2, 256, 0.0625, 3, oracle.INT_MAX, seed=41, gate=True)
    run_case(ops, 150, 400, 6, 2, 256, 0.0625, 3, oracle.INT_MAX, seed=41, gate=True, num_splits=2)


def test_explicit_mask_equals_inline_rule(ops):
    seq, kv_len, nq, nkv, hd = 140, 260, 4, 2, 128
    q, k, v = seeded_bf16(seq, nq, hd, seed=51).cuda(), seeded_bf16(kv_len, nkv, hd, seed=52).cuda(), \
        seeded_bf16(kv_len, nkv, hd, seed=53).cuda()
    mask = ops.fill_causal_mask(seq, kv_len, past_offset=kv_len - seq, sliding_window=50)
    assert torch.equal(mask.cpu(), torch.from_numpy(oracle.fill_causal_mask(seq, kv_len, kv_len - seq, 50)))
    a = ops.sdpa_prefill(q, k, v, scale=0.1, mask_type=ops.MASK_EXPLICIT, mask=mask)
    b = ops.sdpa_prefill(q, k, v, scale=0.1, mask_type=ops.MASK_CAUSAL, window=50)
    assert_close(a, b.float(), "explicit vs inline", rel_tol=2e-3, abs_tol=4e-3)


def test_batched_strided_inputs_and_output_aliasing_query(ops):
    """batch 3 inside a larger cache allocation (token and batch strides), out written over q."""
    B, S, L, cap, nq, nkv, hd = 3, 140, 200, 256, 8, 4, 128
    q = seeded_bf16(B, S, nq, hd, seed=61)
    kc = seeded_bf16(B, cap, nkv, hd, seed=62)
    vc = seeded_bf16(B, cap, nkv, hd, seed=63)
    qd = q.cuda()
    out = ops.sdpa_prefill(qd, kc.cuda()[:, :L], vc.cuda()[:, :L], scale=0.09, mask_type=3, out=qd)
    assert out.data_ptr() == qd.data_ptr()
    for b in range(B):
        want, _ = oracle.sdpa_f32(q[b], kc[b, :L], vc[b, :L], scale=0.09, mask_type=3)
        assert_close(out[b], want, f"batch {b}")


def test_reference_named_entry_points(ops):
    seq, past, nq, nkv, hd = 130, 70, 8, 2, 256
    q, k, v = seeded_bf16(seq, nq, hd, seed=71), seeded_bf16(past + seq, nkv, hd, seed=72), seeded_bf16(past + seq, nkv, hd, seed=73)
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    # qwen35_xmx_attention: causal over past + seq keys, output aliasing the query buffer
    buf = qd.clone()
    ops.qwen35_xmx_attention(buf, kd, vd, buf, seq, past, nq, nkv, hd, 0.0625)
    assert_close(buf, oracle.qwen35_online_attention(q, k, v, seq=seq, past=past, scale=0.0625).float(), "qwen35")
    # gqa_attention: no scale; inputs scaled down so the softmax is not one-hot
    qs = (q.float() * 0.25).bfloat16()
    got = ops.gqa_attention(qs.cuda(), seq, nq, hd, kd, vd, past + seq, nkv, past, 64, True)
    want, _ = oracle.sdpa_f32(qs, k, v, scale=1.0, mask_type=3, window=64)
    assert_close(got, want, "gqa_attention")
    # the restated matmul path keeps scores and probabilities in bf16, so it is itself
    # ~5e-2 away from the fp32 oracle at these magnitudes; this is a sanity bound, not the gate
    assert_close(got, oracle.gqa_attention(qs, k, v, past_offset=past, sliding_window=64, causal=True).float(),
                 "gqa_attention vs its restatement", rel_tol=2e-2, abs_tol=1.5e-1)
    got = ops.batched_attention(q.cuda(), seq, nq, hd, kd, vd, past + seq, nkv, hd, past, oracle.INT_MAX, scale=0.0625)
    assert_close(got, oracle.batched_attention(q, k, v, past_offset=past, scale=0.0625).float(), "batched_attention",
                 rel_tol=2e-2, abs_tol=1.5e-1)
    assert_close(got, oracle.sdpa_f32(q, k, v, scale=0.0625, mask_type=3)[0], "batched_attention vs fp32 oracle")
    with pytest.raises(ValueError):  # block ids must cover every key position
        ops.batched_attention(q.cuda(), seq, nq, hd, kd, vd, past + seq, nkv, hd, past, oracle.INT_MAX,
                              block_ids=torch.zeros(1, dtype=torch.int32, device="cuda"))


def test_outputs_too_small_for_the_result_are_refused(ops):
    """The library is given addresses and strides: what it would write past its end has to be refused here.  Larger ones
    are filled from their start."""
    seq, nq, nkv, hd = 20, 4, 2, 128
    q, k = seeded_bf16(seq, nq, hd, seed=1).cuda(), seeded_bf16(seq, nkv, hd, seed=2).cuda()
    new = lambda *n: torch.zeros(*n, dtype=torch.bfloat16, device="cuda")  # noqa: E731
    want = ops.sdpa_prefill(q, k, k, scale=0.1)
    for small in (new(seq - 1, nq, hd), new(seq, nq - 1, hd), new(seq, nq, hd - 8)):
        with pytest.raises(ValueError):
            ops.sdpa_prefill(q, k, k, scale=0.1, out=small)
        with pytest.raises(ValueError):
            ops.sdpa_prefill(q, k, k, scale=0.1, out=small, gate=small.clone())
        with pytest.raises(ValueError):
            ops.gqa_attention_sdpa(q, seq, nq, hd, k, k, seq, nkv, out=small)
    with pytest.raises(ValueError):
        ops.sdpa_prefill(q[None].repeat(2, 1, 1, 1), k[None].repeat(2, 1, 1, 1), k[None].repeat(2, 1, 1, 1), scale=0.1, out=new(1, seq, nq, hd))
    with pytest.raises(ValueError):
        ops.qwen35_xmx_attention(q, k, k, new(seq - 1, nq, hd), seq, 0, nq, nkv, hd, 0.1)
    large = new(seq + 3, nq + 1, hd)
    ops.sdpa_prefill(q, k, k, scale=0.1, out=large)
    assert torch.equal(large[:seq, :nq], want) and not large[seq:].any() and not large[:, nq:].any()
    for fill in (lambda o: ops.fill_causal_mask(8, 16, 8, out=o), lambda o: ops.fill_causal_mask_with_block_ids(None, 8, 16, 8, out=o)):
        for bad in (torch.zeros(8, 15, device="cuda"), torch.zeros(16, 8, device="cuda").t()):
            with pytest.raises(ValueError):
                fill(bad)
        assert torch.equal(fill(torch.ones(9, 16, device="cuda"))[:8], ops.fill_causal_mask(8, 16, 8))


def test_caches_of_other_dimensions_stay_refused(ops):
    """One-dimensional caches belong to gqa_attention_sdpa; pre-processing takes all tensors with the same number of dims."""
    seq, nq, nkv, hd = 20, 4, 2, 128
    q, k = seeded_bf16(seq, nq, hd, seed=1).cuda(), seeded_bf16(seq, nkv, hd, seed=2).cuda()
    want = ops.gqa_attention_sdpa(q, seq, nq, hd, k, k, seq, nkv)
    assert torch.equal(ops.gqa_attention_sdpa(q, seq, nq, hd, k.flatten(), k.flatten(), seq, nkv), want)
    with pytest.raises(ValueError):
        ops.gqa_attention(q, seq, nq, hd, k.flatten(), k.flatten(), seq, nkv, 0, ops.NO_WINDOW, True)
    with pytest.raises(ValueError):
        ops.batched_attention(q, seq, nq, hd, k.flatten(), k.flatten(), seq, nkv, hd, 0, ops.NO_WINDOW)
    cache = torch.zeros(1, seq + 4, nkv, hd, dtype=torch.bfloat16, device="cuda")
    with pytest.raises((ValueError, IndexError)):
        ops.qkv_prepare(q, k, k.clone(), k_cache=cache, v_cache=cache.clone(), eps=1e-6, theta=1e4)
    with pytest.raises((ValueError, IndexError)):
        ops.qkv_prepare(q[None], k[None], k[None].clone(), k_cache=cache[0], v_cache=cache[0].clone(), eps=1e-6, theta=1e4)


def test_error_statuses(ops):
    from arcaine_b200 import _lib
    q = torch.zeros(8, 4, 64, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(ops.ArcError) as e:
        ops.sdpa_prefill(q, q, q, scale=1.0)
    assert e.value.status == _lib.ARC_ERR_UNSUPPORTED_HEAD_DIM
    q = torch.zeros(8, 6, 128, dtype=torch.bfloat16, device="cuda")
    k = torch.zeros(8, 4, 128, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(ops.ArcError) as e:
        ops.sdpa_prefill(q, k, k, scale=1.0)
    assert e.value.status == _lib.ARC_ERR_BAD_SHAPE
    q = torch.zeros(8, 4, 128, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(ops.ArcError) as e:
        ops.sdpa_prefill(q, k, k, scale=-1.0)
    assert e.value.status == _lib.ARC_ERR_BAD_SHAPE
    # raw ABI: misaligned pointer, missing workspace for a forced split
    p = _lib.PrefillParams()
    big = torch.zeros(600, 4, 128, dtype=torch.bfloat16, device="cuda")
    p.q = p.k = p.v = p.out = big.data_ptr()
    p.batch, p.seq, p.kv_len, p.nq, p.nkv, p.hd = 1, 600, 600, 4, 4, 128
    for f in ("q", "k", "v", "o"):
        setattr(p, f + "_stride_t", 512)
        setattr(p, f + "_stride_b", 600 * 512)
    p.scale, p.mask_type, p.window, p.num_splits = 1.0, 0, ops.NO_WINDOW, 2
    L = _lib.load()
    assert L.arc_sdpa_prefill(C.byref(p), None) == _lib.ARC_ERR_WORKSPACE_TOO_SMALL
    p.num_splits = 1
    p.q = big.data_ptr() + 2
    assert L.arc_sdpa_prefill(C.byref(p), None) == _lib.ARC_ERR_ALIGNMENT
    assert L.arc_sdpa_prefill(None, None) == _lib.ARC_ERR_NULL_POINTER


def test_vision_block_mask_buffer_and_attention(ops):
    """Gemma4 vision blocks: the mask kernel against its restatement (bit for bit), then attention through
    the explicit-mask path against the oracle with the same buffer."""
    import numpy as np
    seq, kv_len, past, nq, nkv, hd = 150, 230, 80, 4, 2, 128
    ids = np.full(past + seq, -1, dtype=np.int32)
    ids[70:100] = 0
    ids[140:200] = 1
    for window in (oracle.INT_MAX, 64):
        want_mask = oracle.fill_causal_mask_with_block_ids(ids, seq, kv_len, past, window)
        mask = ops.fill_causal_mask_with_block_ids(torch.from_numpy(ids).cuda(), seq, kv_len, past, window)
        assert np.array_equal(mask.cpu().numpy(), want_mask)
        q, k, v = seeded_bf16(seq, nq, hd, seed=71), seeded_bf16(kv_len, nkv, hd, seed=72), seeded_bf16(kv_len, nkv, hd, seed=73)
        out = ops.sdpa_prefill(q.cuda(), k.cuda(), v.cuda(), scale=hd ** -0.5, mask_type=ops.MASK_EXPLICIT, mask=mask)
        want = oracle.sdpa_f32(q, k, v, scale=hd ** -0.5, mask_type=1, mask=want_mask)
        assert_close(out, want[0], f"vision blocks, window {window}")
    plain = ops.fill_causal_mask_with_block_ids(None, seq, kv_len, past, 64, out=torch.empty(seq, kv_len, device="cuda"))
    assert torch.equal(plain, ops.fill_causal_mask(seq, kv_len, past, 64))


@pytest.mark.parametrize("hd", [128, 256])
def test_vision_block_ids_inside_the_kernel(ops, hd):
    """Gemma4 vision blocks evaluated in the attention kernel (no (seq, kv_len) buffer): against the oracle
    fed with the restated mask of src/common/kernels/attention_mask.hpp:44-73, with and without a window,
    a block that straddles query tiles and one that starts in the past; and through batched_attention."""
    import numpy as np
    seq, kv_len, nq, nkv = 300, 420, 4, 2
    past = kv_len - seq  # the cache holds every position from 0
    ids = np.full(kv_len, -1, dtype=np.int32)
    ids[100:190] = 0      # starts before the first query (position 120), ends inside the first tile
    ids[230:340] = 1      # straddles the first and second query tile
    ids[400:420] = 2      # runs to the end of the sequence
    ids_d = torch.from_numpy(ids).cuda()
    q, k, v = seeded_bf16(seq, nq, hd, seed=171), seeded_bf16(kv_len, nkv, hd, seed=172), seeded_bf16(kv_len, nkv, hd, seed=173)
    for window in (oracle.INT_MAX, 150):
        want_mask = oracle.fill_causal_mask_with_block_ids(ids, seq, kv_len, past, window)
        want = oracle.sdpa_f32(q, k, v, scale=hd ** -0.5, mask_type=1, mask=want_mask)
        out = ops.sdpa_prefill(q.cuda(), k.cuda(), v.cuda(), scale=hd ** -0.5, mask_type=ops.MASK_CAUSAL, window=window,
                               block_ids=ids_d)
        assert_close(out, want[0], f"block ids in the kernel, window {window}")
        plain = ops.sdpa_prefill(q.cuda(), k.cuda(), v.cuda(), scale=hd ** -0.5, mask_type=ops.MASK_CAUSAL, window=window)
        assert not torch.equal(plain, out)  # the blocks do change the result
    # the reference-named call: K holds only the last 350 positions, so key 0 sits at absolute position 70
    kv2 = 350
    got = ops.batched_attention(q.cuda(), seq, nq, hd, k.cuda()[kv_len - kv2:], v.cuda()[kv_len - kv2:], kv2, nkv, hd,
                                past, oracle.INT_MAX, scale=0.08, block_ids=ids_d)
    want_mask = oracle.fill_causal_mask_with_block_ids(ids, seq, kv2, past, oracle.INT_MAX)
    want = oracle.sdpa_f32(q, k[kv_len - kv2:], v[kv_len - kv2:], scale=0.08, mask_type=1, mask=want_mask)
    assert_close(got, want[0], "batched_attention with block ids")


def test_gemma4_decode_wrappers(ops):
    """sliding_decode_attention (src/modeling/gemma4_unified/attention.cpp:93-137) over rows
    [kv_start, kv_start + kv_len) of the token-major cache, and the nkv == 1 path (:274-288) with more than
    16 query heads on the one KV head; no scale."""
    nq, nkv, hd, max_seq, kv_start, kv_len = 16, 8, 256, 700, 123, 512
    q = (seeded_bf16(nq, hd, seed=181).float() * 0.25).bfloat16()
    kc, vc = (seeded_bf16(max_seq, nkv, hd, seed=182).float() * 0.25).bfloat16(), seeded_bf16(max_seq, nkv, hd, seed=183)
    got = ops.gemma4_sliding_decode_attention(q.cuda(), kc.cuda(), vc.cuda(), kv_len, kv_start, nq, nkv, hd)
    want, _ = oracle.sdpa_f32(q[None], kc[kv_start:kv_start + kv_len], vc[kv_start:kv_start + kv_len], scale=1.0)
    assert_close(got, want[0], "gemma4 sliding decode")
    nq1, hd1, n = 32, 128, 333
    q1 = (seeded_bf16(nq1, hd1, seed=184).float() * 0.3).bfloat16()
    k1, v1 = (seeded_bf16(n, 1, hd1, seed=185).float() * 0.3).bfloat16(), seeded_bf16(n, 1, hd1, seed=186)
    got1 = ops.gemma4_full_decode_attention(q1.cuda(), k1.cuda(), v1.cuda(), n, nq1, hd1)
    want1, _ = oracle.sdpa_f32(q1[None], k1, v1, scale=1.0)
    assert_close(got1, want1[0], "gemma4 full-attention decode, one KV head")


@pytest.mark.parametrize("window", [523, 540, 600])
def test_few_keys_in_the_first_block_repeat_bit_for_bit(ops, window):
    """A window that leaves most rows a few keys of their first key block: the next block raises their maximum by far
    more than 2^8, so the accumulator is rescaled while earlier P V products may still run.  One tile in two chains."""
    seq, kv_len, nq, nkv, hd = 400, 1466, 16, 8, 128
    q, k, v = seeded_bf16(1, seq, nq, hd, seed=61), seeded_bf16(1, kv_len, nkv, hd, seed=62), seeded_bf16(1, kv_len, nkv, hd, seed=63)
    want = oracle.sdpa_f32(q[0], k[0], v[0], scale=hd ** -0.5, mask_type=3, window=window)[0]
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    run = lambda: ops.sdpa_prefill(qd, kd, vd, scale=hd ** -0.5, mask_type=3, window=window, num_splits=1)  # noqa: E731
    first = run()
    assert_close(first[0], want, f"window {window}")
    for _ in range(40):
        assert torch.equal(first, run())


@pytest.mark.parametrize("nq,nkv,seq", [
    (8, 4, 1150), (6, 2, 1150),    # single tiles in two chains
    (24, 4, 2700), (28, 4, 2450),  # two tiles a CTA, 9 % and more faster by the rule: two heads of one tile, two tiles of one head
])
def test_vision_blocks_two_tiles_per_cta(ops, nq, nkv, seq):
    """Block ids looked up in the kernel against the additive buffer of the same rule: blocks of one token, across tiles, up
    to the last key; with a window that hides a block's first keys; the last tile ragged.  (That the two-tile kernel
    runs is certain where it is forced: test_prefill_pair_gpu.py.)"""
    kv, hd = seq + 100, 128
    ids = torch.full((kv,), -1, dtype=torch.int32)
    for i, (a, b) in enumerate([(30, 31), (31, 100), (140, 160), (227, 260), (300, 711), (840, 1096), (kv - 50, kv)]):
        ids[a:b] = i
    q, k, v = (seeded_bf16(n, h, hd, seed=50 + h).cuda() for n, h in ((seq, nq), (kv, nkv), (kv, nkv)))
    for window in (oracle.INT_MAX, 200):
        mask = ops.fill_causal_mask_with_block_ids(ids.cuda(), seq, kv, kv - seq, window)
        want, want_lse = ops.sdpa_prefill(q, k, v, scale=0.09, mask_type=ops.MASK_EXPLICIT, mask=mask, return_lse=True, num_splits=1)
        before = ops.launch_count()
        got, lse = ops.sdpa_prefill(q, k, v, scale=0.09, mask_type=ops.MASK_CAUSAL, window=window, block_ids=ids.cuda(), return_lse=True, num_splits=1)
        assert ops.launch_count() - before == 1
        # the same visible keys; blocks may be skipped in one form and fully masked in the other
        assert_close(got, want.float(), f"window {window}", rel_tol=4e-3, abs_tol=1.6e-2)
        assert torch.allclose(lse, want_lse, atol=2e-3)


def test_vision_blocks_need_no_workspace(ops):
    """The kernels look the ends of vision blocks up themselves: an unsplit call of head dim 128 brings no workspace."""
    from arcaine_b200 import _lib
    seq, nq, nkv, hd = 200, 4, 2, 128
    q, k, v = (seeded_bf16(seq, h, hd, seed=90 + i).cuda() for i, h in enumerate((nq, nkv, nkv)))
    ids = torch.full((seq,), -1, dtype=torch.int32, device="cuda")
    ids[30:170] = 3
    want = ops.sdpa_prefill(q, k, v, scale=0.09, mask_type=ops.MASK_CAUSAL, window=100, block_ids=ids, num_splits=1)
    out = torch.empty_like(q)
    p = _lib.PrefillParams()
    p.q, p.k, p.v, p.out, p.block_ids = q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), ids.data_ptr()
    p.batch, p.seq, p.kv_len, p.nq, p.nkv, p.hd = 1, seq, seq, nq, nkv, hd
    for f, heads in (("q", nq), ("k", nkv), ("v", nkv), ("o", nq)):
        setattr(p, f + "_stride_t", heads * hd)
        setattr(p, f + "_stride_b", seq * heads * hd)
    p.scale, p.mask_type, p.window, p.num_splits = 0.09, 3, 100, 1
    L = _lib.load()
    assert L.arc_sdpa_prefill_workspace_bytes(C.byref(p)) == 0
    torch.cuda.synchronize()
    assert L.arc_sdpa_prefill(C.byref(p), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert torch.equal(out, want)


@pytest.mark.parametrize("q_len,kv_len", [(4100, 1030), (4097, 1000), (2049, 2050)])  # from 4097 blocks of a row on, a block writes four
@pytest.mark.parametrize("window", [300, oracle.INT_MAX])
def test_mask_fill_of_many_rows(ops, q_len, kv_len, window):
    past = max(0, kv_len - q_len)
    got = ops.fill_causal_mask(q_len, kv_len, past, window).cpu().numpy()
    assert (got == oracle.fill_causal_mask(q_len, kv_len, past, window)).all()
