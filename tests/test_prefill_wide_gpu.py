"""Head dim 256 on pairs of CTAs (prefill_wide_sm100.cuh): the shapes where its splits, orders and hand-overs can go
wrong, against the oracle."""
import pytest
import torch

from helpers import assert_close, seeded_bf16
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,seq,kv,nq,nkv,mask,window,gate", [
    (1, 129, 129, 2, 2, 0, 0, False),     # odd group: 256 tokens of one head a pair, the second tile one row
    (1, 100, 300, 3, 3, 3, 0, True),      # the second CTA's tile has no row at all
    (2, 385, 385, 6, 2, 3, 200, True),    # odd group of three, two sequences, window edges inside blocks
    (1, 257, 130, 4, 2, 3, 0, False),     # fewer keys than queries: whole tiles see nothing
    (1, 300, 300, 4, 1, 3, 1, True),      # a window of one key
    (4, 200, 200, 48, 2, 3, 150, False),  # 192 one-block units of 128 tokens and more: several waves
    (4, 200, 200, 48, 2, 3, 0, True),     # the same without a window: longest units first
    (1, 700, 1900, 16, 2, 3, 0, False),   # two waves of unequal units, a ragged past
])
def test_against_oracle(batch, seq, kv, nq, nkv, mask, window, gate):
    from arcaine_b200 import ops
    ops.clear_device_status()
    hd, win = 256, window or oracle.INT_MAX
    q, k, v = seeded_bf16(batch, seq, nq, hd, seed=1), seeded_bf16(batch, kv, nkv, hd, seed=2), seeded_bf16(batch, kv, nkv, hd, seed=3)
    g = seeded_bf16(batch, seq, nq, hd, seed=4) if gate else None
    qd, kd, vd, gd = q.cuda(), k.cuda(), v.cuda(), g.cuda() if gate else None
    run = lambda: ops.sdpa_prefill(qd, kd, vd, scale=hd ** -0.5, mask_type=mask, window=win, gate=gd, num_splits=1,  # noqa: E731
                                   return_lse=True)
    out, lse = run()
    for _ in range(5):  # the order of hand-overs between the warps differs from run to run, the result must not
        again, lse2 = run()
    assert ops.device_status() == (0, 0)
    assert torch.equal(out, again) and torch.equal(lse, lse2)
    for b in range(batch):
        rows = sorted({r for t in (0, 1, 127, 128, seq // 2, seq - 2, seq - 1) if 0 <= t < seq for r in range(t * nq, t * nq + nq)})
        want = oracle.sdpa_f32(q[b], k[b], v[b], scale=hd ** -0.5, mask_type=mask, window=win, rows=rows,
                               gate=g[b] if gate else None)
        assert_close(out[b].reshape(-1, hd)[rows], want[1].float() if gate else want[0], f"sequence {b}")


def test_consecutive_one_block_units_keep_the_epilogue_in_step():
    """Units of one key block each, many per pair: the softmax may run two units ahead of a busy epilogue."""
    from arcaine_b200 import ops
    ops.clear_device_status()
    q, k, v = (seeded_bf16(2, 37 * 128, h, 256, seed=7 + i).cuda() for i, h in enumerate((16, 2, 2)))
    out = ops.sdpa_prefill(q, k, v, scale=0.0625, mask_type=ops.MASK_CAUSAL, window=100, num_splits=1)
    for _ in range(10):
        again = ops.sdpa_prefill(q, k, v, scale=0.0625, mask_type=ops.MASK_CAUSAL, window=100, num_splits=1)
    assert ops.device_status() == (0, 0) and torch.equal(out, again)
    solo = ops.sdpa_prefill(q[1:, :128], k[1:, :128], v[1:, :128], scale=0.0625, mask_type=ops.MASK_CAUSAL, window=100, num_splits=1)
    assert torch.equal(out[1:, :128], solo)


@pytest.mark.parametrize("seq,kv,nq,nkv,kind", [
    (200, 333, 8, 4, "window"),   # rows of the buffer not 16-byte aligned
    (129, 900, 6, 2, "random"),   # odd group; keys hidden at random
    (300, 1300, 4, 2, "blocks"),  # whole key blocks nobody sees, at either end and inside; a row without any key
    (150, 260, 4, 2, "values"),   # finite values, a bias per key, and -inf
    (1, 1, 2, 1, "window"),
])
def test_additive_mask(seq, kv, nq, nkv, kind):
    from arcaine_b200 import _lib, ops
    import ctypes as C
    ops.clear_device_status()
    hd, inf = 256, float("inf")
    g = torch.Generator().manual_seed(3)
    mask = torch.zeros(seq, kv)
    if kind == "window":
        mask = torch.from_numpy(oracle.fill_causal_mask(seq, kv, kv - seq, 100))
        assert torch.equal(ops.fill_causal_mask(seq, kv, kv - seq, 100).cpu(), mask)
    elif kind == "random":
        mask[torch.rand(seq, kv, generator=g) < 0.5] = -inf
    elif kind == "blocks":
        mask[:, :140], mask[:, 400:700], mask[:, 1200:] = -inf, -inf, -inf
        mask[7] = -inf
    else:
        mask = torch.randn(seq, kv, generator=g) * 2
        mask[:, 130:] = 0.0
        mask[torch.rand(seq, kv, generator=g) < 0.2] = -inf
    q, k, v = seeded_bf16(seq, nq, hd, seed=1), seeded_bf16(kv, nkv, hd, seed=2), seeded_bf16(kv, nkv, hd, seed=3)
    gate = seeded_bf16(seq, nq, hd, seed=4)
    dev = [t.cuda() for t in (q, k, v, gate, mask.float().contiguous())]
    out, lse = ops.sdpa_prefill(dev[0], dev[1], dev[2], scale=0.0625, mask_type=ops.MASK_EXPLICIT, mask=dev[4], return_lse=True)
    gated = ops.sdpa_prefill(dev[0], dev[1], dev[2], scale=0.0625, mask_type=ops.MASK_EXPLICIT, mask=dev[4], gate=dev[3])
    want = oracle.sdpa_f32(q, k, v, scale=0.0625, mask_type=1, mask=mask.numpy(), want_lse=True)
    assert_close(out, want[0], kind)
    fin = torch.isfinite(want[2])
    assert torch.equal(torch.isfinite(lse.cpu()), fin) and torch.allclose(lse.cpu()[fin], want[2][fin], atol=2e-3)
    assert_close(gated, oracle.sdpa_f32(q, k, v, scale=0.0625, mask_type=1, mask=mask.numpy(), gate=gate)[1].float(), kind + " gated")
    # without a workspace the call still works (the mask is then read by the attention kernel itself)
    p = _lib.PrefillParams()
    o2 = torch.empty_like(out)
    p.q, p.k, p.v, p.out, p.mask = (t.data_ptr() for t in (dev[0], dev[1], dev[2], o2, dev[4]))
    p.batch, p.seq, p.kv_len, p.nq, p.nkv, p.hd = 1, seq, kv, nq, nkv, hd
    p.q_stride_t = p.o_stride_t = nq * hd
    p.k_stride_t = p.v_stride_t = nkv * hd
    p.q_stride_b, p.o_stride_b, p.k_stride_b, p.v_stride_b = seq * nq * hd, seq * nq * hd, kv * nkv * hd, kv * nkv * hd
    p.scale, p.mask_type, p.window, p.num_splits = 0.0625, ops.MASK_EXPLICIT, ops.NO_WINDOW, 1
    assert _lib.load().arc_sdpa_prefill(C.byref(p), torch.cuda.current_stream().cuda_stream) == _lib.ARC_OK
    assert_close(o2, want[0], kind + " without a workspace")
    assert ops.device_status() == (0, 0)


@pytest.mark.parametrize("seq,kv,nq,nkv,kind,launches", [
    (16, 5000, 8, 4, "causal", 3),     # eight parts, one ragged tile: scan, attention, merge
    (180, 4200, 24, 4, "random", 3),   # 24 units in three parts
    (200, 4300, 32, 4, "blocks", 2),   # 32 units in two parts, a cluster each; a row without any key, unseen blocks at a part's ends
    (64, 4096, 6, 2, "values", 3),     # odd group, finite values
    (130, 1200, 3, 3, "window", 3),    # odd group, the second tile two rows; parts that see nothing
    (256, 2304, 8, 4, "causal", 2),    # too many rows for so few blocks: whole units
])
def test_additive_mask_over_parts_of_the_key_range(seq, kv, nq, nkv, kind, launches):
    """Few queries over a long cache: the library splits a masked call as it does others.  Gated, and with log-sum-exp and
    a copy of the output, as the whole range gives them."""
    from arcaine_b200 import ops
    ops.clear_device_status()
    hd, inf = 256, float("inf")
    g = torch.Generator().manual_seed(9)
    mask = torch.from_numpy(oracle.fill_causal_mask(seq, kv, kv - seq, 200 if kind == "window" else oracle.INT_MAX)).clone()
    if kind == "random":
        mask[torch.rand(seq, kv, generator=g) < 0.5] = -inf
    elif kind == "blocks":
        mask[:, :700], mask[:, 1900:2700], mask[7] = -inf, -inf, -inf
    elif kind == "values":
        mask += torch.randn(seq, kv, generator=g) * 2
    mask = mask.cuda()
    q, k, v, gate = (seeded_bf16(n, h, hd, seed=90 + i).cuda() for i, (n, h) in enumerate([(seq, nq), (kv, nkv), (kv, nkv), (seq, nq)]))
    run = lambda n, **kw: ops.sdpa_prefill(q, k, v, scale=0.0625, mask_type=ops.MASK_EXPLICIT, mask=mask, num_splits=n, **kw)  # noqa: E731
    copy = torch.empty_like(q)
    before = ops.launch_count()
    out, lse = run(0, return_lse=True, out_copies=torch.tensor([copy.data_ptr()], device="cuda"))
    assert ops.launch_count() - before == launches
    want, want_lse = run(1, return_lse=True)
    assert_close(out, want.float().cpu(), kind, rel_tol=4e-3, abs_tol=1.6e-2)  # (as in test_parts_of_the_key_range)
    assert torch.equal(copy, out)
    fin = torch.isfinite(want_lse)
    assert torch.equal(torch.isfinite(lse), fin) and torch.allclose(lse[fin], want_lse[fin], atol=2e-3)
    assert_close(run(0, gate=gate), run(1, gate=gate).float().cpu(), kind + " gated", rel_tol=4e-3, abs_tol=1.6e-2)
    for _ in range(5):
        assert torch.equal(run(0), out)
    assert ops.device_status() == (0, 0)


@pytest.mark.parametrize("hd", [128, 256])
@pytest.mark.parametrize("kv", [260, 333])  # rows of whole groups of four values, and not
def test_additive_mask_at_any_alignment(hd, kv):
    """A mask whose buffer, or whose rows, do not start at multiples of 16 bytes gives the same bits."""
    from arcaine_b200 import ops
    ops.clear_device_status()
    seq, nq, nkv = 150, 4, 2
    q, k, v = seeded_bf16(seq, nq, hd, seed=1).cuda(), seeded_bf16(kv, nkv, hd, seed=2).cuda(), seeded_bf16(kv, nkv, hd, seed=3).cuda()
    g = torch.Generator().manual_seed(5)
    mask = torch.randn(seq, kv, generator=g)
    mask[torch.rand(seq, kv, generator=g) < 0.2] = -float("inf")
    got = []
    for shift in range(4):
        buf = torch.empty(seq * kv + 4, device="cuda")[shift:shift + seq * kv].view(seq, kv)
        buf.copy_(mask)
        got.append(ops.sdpa_prefill(q, k, v, scale=0.0625, mask_type=ops.MASK_EXPLICIT, mask=buf))
    assert_close(got[0], oracle.sdpa_f32(q.cpu(), k.cpu(), v.cpu(), scale=0.0625, mask_type=1, mask=mask.numpy())[0], f"kv {kv}")
    assert all(torch.equal(o, got[0]) for o in got) and ops.device_status() == (0, 0)


@pytest.mark.parametrize("scale", [0.0625, 1.0, 1.5])
def test_additive_mask_of_the_lowest_value_infinity_and_nan(scale):
    """Scanned or read by the attention kernel itself (no workspace), a mask means the same: the type's lowest value hides
    a key as -inf does, NaN and +inf go on to their row only."""
    from arcaine_b200 import _lib, ops
    import ctypes as C
    ops.clear_device_status()
    seq, kv, nq, nkv, hd, inf, lowest = 40, 300, 4, 2, 256, float("inf"), torch.finfo(torch.float32).min
    q = (seeded_bf16(seq, nq, hd, seed=1).float() * hd ** -0.5).bfloat16().cuda()
    k, v = seeded_bf16(kv, nkv, hd, seed=2).cuda(), seeded_bf16(kv, nkv, hd, seed=3).cuda()
    mask = torch.zeros(seq, kv, device="cuda")
    mask[0] = lowest
    mask[1, 20:] = lowest
    mask[2, 7], mask[3, 8] = float("nan"), inf
    mask[4] = -2.0e38  # finite, large: the same for every key, so that it changes nothing
    mask[5], mask[5, 250:] = lowest, 1.0
    run = lambda m: ops.sdpa_prefill(q, k, v, scale=scale, mask_type=ops.MASK_EXPLICIT, mask=m, num_splits=1, return_lse=True)  # noqa: E731
    out, lse = run(mask)
    own, own_lse = torch.empty_like(out), torch.empty_like(lse)
    p = _lib.PrefillParams()
    p.q, p.k, p.v, p.out, p.mask, p.out_lse = (t.data_ptr() for t in (q, k, v, own, mask, own_lse))
    p.batch, p.seq, p.kv_len, p.nq, p.nkv, p.hd = 1, seq, kv, nq, nkv, hd
    p.q_stride_t = p.o_stride_t = nq * hd
    p.k_stride_t = p.v_stride_t = nkv * hd
    p.scale, p.mask_type, p.window, p.num_splits = scale, ops.MASK_EXPLICIT, ops.NO_WINDOW, 1
    assert _lib.load().arc_sdpa_prefill(C.byref(p), torch.cuda.current_stream().cuda_stream) == _lib.ARC_OK
    for o, l in ((out, lse), (own, own_lse)):
        assert torch.count_nonzero(o[0].float()) == 0 and (l[0] == -inf).all()
        assert torch.isnan(o[2].float()).all() and torch.isnan(o[3].float()).all()
    hidden = mask.clone()
    hidden[hidden == lowest] = -inf
    hidden[2:5] = 0.0
    want, _ = run(hidden)
    rows = [1, 4] + list(range(5, seq))
    # (-2e38 and a score are -2e38 in fp32: row 4 sees all keys alike)
    want[4] = v.float().mean(0).repeat_interleave(nq // nkv, 0).bfloat16()
    assert_close(out[rows], want[rows].float(), "scanned", rel_tol=4e-3, abs_tol=1.6e-2)
    assert_close(own[rows], want[rows].float(), "read by the kernel", rel_tol=4e-3, abs_tol=1.6e-2)
    assert ops.device_status() == (0, 0)


@pytest.mark.parametrize("room,shift", [(0, 0), (4096, 0), (1 << 26, 4)])  # none, too little, not 16-byte aligned
def test_a_workspace_that_cannot_be_used_costs_time_only(room, shift):
    """A canvas step whose parts have no place for their records runs over the whole key range."""
    from arcaine_b200 import _lib, ops
    import ctypes as C
    ops.clear_device_status()
    seq, kv, nq, nkv, hd = 256, 1400, 8, 4, 256
    q, k, v = (seeded_bf16(n, h, hd, seed=80 + i).cuda() for i, (n, h) in enumerate([(seq, nq), (kv, nkv), (kv, nkv)]))
    out, ws = torch.empty_like(q), torch.zeros(room + 64, dtype=torch.uint8, device="cuda")
    p = _lib.PrefillParams()
    p.q, p.k, p.v, p.out = (t.data_ptr() for t in (q, k, v, out))
    p.batch, p.seq, p.kv_len, p.nq, p.nkv, p.hd = 1, seq, kv, nq, nkv, hd
    p.q_stride_t = p.o_stride_t = nq * hd
    p.k_stride_t = p.v_stride_t = nkv * hd
    p.scale, p.mask_type, p.window, p.num_splits = 0.0625, ops.MASK_NONE, ops.NO_WINDOW, 0
    L = _lib.load()
    assert 4096 < L.arc_sdpa_prefill_workspace_bytes(C.byref(p)) <= 1 << 26
    if room:
        p.workspace, p.workspace_bytes = ws.data_ptr() + shift, room
    assert L.arc_sdpa_prefill(C.byref(p), torch.cuda.current_stream().cuda_stream) == _lib.ARC_OK
    assert torch.equal(out, ops.sdpa_prefill(q, k, v, scale=0.0625, num_splits=1))
    assert ops.device_status() == (0, 0) and not ws.any()


@pytest.mark.parametrize("seq,kv", [(1, 1), (7, 3), (300, 64), (1000, 65), (513, 512), (65, 1025), (70000, 5), (40000, 513)])
def test_mask_buffers_of_any_shape(seq, kv):
    """Rows that share a block, rows of several blocks, more rows than a grid has blocks; nothing beside the buffer."""
    from arcaine_b200 import ops
    past = max(0, kv - seq)
    buf = torch.full((seq * kv + 64,), 7.0, device="cuda")
    ops.fill_causal_mask(seq, kv, past, 50, out=buf[:seq * kv].view(seq, kv))
    i = torch.arange(seq, device="cuda")[:, None] + past
    j = torch.arange(kv, device="cuda")[None] + past - (kv - seq)
    want = torch.zeros(seq, kv, device="cuda").masked_fill_((j > i) | (j < i - 49), -float("inf"))
    assert torch.equal(buf[:seq * kv].view(seq, kv), want) and (buf[seq * kv:] == 7.0).all()


def test_vision_blocks_longer_than_a_search_step():
    """Block ids looked up in the kernel (128 keys a step, 32 rows a warp) against the additive buffer of the same rule:
    blocks of one token, next to each other, across warps and tiles, longer than a step, and up to the last key."""
    from arcaine_b200 import ops
    ops.clear_device_status()
    seq, kv, nq, nkv, hd = 900, 1000, 12, 4, 256
    ids = torch.full((kv,), -1, dtype=torch.int32)
    for i, (a, b) in enumerate([(30, 31), (31, 100), (140, 160), (227, 260), (260, 261), (300, 711), (840, 1000)]):
        ids[a:b] = i
    q, k, v = (seeded_bf16(n, h, hd, seed=40 + h).cuda() for n, h in ((seq, nq), (kv, nkv), (kv, nkv)))
    for window in (oracle.INT_MAX, 200):
        mask = ops.fill_causal_mask_with_block_ids(ids.cuda(), seq, kv, kv - seq, window)
        want = ops.sdpa_prefill(q, k, v, scale=0.0625, mask_type=ops.MASK_EXPLICIT, mask=mask)
        got = ops.sdpa_prefill(q, k, v, scale=0.0625, mask_type=ops.MASK_CAUSAL, window=window, block_ids=ids.cuda())
        # the same visible keys; blocks may be skipped in one form and fully masked in the other
        assert_close(got, want.float(), f"window {window}", rel_tol=2e-3, abs_tol=8e-3)
    assert ops.device_status() == (0, 0)


@pytest.mark.parametrize("batch,seq,kv,nq,nkv,window,gate,vision", [
    (1, 1664, 1664, 24, 4, 0, False, False),  # 156 units on 74 pairs: two or three each, the longest to those with two
    (1, 1024, 2400, 24, 4, 0, True, False),   # 96: one or two, gated
    (3, 300, 2000, 27, 9, 0, False, False),   # odd groups of 256 tokens, 162
    (1, 3000, 3000, 48, 8, 150, False, False),  # a window, 576, as long as each other but for the first
    (1, 1500, 1500, 24, 4, 400, False, True),   # vision blocks, looked up a unit ahead
    (1, 900, 500, 48, 8, 0, False, True),       # and tiles that see nothing between others
    (1, 900, 500, 48, 8, 0, True, True),        # gated
    (20, 130, 128, 8, 4, 0, True, False),       # gated units of one key block, whose scores run ahead of the unit before
])
def test_several_units_a_pair(batch, seq, kv, nq, nkv, window, gate, vision):
    """More units than pairs: the accumulator freed ahead of the output, the two kinds of pairs, the look-up of the next unit."""
    from arcaine_b200 import ops
    ops.clear_device_status()
    hd, win = 256, window or oracle.INT_MAX
    q, k, v, g = (seeded_bf16(batch, n, h, hd, seed=110 + i) for i, (n, h) in enumerate([(seq, nq), (kv, nkv), (kv, nkv), (seq, nq)]))
    qd, kd, vd, copy = q.cuda(), k.cuda(), v.cuda(), torch.empty(batch, seq, nq, hd, dtype=torch.bfloat16, device="cuda")
    ids = torch.full((seq,), -1, dtype=torch.int32)  # (by position of the query; key j is position j + seq - kv)
    base = max(0, seq - kv)
    for i, (a, b) in enumerate([(10, 90), (127, 129), (200, 360), (400, 499)]):
        ids[base + a:base + b] = i
    run = lambda: ops.sdpa_prefill(qd, kd, vd, scale=hd ** -0.5, mask_type=3, window=win, gate=g.cuda() if gate else None, num_splits=1,  # noqa: E731
                                   out_copies=torch.tensor([copy.data_ptr()], device="cuda"), block_ids=ids.cuda() if vision else None,
                                   block_ids_offset=seq - kv if vision else 0)
    out = run()
    assert torch.equal(copy, out)
    for _ in range(5):
        assert torch.equal(run(), out)
    assert ops.device_status() == (0, 0)
    mask = oracle.fill_causal_mask_with_block_ids(ids.numpy(), seq, kv, 0, win) if vision else None
    for b in range(batch):
        rows = sorted({t * nq + h for t in (0, 127, 128, 300, 459, seq // 2, seq - 129, seq - 1) if t < seq for h in (0, 1, nq // 2, nq - 1)})
        want = oracle.sdpa_f32(q[b], k[b], v[b], scale=hd ** -0.5, mask_type=1 if vision else 3, window=win, mask=mask, rows=rows,
                               gate=g[b] if gate else None)
        assert_close(out[b].reshape(-1, hd)[rows], want[1].float() if gate else want[0], f"sequence {b}")


@pytest.mark.parametrize("seq,kv,nq,nkv,gate,parts", [
    (1664, 1664, 24, 4, False, 1), (1664, 1664, 24, 4, True, 1),  # several units a pair
    (161, 202, 24, 4, False, 1), (256, 1100, 8, 4, False, 3), (256, 1100, 8, 4, False, 8),  # one; parts in both forms
])
def test_results_below_the_smallest_normal_number(seq, kv, nq, nkv, gate, parts):
    """V times a power of two: the results times the same, but for the rounding of bf16 down there (half of 2^-133) and of the
    results it is compared with (2^-9 of 2^-126 at most)."""
    from arcaine_b200 import ops
    q, k, v, g = (seeded_bf16(n, h, 256, seed=140 + i).cuda() for i, (n, h) in enumerate([(seq, nq), (kv, nkv), (kv, nkv), (seq, nq)]))
    v = (v * 2.0 ** -124).bfloat16()
    run = lambda v: ops.sdpa_prefill(q, k, v, scale=0.0625, mask_type=3 if seq > 256 else 0, num_splits=parts, gate=g if gate else None).double()  # noqa: E731
    got, want = run(v), run((v.float() * 2.0 ** 124).bfloat16()) * 2.0 ** -124
    small = want.abs() < 2.0 ** -126
    assert small.float().mean() > 0.3 and (got - want)[small].abs().max() <= 2.0 ** -133 * (2 if gate else 1)  # (gated: rounded twice)


def chosen_parts(batch, seq, kv, nq, nkv, window=oracle.INT_MAX, gate=False):
    """Parts of the key range that the library chooses, told by the workspace that it asks for."""
    from arcaine_b200 import _lib
    import ctypes as C
    room = torch.zeros(4, dtype=torch.uint8, device="cuda")
    p = _lib.PrefillParams()
    p.q = p.k = p.v = p.out = room.data_ptr()
    p.gate = room.data_ptr() if gate else None
    p.batch, p.seq, p.kv_len, p.nq, p.nkv, p.hd = batch, seq, kv, nq, nkv, 256
    p.q_stride_t = p.o_stride_t = nq * 256
    p.k_stride_t = p.v_stride_t = nkv * 256
    p.q_stride_b = p.o_stride_b = seq * nq * 256
    p.k_stride_b = p.v_stride_b = kv * nkv * 256
    p.scale, p.mask_type, p.window = 0.0625, 3 if window != oracle.INT_MAX else 0, window
    need = []
    for n in range(9):
        p.num_splits = n
        need.append(_lib.load().arc_sdpa_prefill_workspace_bytes(C.byref(p)))
    return need.index(need[0], 1)


@pytest.mark.parametrize("batch,seq,kv,nq,nkv,window,gate,parts", [
    (1, 45, 663, 8, 4, 533, False, 4),  # behind a window (us): four parts 9.0, six 9.1, three of two masked blocks 9.8
    (1, 63, 663, 4, 2, 533, False, 4),  # 9.3, three 10.0
    (3, 45, 1000, 4, 2, oracle.INT_MAX, True, 4),  # gated: four 10.0, eight 10.6
    (3, 45, 663, 4, 2, 533, True, 6),   # 9.5, three 10.55
    (1, 256, 2304, 16, 8, oracle.INT_MAX, False, 3),  # 15.6, two 17.1
])
def test_parts_that_the_library_chooses(batch, seq, kv, nq, nkv, window, gate, parts):
    assert chosen_parts(batch, seq, kv, nq, nkv, window, gate) == parts


@pytest.mark.parametrize("parts", [2, 3, 4, 8])
@pytest.mark.parametrize("batch,seq,kv,nq,nkv,window", [
    (1, 256, 1100, 8, 4, oracle.INT_MAX),  # two row tiles of pairs of heads, the last key block ragged
    (1, 77, 1030, 4, 2, oracle.INT_MAX),   # one ragged tile: shares of the fold without rows
    (2, 130, 700, 3, 3, oracle.INT_MAX),   # odd group: 256 tokens of one head, the second tile two rows
    (1, 300, 900, 4, 2, 60),               # a window: parts without key blocks, rows that see none of a part's keys
    (3, 200, 600, 24, 4, oracle.INT_MAX),  # more units than clusters or pairs: always a merge launch, several waves
])
def test_parts_of_the_key_range(parts, batch, seq, kv, nq, nkv, window):
    """Two and three parts fold as one cluster where every cluster fits at once, the rest in a launch of their own: the
    gated output, the plain one with its log-sum-exp and its copy, as the whole range gives them."""
    from arcaine_b200 import ops
    ops.clear_device_status()
    hd, mask = 256, 3 if window != oracle.INT_MAX else 0
    q, k, v, gate = (seeded_bf16(batch, n, h, hd, seed=70 + i).cuda() for i, (n, h) in enumerate([(seq, nq), (kv, nkv), (kv, nkv), (seq, nq)]))
    run = lambda n, **kw: ops.sdpa_prefill(q, k, v, scale=0.0625, mask_type=mask, window=window, num_splits=n, **kw)  # noqa: E731
    copy = torch.empty_like(q)
    before = ops.launch_count()
    out, lse = run(parts, return_lse=True, out_copies=torch.tensor([copy.data_ptr()], device="cuda"))
    units = batch * ((seq + 127) // 128 * nq // 2 if nq // nkv % 2 == 0 else (seq + 255) // 256 * nq)
    assert ops.launch_count() - before == (1 if parts <= 3 and units <= 20 else 2)
    want, want_lse = run(1, return_lse=True)
    # the same values but for the bf16 rounding of the probabilities, whose reference a part chooses for itself
    assert_close(out, want.float().cpu(), "out", rel_tol=4e-3, abs_tol=1.6e-2)
    assert torch.equal(copy, out)
    fin = torch.isfinite(want_lse)
    assert torch.equal(torch.isfinite(lse), fin) and torch.allclose(lse[fin], want_lse[fin], atol=2e-3)
    assert_close(run(parts, gate=gate), run(1, gate=gate).float().cpu(), "gated", rel_tol=4e-3, abs_tol=1.6e-2)
    for _ in range(10):
        assert torch.equal(run(parts), out)
    assert ops.device_status() == (0, 0)


@pytest.mark.parametrize("parts", [2, 3, 4, 8])
@pytest.mark.parametrize("batch,seq,kv,nq,nkv,window", [
    (1, 300, 900, 8, 4, oracle.INT_MAX),  # three row tiles of pairs of heads
    (1, 256, 700, 3, 3, 200),             # odd group, a window: parts whose keys some rows do not see
])
def test_vision_blocks_in_parts(parts, batch, seq, kv, nq, nkv, window):
    """Two and three parts in a cluster, four and eight with a merge launch, gated and not, as the whole range gives them; the whole
    range against the oracle."""
    from arcaine_b200 import ops
    ops.clear_device_status()
    q, k, v, g = (seeded_bf16(batch, n, h, 256, seed=150 + i) for i, (n, h) in enumerate([(seq, nq), (kv, nkv), (kv, nkv), (seq, nq)]))
    ids = torch.full((kv,), -1, dtype=torch.int32)
    for i, (a, b) in enumerate([(kv - seq + 10, kv - seq + 90), (kv - seq + 127, kv - seq + 129), (kv - seq + 130, kv - 20)]):
        ids[a:b] = i
    run = lambda n, gate: ops.sdpa_prefill(q.cuda(), k.cuda(), v.cuda(), scale=0.0625, mask_type=3, window=window, num_splits=n,  # noqa: E731
                                           gate=g.cuda() if gate else None, block_ids=ids.cuda())
    mask = oracle.fill_causal_mask_with_block_ids(ids.numpy(), seq, kv, kv - seq, window)
    rows = sorted({t * nq + h for t in (0, 9, 10, 89, 127, 128, 129, 200, seq - 1) for h in (0, nq - 1)})
    for gate in (False, True):
        whole = run(1, gate)
        want = oracle.sdpa_f32(q[0], k[0], v[0], scale=0.0625, mask_type=1, mask=mask, rows=rows, gate=g[0] if gate else None)
        assert_close(whole[0].reshape(-1, 256)[rows], want[1].float() if gate else want[0], "whole")
        before = ops.launch_count()
        got = run(parts, gate)
        assert ops.launch_count() - before == (1 if parts <= 3 else 2)
        assert_close(got, whole.float().cpu(), f"gate {gate}", rel_tol=4e-3, abs_tol=1.6e-2)
        assert torch.equal(run(parts, gate), got)
    assert ops.device_status() == (0, 0)


@pytest.mark.parametrize("batch,seq,kv,nq,nkv,window", [
    (1, 128, 1000, 16, 8, oracle.INT_MAX),  # every row of both tiles, the last key block ragged
    (1, 200, 1500, 3, 3, oracle.INT_MAX),   # odd group, 256 tokens a unit: the second tile ragged
    (1, 1, 512, 8, 2, oracle.INT_MAX),      # one row in each tile, one key block a part
    (3, 100, 900, 4, 2, oracle.INT_MAX),    # three sequences
    (1, 130, 2000, 3, 3, 700),              # a window: rows that see nothing of a part; odd group
])
def test_four_parts_fold_themselves(batch, seq, kv, nq, nkv, window):
    """Where the library chooses four parts, not gated, their cluster folds them: one launch, as the whole range gives it."""
    from arcaine_b200 import ops
    ops.clear_device_status()
    assert chosen_parts(batch, seq, kv, nq, nkv, window) == 4
    mask = 3 if window != oracle.INT_MAX else 0
    q, k, v = (seeded_bf16(batch, n, h, 256, seed=130 + i).cuda() for i, (n, h) in enumerate([(seq, nq), (kv, nkv), (kv, nkv)]))
    copy = torch.empty_like(q)
    run = lambda n: ops.sdpa_prefill(q, k, v, scale=0.0625, mask_type=mask, window=window, num_splits=n, return_lse=True,  # noqa: E731
                                     out_copies=torch.tensor([copy.data_ptr()], device="cuda"))
    want, want_lse = run(1)
    before = ops.launch_count()
    out, lse = run(0)
    assert ops.launch_count() - before == 1 and not torch.equal(lse, want_lse)  # in parts, without a merge launch
    # the same values but for the bf16 rounding of the probabilities, whose reference a part chooses for itself
    assert_close(out, want.float().cpu(), "out", rel_tol=4e-3, abs_tol=1.6e-2)
    assert torch.equal(copy, out)
    fin = torch.isfinite(want_lse)
    assert torch.equal(torch.isfinite(lse), fin) and torch.allclose(lse[fin], want_lse[fin], atol=2e-3)
    for _ in range(10):
        assert torch.equal(run(0)[0], out)
    assert ops.device_status() == (0, 0)
