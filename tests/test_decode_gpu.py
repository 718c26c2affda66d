"""Parity of the split-KV decode kernel and the LSE merge with the CPU oracle, through the C ABI."""
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
    assert o.device_status() == (0, 0), "a bounded device-side wait gave up during the decode tests"


def oracle_decode(q, k_rows, v_rows, scale, gate=None):
    """q (nq, hd), k/v (len, nkv, hd) -> (f32 out, bf16 out, lse)."""
    return oracle.sdpa_f32(q[None], k_rows, v_rows, scale=scale, gate=gate[None] if gate is not None else None,
                           want_lse=True)


@pytest.mark.parametrize("B,nq,nkv,hd,lens", [
    (1, 8, 2, 128, [37]),
    (2, 8, 2, 128, [100, 300]),
    (3, 24, 4, 256, [17, 1000, 257]),
    (2, 16, 2, 128, [5000, 1]),
    (4, 6, 1, 256, [64, 65, 63, 1024]),
    (2, 32, 2, 128, [333, 77]),       # 16 query heads per KV head: two n-tiles
    (2, 32, 16, 128, [200, 31]),      # 16 KV heads: two head groups per key share
    (3, 4, 4, 256, [0, 50, 0]),       # empty sequences give zeros
])
def test_variable_lengths_block_cache(ops, B, nq, nkv, hd, lens):
    cap = max(max(lens), 1) + 5
    q = seeded_bf16(B, nq, hd, seed=1)
    k, v = seeded_bf16(B, cap, nkv, hd, seed=2), seeded_bf16(B, cap, nkv, hd, seed=3)
    g = seeded_bf16(B, nq, hd, seed=4)
    kd, vd = k.cuda(), v.cuda()
    # rows past each sequence's length are never-written cache: poison them
    for b, n in enumerate(lens):
        kd[b, n:] = float("nan")
        vd[b, n:] = float("nan")
    kl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    scale = hd ** -0.5
    out, o32, lse = ops.sdpa_decode(q.cuda(), kd, vd, scale=scale, kv_len=kl, return_partial=True)
    outg = ops.sdpa_decode(q.cuda(), kd, vd, scale=scale, kv_len=kl, gate=g.cuda())
    for b, n in enumerate(lens):
        if n == 0:
            assert torch.count_nonzero(out[b].float()) == 0 and torch.isinf(lse[b]).all()
            continue
        wf, wb, wl = oracle_decode(q[b], k[b, :n], v[b, :n], scale)
        assert_close(out[b], wf[0], f"seq {b} len {n}")
        assert_close(o32[b], wf[0], f"seq {b} f32", rel_tol=3e-3, abs_tol=5e-3)
        assert torch.allclose(lse[b].cpu(), wl[0], atol=2e-3)
        _, wgb, _ = oracle_decode(q[b], k[b, :n], v[b, :n], scale, gate=g[b])
        assert_close(outg[b], wgb[0].float(), f"seq {b} gated")


def test_packed_cache_with_row_offsets_and_cta_counts(ops):
    B, nq, nkv, hd = 5, 24, 4, 256
    lens = [700, 33, 1500, 1, 260]
    offs = [0]
    for n in lens[:-1]:
        offs.append(offs[-1] + n)
    total = sum(lens)
    q = seeded_bf16(B, nq, hd, seed=11)
    k, v = seeded_bf16(total, nkv, hd, seed=12), seeded_bf16(total, nkv, hd, seed=13)
    kl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    ko = torch.tensor(offs, dtype=torch.int64, device="cuda")
    want = [oracle_decode(q[b], k[offs[b]:offs[b] + lens[b]], v[offs[b]:offs[b] + lens[b]], 0.0625)[0][0] for b in range(B)]
    for nctas in (0, 1, 3, 148, 500):
        out = ops.sdpa_decode(q.cuda(), k.cuda(), v.cuda(), scale=0.0625, kv_len=kl, kv_row_offset=ko, num_ctas=nctas)
        for b in range(B):
            assert_close(out[b], want[b], f"num_ctas {nctas} seq {b}")


def test_qwen_single_token_entry_points(ops):
    """seq == 1 through the reference-named calls, bench-recipe inputs, against the restated scalar kernel."""
    nq, nkv, hd, depth = 24, 4, 256, 512
    state = 42
    qb, state = oracle.lcg_fill(nq * hd, state)
    kb, state = oracle.lcg_fill((depth + 1) * nkv * hd, state)
    vb, state = oracle.lcg_fill((depth + 1) * nkv * hd, state)
    gb, state = oracle.lcg_fill(nq * hd, state)
    q = oracle.bits_to_bf16(qb).reshape(1, nq, hd)
    k = oracle.bits_to_bf16(kb).reshape(depth + 1, nkv, hd)
    v = oracle.bits_to_bf16(vb).reshape(depth + 1, nkv, hd)
    g = oracle.bits_to_bf16(gb).reshape(1, nq, hd)
    want = oracle.qwen35_online_attention(q, k, v, seq=1, past=depth, scale=0.0625)
    buf = q.cuda().clone()
    ops.qwen35_xmx_attention(buf, k.cuda(), v.cuda(), buf, 1, depth, nq, nkv, hd, 0.0625)  # out aliases q
    assert_close(buf, want.float(), "qwen35_xmx_attention seq=1")
    out = torch.empty_like(buf)
    ops.qwen35_xmx_attention_decode_gqa(q.cuda(), k.cuda(), v.cuda(), out, depth, nq, nkv, hd, 0.0625, gate=g.cuda())
    assert_close(out, oracle.mul_sigmoid_inplace(want, g).float(), "decode_gqa + gate")
    # the unfused pair of launches gives the same thing
    ops.mul_sigmoid_inplace(buf, g.cuda())
    assert_close(buf, oracle.mul_sigmoid_inplace(want, g).float(), "attention then mul_sigmoid_inplace")


def test_qwen_single_token_over_a_block_of_one_sequence(ops):
    """key and value as (1, capacity, nkv, hd), past + 1 rows of them in use."""
    nq, nkv, hd, depth = 24, 4, 256, 300
    q, g = seeded_bf16(1, nq, hd, seed=1).cuda(), seeded_bf16(1, nq, hd, seed=2).cuda()
    k, v = seeded_bf16(1, depth + 9, nkv, hd, seed=3).cuda(), seeded_bf16(1, depth + 9, nkv, hd, seed=4).cuda()
    want, got = torch.empty_like(q), torch.empty_like(q)
    ops.qwen35_xmx_attention_decode_gqa(q, k[0], v[0], want, depth, nq, nkv, hd, 0.0625, gate=g)
    ops.qwen35_xmx_attention_decode_gqa(q, k, v, got, depth, nq, nkv, hd, 0.0625, gate=g)
    assert torch.equal(got, want)
    ops.qwen35_xmx_attention(q, k[0], v[0], want, 1, depth, nq, nkv, hd, 0.0625)
    ops.qwen35_xmx_attention(q, k, v, got, 1, depth, nq, nkv, hd, 0.0625)
    assert torch.equal(got, want)
    with pytest.raises(ValueError):
        ops.qwen35_xmx_attention(q.expand(2, -1, -1).contiguous(), k, v, torch.empty_like(q).expand(2, -1, -1).contiguous(), 2, depth, nq, nkv, hd, 0.0625)


def test_merge_kernel_against_oracle(ops):
    P, rows, hd = 5, 37, 128
    g = torch.Generator().manual_seed(5)
    po = torch.randn(P, rows, hd, generator=g)
    pl = torch.randn(P, rows, generator=g) * 3
    pl[2] = float("-inf")           # an empty part
    pl[:, 7] = float("-inf")        # a row nobody covers
    gate = seeded_bf16(rows, hd, seed=6)
    want, want_lse = oracle.merge_partials(po, pl)
    out, o32, lse = ops.sdpa_merge(po.cuda(), pl.cuda(), want_f32=True, want_lse=True)
    assert torch.allclose(o32.cpu(), want, atol=1e-5)
    fin = torch.isfinite(want_lse)
    assert torch.allclose(lse.cpu()[fin], want_lse[fin], atol=1e-5) and torch.isinf(lse.cpu()[~fin]).all()
    assert_close(out, want, "bf16 merge", rel_tol=4e-3, abs_tol=2e-2)
    gated = ops.sdpa_merge(po.cuda(), pl.cuda(), gate=gate.cuda())
    assert_close(gated, oracle.mul_sigmoid_inplace(want.bfloat16(), gate).float(), "gated merge", rel_tol=4e-3)
    # strided parts: one packed [out | lse] record per part, merged in place
    from arcaine_b200 import sharded
    n = sharded.record_numel(1, rows, hd)
    rec = torch.zeros(P, n, device="cuda")
    ro, rl = sharded.split_record(rec, 1, rows, hd)
    ro.copy_(po.cuda().view(P, 1, rows, hd))
    rl.copy_(pl.cuda().view(P, 1, rows))
    out2 = ops.sdpa_merge(ro, rl)
    assert torch.equal(out2.view(rows, hd), out)


def test_sequence_sharded_partials_merge_to_the_whole(ops):
    """What each GPU of a sequence-sharded decode computes, emulated on one device: partial
    (out, lse) per key slice, then the merge — must equal decode over the whole range."""
    from arcaine_b200 import sharded
    B, nq, nkv, hd, L, world = 2, 16, 2, 128, 3000, 4
    q = seeded_bf16(B, nq, hd, seed=21)
    k, v = seeded_bf16(B, L, nkv, hd, seed=22), seeded_bf16(B, L, nkv, hd, seed=23)
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    n = sharded.record_numel(B, nq, hd)
    gathered = torch.zeros(world, n, device="cuda")
    for r, (lo, hi) in enumerate(sharded.plan_seq_shards(L, world)):
        po, pl = sharded.split_record(gathered[r], B, nq, hd)
        ops.sdpa_decode(qd, kd[:, lo:hi], vd[:, lo:hi], scale=0.09, return_partial=True, want_out=False,
                        partial_out=po, partial_lse=pl)
    ao, al = sharded.split_record(gathered, B, nq, hd)
    merged = ops.sdpa_merge(ao, al)
    whole = ops.sdpa_decode(qd, kd, vd, scale=0.09)
    assert_close(merged, whole.float(), "merged vs unsplit kernel", rel_tol=3e-3, abs_tol=4e-3)
    for b in range(B):
        assert_close(merged[b], oracle_decode(q[b], k[b], v[b], 0.09)[0][0], f"seq {b}")


def test_error_statuses(ops):
    from arcaine_b200 import _lib
    q = torch.zeros(2, 34, 128, dtype=torch.bfloat16, device="cuda")
    k = torch.zeros(2, 64, 2, 128, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(ops.ArcError) as e:
        ops.sdpa_decode(q, k, k, scale=1.0)
    assert e.value.status == _lib.ARC_ERR_UNSUPPORTED_GQA
    q = torch.zeros(2, 4, 64, dtype=torch.bfloat16, device="cuda")
    k = torch.zeros(2, 64, 2, 64, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(ops.ArcError) as e:
        ops.sdpa_decode(q, k, k, scale=1.0)
    assert e.value.status == _lib.ARC_ERR_UNSUPPORTED_HEAD_DIM
    # raw ABI: workspace too small
    q = torch.zeros(2, 4, 128, dtype=torch.bfloat16, device="cuda")
    k = torch.zeros(2, 64, 2, 128, dtype=torch.bfloat16, device="cuda")
    p = _lib.DecodeParams()
    p.q, p.k, p.v, p.out = q.data_ptr(), k.data_ptr(), k.data_ptr(), q.data_ptr()
    p.batch, p.nq, p.nkv, p.hd, p.kv_len_uniform, p.max_kv_len = 2, 4, 2, 128, 64, 64
    p.q_stride_b = p.o_stride_b = 512
    p.kv_stride_b, p.kv_stride_t, p.kv_rows_total, p.scale = 64, 256, 128, 1.0
    L = _lib.load()
    assert L.arc_sdpa_decode_workspace_bytes(C.byref(p)) > 0
    ws = torch.zeros(64, dtype=torch.uint8, device="cuda")
    p.workspace, p.workspace_bytes = ws.data_ptr(), 64
    assert L.arc_sdpa_decode(C.byref(p), None) == _lib.ARC_ERR_WORKSPACE_TOO_SMALL


def test_peer_wait_gives_up_with_a_status_and_the_device_stays_usable(ops):
    """Sequence-sharded decode on one GPU with a second "rank" whose records never come: the merge
    kernel's wait for them is bounded, expires (a few ms here), records FAULT_WAIT_PEER with the
    missing source rank and returns; while the status is set launches do nothing; after a clear the
    same call without the exchange is correct.  Nothing faults or hangs: the flag is simply never set."""
    B, nq, nkv, hd, n = 1, 4, 1, 128, 300
    q, k, v = seeded_bf16(B, nq, hd, seed=71), seeded_bf16(B, n, nkv, hd, seed=72), seeded_bf16(B, n, nkv, hd, seed=73)
    xbuf = torch.zeros(ops.exchange_bytes(2, B, nq, hd), dtype=torch.uint8, device="cuda")
    peers = torch.tensor([xbuf.data_ptr(), xbuf.data_ptr()], dtype=torch.int64, device="cuda")
    out = torch.full((B, nq, hd), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.sdpa_decode(q.cuda(), k.cuda(), v.cuda(), scale=hd ** -0.5, out=out, exchange=(peers, 2, 0, 1),
                    exchange_wait_cycles=20_000_000)
    assert ops.device_status() == (ops.FAULT_WAIT_PEER, 1)   # source rank 1 never raised its flag
    assert (out.float() == 7.0).all()                         # the merged result was never written
    # sticky: a launch made while the status is set returns at once without touching its output
    ops.sdpa_decode(q.cuda(), k.cuda(), v.cuda(), scale=hd ** -0.5, out=out)
    torch.cuda.synchronize()
    assert (out.float() == 7.0).all()
    ops.clear_device_status()
    assert ops.device_status() == (0, 0)
    got = ops.sdpa_decode(q.cuda(), k.cuda(), v.cuda(), scale=hd ** -0.5, out=out)
    wf, _, _ = oracle_decode(q[0], k[0], v[0], hd ** -0.5)
    assert_close(got[0], wf[0], "decode after the status was cleared")


def test_exchange_fold_with_the_other_ranks_record_already_in_place(ops):
    """The cross-rank fold of the sequence-sharded decode on one GPU, without two kernels waiting for each
    other: "rank 1"'s record is computed first (return_partial) and written into rank 0's exchange buffer
    in the wire format — 8-byte (value, step) words, log-sum-exp in word hd — then rank 0's call finds it
    there, never waits, and must produce the attention over both halves of the keys, gate included."""
    B, nq, nkv, hd, n, step = 2, 8, 2, 128, 700, 5
    q, k, v = seeded_bf16(B, nq, hd, seed=91), seeded_bf16(B, n, nkv, hd, seed=92), seeded_bf16(B, n, nkv, hd, seed=93)
    gate = seeded_bf16(B, nq, hd, seed=94)
    qd, kd, vd, gd = q.cuda(), k.cuda(), v.cuda(), gate.cuda()
    half = 384
    _, o1, l1 = ops.sdpa_decode(qd, kd[:, half:].contiguous(), vd[:, half:].contiguous(), scale=hd ** -0.5, return_partial=True)
    rows, words = B * nq, hd + 2
    assert ops.exchange_bytes(2, B, nq, hd) == 2 * 2 * rows * words * 8
    xbuf = torch.zeros(2, 2, rows, words, 2, dtype=torch.int32, device="cuda")  # [parity][source][row][word][value, step]
    rec = xbuf[step & 1, 1]
    rec[:, :hd, 0] = o1.reshape(rows, hd).contiguous().view(torch.int32)
    rec[:, hd, 0] = l1.reshape(rows).contiguous().view(torch.int32)
    rec[:, :, 1] = step
    scratch = torch.zeros_like(xbuf)  # where rank 0's words for "rank 1" go
    peers = torch.tensor([xbuf.data_ptr(), scratch.data_ptr()], dtype=torch.int64, device="cuda")
    out = ops.sdpa_decode(qd, kd[:, :half].contiguous(), vd[:, :half].contiguous(), scale=hd ** -0.5, gate=gd,
                          exchange=(peers, 2, 0, step), exchange_wait_cycles=20_000_000)
    assert ops.device_status() == (0, 0)
    whole = ops.sdpa_decode(qd, kd, vd, scale=hd ** -0.5, gate=gd)
    assert_close(out, whole.float(), "two halves folded vs one pass", rel_tol=4e-3, abs_tol=2e-3)
    for b in range(B):
        _, want, _ = oracle.sdpa_f32(q[b:b + 1], k[b], v[b], scale=hd ** -0.5, gate=gate[b:b + 1], want_lse=True)
        assert_close(out[b], want[0].float(), f"sequence {b}")
    # rank 0's own words went out to both buffers, tagged with the step
    assert (xbuf[step & 1, 0, :, :, 1] == step).all() and (scratch[step & 1, 0, :, :, 1] == step).all()


@pytest.mark.parametrize("on_device", [False, True])
@pytest.mark.parametrize("ctas,launches", [(0, 1), (148, 2)])
def test_no_form_writes_a_result_under_a_status(ops, on_device, ctas, launches):
    """Any status keeps a call from its outputs, whichever form it takes and whoever knows the lengths.  (A wait that runs out
    in the middle of the one-launch form does the same through a flag in every CTA of the cluster; it cannot be made to run
    out here without a broken kernel.)"""
    B, nq, nkv, hd, n = 2, 8, 2, 128, 300
    q, k = seeded_bf16(B, nq, hd, seed=1).cuda(), seeded_bf16(B, n, nkv, hd, seed=2).cuda()
    lens = torch.full((B,), n, dtype=torch.int32, device="cuda")
    ops.sdpa_decode(q, k, k, scale=0.1, kv_len=lens + 1)  # past the cache: sets a status
    assert ops.device_status()[0] == ops.FAULT_BAD_KV_RANGE
    out, o32, lse = (torch.full(s, 3.0, dtype=t, device="cuda") for s, t in
                     (((B, nq, hd), torch.bfloat16), ((B, nq, hd), torch.float32), ((B, nq), torch.float32)))
    before = ops.launch_count()
    ops.sdpa_decode(q, k, k, scale=0.1, kv_len=lens if on_device else n, num_ctas=ctas, out=out, return_partial=True, partial_out=o32,
                    partial_lse=lse)
    assert ops.launch_count() - before == launches
    torch.cuda.synchronize()
    assert all((t.float() == 3.0).all() for t in (out, o32, lse))
    ops.clear_device_status()
    assert not (ops.sdpa_decode(q, k, k, scale=0.1, kv_len=lens if on_device else n, num_ctas=ctas, out=out).float() == 3.0).all()


def test_exchange_of_one_rank_as_a_list(ops):
    q, k, v = seeded_bf16(1, 4, 128, seed=71).cuda(), seeded_bf16(1, 300, 1, 128, seed=72).cuda(), seeded_bf16(1, 300, 1, 128, seed=73).cuda()
    peers = torch.zeros(1, dtype=torch.int64, device="cuda")
    want = ops.sdpa_decode(q, k, v, scale=0.1)
    for exchange in ((peers, 1, 0, 1), [peers, 1, 0, 1]):
        assert torch.equal(ops.sdpa_decode(q, k, v, scale=0.1, exchange=exchange), want)
    with pytest.raises((ValueError, IndexError)):
        ops.sdpa_decode(q, k, v, scale=0.1, exchange=[peers, 1, 0])


def test_device_side_length_past_the_cache_is_a_status_not_a_wrong_result(ops):
    from arcaine_b200 import _lib
    B, nq, nkv, hd, cap = 2, 8, 2, 128, 64
    q, k, v = seeded_bf16(B, nq, hd, seed=81), seeded_bf16(B, cap, nkv, hd, seed=82), seeded_bf16(B, cap, nkv, hd, seed=83)
    out = torch.full((B, nq, hd), 3.0, dtype=torch.bfloat16, device="cuda")
    bad = torch.tensor([cap, cap + 1], dtype=torch.int32, device="cuda")  # sequence 1 claims one row too many
    ops.sdpa_decode(q.cuda(), k.cuda(), v.cuda(), scale=0.1, kv_len=bad, out=out)
    assert ops.device_status() == (ops.FAULT_BAD_KV_RANGE, 1)
    code, detail = C.c_uint32(0), C.c_uint32(0)
    assert _lib.load().arc_sdpa_device_status(C.byref(code), C.byref(detail)) == _lib.ARC_ERR_DEVICE_BAD_RANGE
    assert (out.float() == 3.0).all()
    ops.clear_device_status()
    # known on the host: refused before anything is launched
    with pytest.raises(ValueError):
        ops.sdpa_decode(q.cuda(), k.cuda(), v.cuda(), scale=0.1, kv_len=cap + 1, out=out)
    good = torch.tensor([cap, 5], dtype=torch.int32, device="cuda")
    got = ops.sdpa_decode(q.cuda(), k.cuda(), v.cuda(), scale=0.1, kv_len=good, out=out)
    wf, _, _ = oracle_decode(q[1], k[1, :5], v[1, :5], 0.1)
    assert_close(got[1], wf[0], "decode after the status was cleared")


def test_empty_cache_slice_gives_empty_records(ops):
    """A sequence-sharded rank whose slice holds no keys still produces its records: zeros with lse = -inf."""
    B, nq, nkv, hd = 2, 8, 2, 128
    q = seeded_bf16(B, nq, hd, seed=91).cuda()
    k = torch.empty(B, 0, nkv, hd, dtype=torch.bfloat16, device="cuda")
    out, o32, lse = ops.sdpa_decode(q, k, k, scale=0.1, return_partial=True)
    assert torch.count_nonzero(out.float()) == 0 and torch.count_nonzero(o32) == 0
    assert torch.isinf(lse).all() and (lse < 0).all()


@pytest.mark.parametrize("B,nq,nkv,hd,lens", [
    (1, 24, 4, 256, [1]),                      # one key: seven of eight CTAs of a cluster have none
    (1, 6, 1, 128, [1000]),                    # one group of heads
    (5, 32, 2, 128, [129, 16, 0, 640, 333]),   # 16 query heads per KV head, an empty sequence
    (37, 24, 4, 256, [i * 7 for i in range(37)]),   # as many clusters of one CTA as fit
    (70, 16, 8, 256, [40 + i for i in range(70)]),  # several KV heads per CTA
])
def test_one_launch_form(ops, B, nq, nkv, hd, lens):
    """Short calls: a cluster per sequence and group of heads writes the result itself (one launch), from a block cache and
    from a packed one, with the gate and with the partial outputs."""
    cap = max(lens)
    q, k, v = seeded_bf16(B, nq, hd, seed=1), seeded_bf16(B, cap, nkv, hd, seed=2), seeded_bf16(B, cap, nkv, hd, seed=3)
    g = seeded_bf16(B, nq, hd, seed=4)
    kl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    before = ops.launch_count()
    out, o32, lse = ops.sdpa_decode(q.cuda(), k.cuda(), v.cuda(), scale=hd ** -0.5, kv_len=kl, gate=g.cuda(), return_partial=True)
    assert ops.launch_count() - before == 1
    kp, vp = (torch.cat([t[b, :n] for b, n in enumerate(lens)]).cuda() for t in (k, v))
    offs = torch.tensor([sum(lens[:b]) for b in range(B)], dtype=torch.int64, device="cuda")
    packed = ops.sdpa_decode(q.cuda(), kp, vp, scale=hd ** -0.5, kv_len=kl, kv_row_offset=offs, gate=g.cuda())
    two = ops.sdpa_decode(q.cuda(), k.cuda(), v.cuda(), scale=hd ** -0.5, kv_len=kl, gate=g.cuda(), num_ctas=148)  # shares and merge
    assert_close(packed, two.float(), "packed", rel_tol=5e-3)
    for b in range(0, B, max(1, B // 8)):
        if lens[b] == 0:
            assert torch.count_nonzero(out[b].float()) == 0 and torch.isinf(lse[b]).all()
            continue
        wf, _, wl = oracle_decode(q[b], k[b, :lens[b]], v[b, :lens[b]], hd ** -0.5)
        _, wgb, _ = oracle_decode(q[b], k[b, :lens[b]], v[b, :lens[b]], hd ** -0.5, gate=g[b])
        assert_close(o32[b], wf[0], f"seq {b} f32", rel_tol=3e-3, abs_tol=5e-3)
        assert_close(out[b], wgb[0].float(), f"seq {b} gated")
        assert torch.allclose(lse[b].cpu(), wl[0], atol=2e-3)


@pytest.mark.parametrize("lens,nq,nkv,hd,block,packed", [
    ([20000] + [400] * 31, 16, 2, 128, 2, 2),  # its cluster alone would take three times as long
    ([8000] + [14] * 15, 24, 4, 256, 2, 2),
    ([700] * 3, 24, 4, 256, 1, 1),             # whatever the lengths were, a cluster is fast enough
    ([500, 16000], 8, 4, 128, 1, 1),
])
def test_batches_that_may_be_one_long_sequence(ops, lens, nq, nkv, hd, block, packed):
    """Launches of a call whose lengths only the device knows, over a block cache as long as the longest sequence and over
    a packed one; the same result either way."""
    B, cap = len(lens), max(lens)
    q = seeded_bf16(B, nq, hd, seed=1).cuda()
    kp, vp = seeded_bf16(sum(lens), nkv, hd, seed=2).cuda(), seeded_bf16(sum(lens), nkv, hd, seed=3).cuda()
    offs = [sum(lens[:b]) for b in range(B)]
    k, v = (torch.zeros(B, cap, nkv, hd, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    for b, n in enumerate(lens):
        k[b, :n], v[b, :n] = kp[offs[b]:offs[b] + n], vp[offs[b]:offs[b] + n]
    kl, ko = torch.tensor(lens, dtype=torch.int32, device="cuda"), torch.tensor(offs, dtype=torch.int64, device="cuda")
    launches = []
    for call in (lambda: ops.sdpa_decode(q, k, v, scale=hd ** -0.5, kv_len=kl),
                 lambda: ops.sdpa_decode(q, kp, vp, scale=hd ** -0.5, kv_len=kl, kv_row_offset=ko)):
        before = ops.launch_count()
        out = call()
        launches.append(ops.launch_count() - before)
        for b in {0, 1, B - 1}:
            want = oracle_decode(q[b].cpu(), kp[offs[b]:offs[b] + lens[b]].cpu(), vp[offs[b]:offs[b] + lens[b]].cpu(), hd ** -0.5)
            assert_close(out[b], want[0][0], f"seq {b}")
    assert launches == [block, packed]


@pytest.mark.parametrize("B,nq,nkv,hd,length,ctas", [
    (1, 24, 4, 256, 6100, 148),   # few rows: 64 columns of a row per merge block, every share one record
    (1, 6, 2, 128, 9000, 600),    # more records of a row than a lane of the merge block keeps of their log-sum-exps
    (2, 16, 16, 128, 700, 64),    # two slices per record at a sequence's end
    (1, 32, 2, 128, 3000, 40),    # sixteen query heads per KV head
    (40, 16, 8, 256, 130, 148),   # many rows: whole rows per block
])
def test_lengths_known_to_the_host_and_merge_blocks(ops, B, nq, nkv, hd, length, ctas):
    """A length the host states gives what the same length on the device gives, bit for bit: shares found before or
    after the wait for the kernels in front, one launch or two; all against the oracle."""
    q, k, v, g = seeded_bf16(B, nq, hd, seed=1), seeded_bf16(B, length, nkv, hd, seed=2), seeded_bf16(B, length, nkv, hd, seed=3), seeded_bf16(B, nq, hd, seed=4)
    dev = [t.cuda() for t in (q, k, v)]
    kl = torch.full((B,), length, dtype=torch.int32, device="cuda")
    for n in (0, ctas):
        on_host = ops.sdpa_decode(*dev, scale=hd ** -0.5, gate=g.cuda(), num_ctas=n, return_partial=True)
        on_device = ops.sdpa_decode(*dev, scale=hd ** -0.5, kv_len=kl, gate=g.cuda(), num_ctas=n, return_partial=True)
        assert all(torch.equal(a, b) for a, b in zip(on_host, on_device))
        for b in range(0, B, max(1, B // 4)):
            wf, _, wl = oracle_decode(q[b], k[b], v[b], hd ** -0.5)
            _, wgb, _ = oracle_decode(q[b], k[b], v[b], hd ** -0.5, gate=g[b])
            assert_close(on_host[1][b], wf[0], f"seq {b} f32", rel_tol=3e-3, abs_tol=5e-3)
            assert_close(on_host[0][b], wgb[0].float(), f"seq {b} gated")
            assert torch.allclose(on_host[2][b].cpu(), wl[0], atol=2e-3)


@pytest.mark.parametrize("B,nq,nkv,n", [
    # groups of six and of sixteen heads, of one, which takes four slices; one step of six slices, its last full one, two steps, a
    # ragged second one
    *((1, nq, nkv, n) for nq, nkv in ((24, 4), (8, 8), (16, 1)) for n in (513, 768, 769, 1501)),
    # a CTA alone a sequence and KV head: one step and three of six slices, groups of one, four and eight heads
    (16, 8, 8, 65), (16, 8, 8, 270), (60, 8, 2, 288), (40, 16, 2, 257), (110, 8, 1, 96),
])
def test_one_launch_form_in_steps_of_six_slices(ops, B, nq, nkv, n):
    q, k, v, g = (seeded_bf16(*shape, seed=400 + i) for i, shape in enumerate([(B, nq, 256), (B, n + 30, nkv, 256), (B, n + 30, nkv, 256), (B, nq, 256)]))
    before = ops.launch_count()
    got = ops.sdpa_decode(q.cuda(), k.cuda(), v.cuda(), scale=0.0625, kv_len=n, gate=g.cuda())
    assert ops.launch_count() - before == 1
    for b in {0, B // 2, B - 1}:
        assert_close(got[b], oracle_decode(q[b], k[b, :n], v[b, :n], 0.0625, gate=g[b])[1][0].float(), f"{n} keys, sequence {b}")


def check_ragged_batch(ops, q, k, v, g, lens, rows=None):
    """One launch, and every sixth sequence's results against the oracle; rows: first rows of a packed cache."""
    hd = q.shape[2]
    before = ops.launch_count()
    got, o32, lse = ops.sdpa_decode(q.cuda(), k.cuda(), v.cuda(), scale=hd ** -0.5, kv_len=torch.tensor(lens, dtype=torch.int32, device="cuda"),
                                    kv_row_offset=None if rows is None else torch.tensor(rows, dtype=torch.int64, device="cuda"),
                                    gate=g.cuda(), return_partial=True)
    assert ops.launch_count() - before == 1
    for b in sorted({*range(0, len(lens), max(1, len(lens) // 6)), len(lens) - 1}):
        kb, vb = (k[b, :lens[b]], v[b, :lens[b]]) if rows is None else (k[rows[b]:rows[b] + lens[b]], v[rows[b]:rows[b] + lens[b]])
        if lens[b] == 0:
            assert torch.count_nonzero(got[b].float()) == 0 and torch.isinf(lse[b]).all()
            continue
        wf, _, wl = oracle_decode(q[b], kb, vb, hd ** -0.5)
        _, wgb, _ = oracle_decode(q[b], kb, vb, hd ** -0.5, gate=g[b])
        assert_close(o32[b], wf[0], f"seq {b} f32", rel_tol=3e-3, abs_tol=5e-3)
        assert_close(got[b], wgb[0].float(), f"seq {b} gated")
        assert torch.allclose(lse[b].cpu(), wl[0], atol=2e-3)


@pytest.mark.parametrize("B,nq,nkv,hd,n", [
    (12, 16, 2, 128, 1700),  # 24 clusters: five CTAs each, four of which finish columns
    (5, 24, 4, 256, 900),    # 20: six would fit, but four are enough for so few keys
    (7, 24, 4, 256, 1000),   # 28: four of five
    (45, 8, 1, 128, 600),    # three, two of which finish columns
    (12, 32, 2, 256, 800),   # sixteen heads a KV head
])
def test_one_launch_form_in_clusters_of_any_size(ops, B, nq, nkv, hd, n):
    lens = [max(1, n - 53 * b) for b in range(B)]
    q, k, v, g = (seeded_bf16(*shape, seed=500 + i) for i, shape in enumerate([(B, nq, hd), (B, n, nkv, hd), (B, n, nkv, hd), (B, nq, hd)]))
    check_ragged_batch(ops, q, k, v, g, lens)


@pytest.mark.parametrize("B,nq,nkv,hd,n", [
    (2, 3, 1, 256, 100), (1, 7, 7, 128, 500), (3, 9, 1, 256, 700), (2, 13, 1, 128, 300),  # an odd number of rows, one and two tiles of heads
    (30, 25, 5, 128, 200),                          # a CTA alone, one KV head
    (60, 15, 5, 128, 90), (100, 14, 2, 256, 50),    # several
])
def test_one_launch_form_of_any_group(ops, B, nq, nkv, hd, n):
    lens = [0 if b % 20 == 10 else max(1, n - b % 7 * 11) for b in range(B)]
    q, k, v, g = (seeded_bf16(*shape, seed=700 + i) for i, shape in enumerate([(B, nq, hd), (B, n, nkv, hd), (B, n, nkv, hd), (B, nq, hd)]))
    check_ragged_batch(ops, q, k, v, g, lens)


@pytest.mark.parametrize("B,nq,nkv,hd,n,warp_keys", [
    (12, 16, 2, 128, 1700, 64), (2, 32, 2, 128, 700, 32), (5, 24, 4, 256, 900, 96), (1, 8, 8, 256, 1501, 64),  # clusters
    (16, 8, 8, 256, 270, 64),  # a CTA alone
])
def test_one_launch_form_keeps_values_that_its_records_can_hold(ops, B, nq, nkv, hd, n, warp_keys):
    """All scores zero, all values as large as the sum over a warp's keys, of which there are `warp_keys` at most, lets them be: the
    result is that value, whatever the sum over the CTA's keys."""
    q, k = torch.zeros(B, nq, hd, dtype=torch.bfloat16), seeded_bf16(B, n, nkv, hd, seed=720)
    value = torch.tensor(3.3e38 / warp_keys).bfloat16()
    v = value.expand(B, n, nkv, hd).contiguous()
    before = ops.launch_count()
    out, o32, lse = ops.sdpa_decode(q.cuda(), k.cuda(), v.cuda(), scale=0.1, kv_len=n, return_partial=True)
    assert ops.launch_count() - before == 1
    assert (out == value.cuda()).all() and ((o32 / value.float().cuda() - 1).abs() <= 1e-6).all()
    assert torch.allclose(lse.cpu(), torch.full((B, nq), n, dtype=torch.float32).log(), atol=1e-6)


@pytest.mark.parametrize("B,nq,nkv,hd,n", [(12, 16, 2, 128, 1700), (5, 24, 4, 256, 900), (1, 24, 4, 256, 600)])
def test_one_launch_form_has_the_log_sum_exps_of_the_shares(ops, B, nq, nkv, hd, n):
    """They are no further off than those that equal shares and a merge give (1.6 times as far with a rounding and an approximate
    logarithm more)."""
    q, k, v = (seeded_bf16(*shape, seed=730 + i).cuda() for i, shape in enumerate([(B, nq, hd), (B, n, nkv, hd), (B, n, nkv, hd)]))
    want = torch.einsum("bhgd,bnhd->bhgn", q.double().view(B, nkv, -1, hd), k.double()).mul(hd ** -0.5).logsumexp(-1).view(B, nq)
    off, launches = [], []
    for ctas in (0, 148):
        before = ops.launch_count()
        lse = ops.sdpa_decode(q, k, v, scale=hd ** -0.5, kv_len=n, num_ctas=ctas, return_partial=True)[2]
        launches.append(ops.launch_count() - before)
        off.append((lse.double() / want - 1).square().mean().sqrt().item())
    assert launches == [1, 2] and off[0] <= 1.25 * off[1], off


@pytest.mark.parametrize("B,nq,nkv,hd,n", [(12, 16, 2, 128, 1700), (2, 32, 2, 128, 700), (1, 24, 4, 256, 600), (30, 25, 5, 128, 200)])
def test_one_launch_form_hands_on_what_is_no_number(ops, B, nq, nkv, hd, n):
    """A query, or a key, that is none: NaN in the results and in the log-sum-exps of the heads that see it, so that a merge with
    another part keeps it; the other heads, and a head whose keys all score -inf, as ever."""
    q, k, v = (seeded_bf16(*shape, seed=740 + i).cuda() for i, shape in enumerate([(B, nq, hd), (B, n, nkv, hd), (B, n, nkv, hd)]))
    G = nq // nkv
    q[:, 1, 5] = float("nan")  # a head of the first group
    k[0, n // 2, nkv - 1, 3] = float("nan")  # the last group of the first sequence
    out, o32, lse = ops.sdpa_decode(q, k, v, scale=hd ** -0.5, kv_len=n, return_partial=True)
    bad = torch.zeros(B, nq, dtype=torch.bool, device="cuda")
    bad[:, 1] = True
    bad[0, nq - G:] = True
    assert torch.equal(lse.isnan(), bad) and torch.equal(o32.isnan(), bad[..., None].expand_as(o32)) and torch.equal(out.isnan(), o32.isnan())
    part = torch.randn(1, B * nq, hd, device="cuda"), torch.zeros(1, B * nq, device="cuda")
    merged = ops.sdpa_merge(torch.cat([o32.view(1, -1, hd), part[0]]), torch.cat([lse.view(1, -1), part[1]]))
    assert torch.equal(merged.view(B, nq, hd).isnan(), o32.isnan())
    q[:, 1], q[..., 0], k[0, n // 2, nkv - 1, 3], k[..., 0] = 0.0, 1.0, 0.0, -float("inf")
    out, o32, lse = ops.sdpa_decode(q, k, v, scale=hd ** -0.5, kv_len=n, return_partial=True)
    assert not out.any() and not o32.any() and (lse == -float("inf")).all()


@pytest.mark.parametrize("B,nq,nkv,total", [
    (5, 24, 4, 7600),   # 20 clusters of six CTAs in steps of six slices
    (12, 16, 2, 7600),  # 24 of five, groups of eight heads
    (40, 6, 1, 4300),   # 40 of three, two of which finish columns
    (10, 32, 2, 1900),  # 20 of six, sixteen heads a KV head
])
def test_one_launch_form_in_uneven_clusters_at_head_dim_256(ops, B, nq, nkv, total):
    """Packed caches in which one sequence could hold so many keys that a power of two of CTAs would be judged too slow for it
    and equal shares, two launches, taken: one launch says that all CTAs that fit were.  Two sequences have nearly all
    keys, the others so few that the last CTAs have none."""
    short = [b * 7 % 40 for b in range(B - 2)]  # (none at all for the first)
    lens = [*short, (total - sum(short)) // 3, total - sum(short) - (total - sum(short)) // 3]
    rows = [sum(lens[:b]) for b in range(B)]
    q, k, v, g = (seeded_bf16(*shape, seed=600 + i) for i, shape in enumerate([(B, nq, 256), (total, nkv, 256), (total, nkv, 256), (B, nq, 256)]))
    check_ragged_batch(ops, q, k, v, g, lens, rows)
