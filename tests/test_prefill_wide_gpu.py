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
