"""Head dim 128: one tile per CTA in two chains of key blocks, and tiles dealt longest first, where either can go wrong: one
to five key blocks (a chain without any), parts of a key range without keys, scores that grow between the blocks of one
chain only, additive masks with and without values, several tiles per CTA.  (The tail of single heads behind a launch of
pairs: test_prefill_gpu.py.)  Against the CPU oracle with the tolerance of every attention test (tests/helpers.py)."""
import numpy as np
import pytest
import torch

import oracle
from helpers import assert_close, seeded_bf16
from test_prefill_gpu import ops, run_case  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [0, 2, 5])
@pytest.mark.parametrize("kv_len", [1, 128, 129, 256, 300, 512, 640])
def test_few_key_blocks(ops, kv_len, splits):
    run_case(ops, 140, kv_len, 6, 2, 128, 0.09, 0, oracle.INT_MAX, seed=kv_len, num_splits=splits, gate=kv_len % 2 == 0, lse=True)


@pytest.mark.parametrize("window", [oracle.INT_MAX, 130])
def test_causal_with_a_past_and_gate(ops, window):
    run_case(ops, 333, 900, 6, 2, 128, 0.09, 3, window, seed=4, gate=True, lse=True)


@pytest.mark.parametrize("at,gain", [(128, 40.0), (256, 40.0), (300, 200.0)])
def test_scores_that_grow_in_one_chain(ops, at, gain):
    """Keys from `at` on are larger: one chain, then the other moves its reference by more than 2^8."""
    q, k, v = seeded_bf16(130, 4, 128, seed=61), seeded_bf16(700, 2, 128, seed=62), seeded_bf16(700, 2, 128, seed=63)
    k = k.float()
    k[at:at + 128] *= gain
    k = k.bfloat16()
    out, lse = ops.sdpa_prefill(q.cuda(), k.cuda(), v.cuda(), scale=0.09, num_splits=1, return_lse=True)
    want = oracle.sdpa_f32(q, k, v, scale=0.09, want_lse=True)
    assert_close(out, want[0], f"growth at {at}")
    assert torch.allclose(lse.cpu(), want[2], atol=2e-3, rtol=1e-5)


@pytest.mark.parametrize("splits", [0, 3])
@pytest.mark.parametrize("kv_len", [300, 301])  # rows of the mask 16-byte aligned, and not
@pytest.mark.parametrize("seq,gate", [(200, False), (203, True), (73, False)])  # the mask is read eight rows at a time
def test_additive_mask(ops, kv_len, splits, seq, gate):
    nq, nkv = 4, 2
    q, k, v = seeded_bf16(seq, nq, 128, seed=71), seeded_bf16(kv_len, nkv, 128, seed=72), seeded_bf16(kv_len, nkv, 128, seed=73)
    g = seeded_bf16(seq, nq, 128, seed=74)
    mask = np.random.default_rng(7).normal(0.0, 2.0, (seq, kv_len)).astype(np.float32)
    mask[:70] = 0.0                    # blocks without values for the first two warps of rows
    mask[:, 20:60] = -np.inf
    mask[10, 128:] = np.finfo(np.float32).min
    mask[40] = -np.inf                 # a row that sees nothing
    got = ops.sdpa_prefill(q.cuda(), k.cuda(), v.cuda(), scale=0.09, mask_type=ops.MASK_EXPLICIT, mask=torch.from_numpy(mask).cuda(), num_splits=splits,
                           gate=g.cuda() if gate else None)
    want = oracle.sdpa_f32(q, k, v, scale=0.09, mask_type=oracle.MASK_EXPLICIT, mask=mask, gate=g if gate else None)
    assert_close(got, want[1].float() if gate else want[0], f"mask {kv_len}")


@pytest.mark.parametrize("gate", [False, True])
@pytest.mark.parametrize("copies", [0, 2])
def test_vision_blocks_gated_and_copied(ops, gate, copies):
    seq, kv_len, nq, nkv = 300, 420, 4, 2
    ids = np.full(kv_len, -1, dtype=np.int32)
    ids[100:190], ids[230:340], ids[400:420] = 0, 1, 2
    q, k, v, g = (seeded_bf16(n, h, 128, seed=80 + i) for i, (n, h) in enumerate([(seq, nq), (kv_len, nkv), (kv_len, nkv), (seq, nq)]))
    bufs = [torch.zeros(seq, nq, 128, dtype=torch.bfloat16, device="cuda") for _ in range(copies)]
    out = ops.sdpa_prefill(q.cuda(), k.cuda(), v.cuda(), scale=0.09, mask_type=ops.MASK_CAUSAL, window=150, block_ids=torch.from_numpy(ids).cuda(),
                           gate=g.cuda() if gate else None,
                           out_copies=torch.tensor([b.data_ptr() for b in bufs], dtype=torch.int64, device="cuda") if copies else None)
    mask = oracle.fill_causal_mask_with_block_ids(ids, seq, kv_len, kv_len - seq, 150)
    want = oracle.sdpa_f32(q, k, v, scale=0.09, mask_type=1, mask=mask, gate=g if gate else None)
    assert_close(out, want[1].float() if gate else want[0], "vision")
    torch.cuda.synchronize()
    assert all(torch.equal(b, out) for b in bufs)


@pytest.mark.parametrize("batch,seq,kv_len,nq,nkv,window", [
    (1, 1300, 1300, 16, 8, oracle.INT_MAX),   # 176 tiles, two waves
    (2, 700, 900, 16, 2, oracle.INT_MAX),     # 192 tiles of two sequences
    (1, 1900, 1900, 28, 4, oracle.INT_MAX),   # 420 tiles of an odd group, three waves
    (2, 700, 700, 28, 4, oracle.INT_MAX),     # odd group: 168 pairs of token tiles, two waves
    (1, 1664, 3200, 32, 16, oracle.INT_MAX),  # 416 tiles, three waves
    (1, 2100, 2100, 32, 16, 300),             # windowed, two waves of pairs
])
def test_tiles_longest_first(ops, batch, seq, kv_len, nq, nkv, window):
    g = torch.Generator().manual_seed(seq)
    q, k, v = (torch.randn(batch, n, h, 128, generator=g).bfloat16() for n, h in ((seq, nq), (kv_len, nkv), (kv_len, nkv)))
    out = ops.sdpa_prefill(q.cuda(), k.cuda(), v.cuda(), scale=0.09, mask_type=ops.MASK_CAUSAL, window=window).cpu()
    rows = list(range(0, seq * nq, 37)) + list(range(seq * nq - nq, seq * nq))
    for b in range(batch):
        want = oracle.sdpa_f32(q[b], k[b], v[b], scale=0.09, mask_type=3, window=window, rows=rows)[0]
        assert_close(out[b].reshape(-1, 128)[rows], want, f"sequence {b}")
