"""Calls on two CUDA streams at once, with a workspace for each and with none, from captured graphs and over scratch that
nobody else holds: the library keeps no per-call state outside the caller's buffers (the status word is the one thing the
calls share), so the results must be the ones the same calls give one after the other."""
import weakref

import pytest
import torch

from helpers import seeded_bf16

pytestmark = pytest.mark.gpu


def test_prefill_and_decode_on_two_streams_equal_the_serial_results():
    from arcaine_b200 import ops
    ops.clear_device_status()
    dev = torch.device("cuda", 0)
    # stream A: canvas-like prefill (key range in parts) and a windowed hd128 prefill (two-tile kernel)
    qa, ka, va = (seeded_bf16(256, 8, 256, seed=1).cuda(), seeded_bf16(2304, 4, 256, seed=2).cuda(),
                  seeded_bf16(2304, 4, 256, seed=3).cuda())
    qw, kw, vw = (seeded_bf16(2048, 16, 128, seed=4).cuda(), seeded_bf16(2048, 8, 128, seed=5).cuda(),
                  seeded_bf16(2048, 8, 128, seed=6).cuda())
    # stream B: gated decode with per-sequence lengths and a long single-sequence decode
    qd, kd, vd = (seeded_bf16(6, 24, 256, seed=7).cuda(), seeded_bf16(6, 3000, 4, 256, seed=8).cuda(),
                  seeded_bf16(6, 3000, 4, 256, seed=9).cuda())
    gd = seeded_bf16(6, 24, 256, seed=10).cuda()
    lens = torch.tensor([3000, 17, 1024, 2999, 1, 512], dtype=torch.int32, device=dev)
    ql, kl, vl = (seeded_bf16(1, 16, 128, seed=11).cuda(), seeded_bf16(1, 40000, 2, 128, seed=12).cuda(),
                  seeded_bf16(1, 40000, 2, 128, seed=13).cuda())

    def side_a(ws):
        return (ops.sdpa_prefill(qa, ka, va, scale=0.0625, workspace=ws),
                ops.sdpa_prefill(qw, kw, vw, scale=128 ** -0.5, mask_type=ops.MASK_CAUSAL, window=512, workspace=ws))

    def side_b(ws):
        return (ops.sdpa_decode(qd, kd, vd, scale=0.0625, kv_len=lens, gate=gd, workspace=ws),
                ops.sdpa_decode(ql, kl, vl, scale=128 ** -0.5, workspace=ws))

    ws_a, ws_b = ops.Workspace(dev), ops.Workspace(dev)
    want = side_a(ws_a) + side_b(ws_b)
    torch.cuda.synchronize()
    sa, sb = torch.cuda.Stream(), torch.cuda.Stream()
    got_a, got_b = [], []
    for _ in range(8):  # several rounds, so that the two sides really overlap
        with torch.cuda.stream(sa):
            got_a.append(side_a(ws_a))
        with torch.cuda.stream(sb):
            got_b.append(side_b(ws_b))
    torch.cuda.synchronize()
    assert ops.device_status() == (0, 0)
    for ra, rb in zip(got_a, got_b):
        for g, w in zip(ra + rb, want):
            assert torch.equal(g, w)


def canvas_and_masked(seed):
    """A canvas step (partial records) and a masked layer (bits of the mask) of one user, through calls that take no
    workspace: head dim 256."""
    from arcaine_b200 import ops
    seq, prompt, nq, nkv, hd = 256, 1500 + 300 * seed, 8, 4, 256
    kv = seq + prompt
    q = (seeded_bf16(seq, nq, hd, seed=20 + seed).float() * hd ** -0.5).bfloat16().cuda()
    k, v = seeded_bf16(kv, nkv, hd, seed=30 + seed).cuda(), seeded_bf16(kv, nkv, hd, seed=40 + seed).cuda()
    mask = torch.zeros(seq, kv)
    mask[torch.rand(seq, kv, generator=torch.Generator().manual_seed(seed)) < 0.5] = -float("inf")
    mask = mask.cuda()
    return lambda: (ops.gqa_attention_sdpa(q, seq, nq, hd, k, v, kv, nkv),
                    ops.gqa_attention_sdpa(q, seq, nq, hd, k, v, kv, nkv, mask, ops.MASK_EXPLICIT))


def test_calls_without_a_workspace_on_two_streams_equal_the_serial_results():
    from arcaine_b200 import ops
    ops.clear_device_status()
    sides = [canvas_and_masked(0), canvas_and_masked(1)]
    want = [side() for side in sides]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[], []]
    for _ in range(20):
        for stream, side, outs in zip(streams, sides, got):
            with torch.cuda.stream(stream):
                outs.append(side())
    torch.cuda.synchronize()
    assert ops.device_status() == (0, 0)
    for w, outs in zip(want, got):
        for o in outs:
            assert all(torch.equal(a, b) for a, b in zip(o, w))


def test_captured_calls_keep_scratch_of_their_own():
    """Two graphs replayed at once, with larger calls in between that would have grown a shared buffer."""
    from arcaine_b200 import ops
    ops.clear_device_status()
    sides = [canvas_and_masked(0), canvas_and_masked(1)]
    want = [side() for side in sides]
    graphs, outs = [], []
    for side in sides:
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            outs.append(side())
    large = canvas_and_masked(6)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(5):
        for o in outs:
            for t in o:
                t.zero_()
        torch.cuda.synchronize()
        for graph, stream in zip(graphs, streams):
            with torch.cuda.stream(stream):
                graph.replay()
        large()
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            assert all(torch.equal(a, b) for a, b in zip(o, w))
    assert ops.device_status() == (0, 0)


def test_scratch_is_held_until_the_kernels_are_enqueued():
    """A workspace that lets go of its buffer at once (as one that another thread makes grow does): the call keeps it."""
    from arcaine_b200 import ops
    launches_at_the_end = []

    class Fleeting:
        def reserve(self, nbytes):
            buf = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
            weakref.finalize(buf, lambda: launches_at_the_end.append(ops.launch_count()))
            return buf

    q, k, v = (seeded_bf16(n, h, 256, seed=50 + h).cuda() for n, h in ((256, 8), (2304, 4), (2304, 4)))
    for call in (lambda: ops.sdpa_prefill(q, k, v, scale=0.0625, workspace=Fleeting()),
                 lambda: ops.sdpa_decode(q[:1], k[None], v[None], scale=0.0625, workspace=Fleeting())):
        before = ops.launch_count()
        call()
        assert launches_at_the_end.pop() == ops.launch_count() > before
