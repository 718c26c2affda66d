"""The C++ host interface (reference-shaped free functions) driven by the kbench-style program,
checked the way the reference's own bench checks its kernels: against the scalar online-softmax
kernel (src/bench/qwen35_attention_bench.cpp:124-159), here restated on the CPU."""
import os
import re
import subprocess

import numpy as np
import pytest
import torch

from helpers import assert_close
import oracle

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BIN = os.path.join(ROOT, "arcaine_b200", "arc_attention_bench")


def test_bench_cells_match_the_scalar_reference_kernel(tmp_path):
    if not os.path.exists(BIN):
        from arcaine_b200 import build
        build.build_attention_bench()
    prefills, depths = [128, 512], [0, 512, 1024]
    res = subprocess.run([BIN, "qwen35-attention", "--warmup", "1", "--runs", "3", "--dump", str(tmp_path)],
                         capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr
    rows = re.findall(r"qwen35_attention kind=(\w+) kernel=(sdpa\S*) q=(\d+) kv=(\d+) mean_ms=([\d.]+) sd_ms=[\d.]+ "
                      r"max_abs=([\d.]+) max_rel=([\d.]+)", res.stdout)
    assert len(rows) == len(prefills) + 2 * len(depths)
    # the row's own check: the library against the bench's scalar kernel on the device
    assert all(float(r[5]) <= 2e-2 for r in rows), rows
    assert len(re.findall(r"kernel=baseline", res.stdout)) == len(rows)
    listing = subprocess.run([BIN, "--list"], capture_output=True, text=True, timeout=60).stdout
    assert all(name in listing for name in ("qwen35-attention", "sdpa-prefill", "sdpa-decode"))
    nq, nkv, hd, scale = 24, 4, 256, 0.0625
    max_q, max_kv = max(prefills), max(max(prefills), max(depths) + 1)
    state = 42
    qb, state = oracle.lcg_fill(max_q * nq * hd, state)
    kb, state = oracle.lcg_fill(max_kv * nkv * hd, state)
    vb, state = oracle.lcg_fill(max_kv * nkv * hd, state)
    gb, state = oracle.lcg_fill(max_q * nq * hd, state)
    q = oracle.bits_to_bf16(qb).reshape(max_q, nq, hd)
    k = oracle.bits_to_bf16(kb).reshape(max_kv, nkv, hd)
    v = oracle.bits_to_bf16(vb).reshape(max_kv, nkv, hd)
    g = oracle.bits_to_bf16(gb).reshape(max_q, nq, hd)

    def load(kind, seq, kv):
        a = np.fromfile(os.path.join(tmp_path, f"{kind}_q{seq}_kv{kv}.bin"), dtype=np.uint16)
        return oracle.bits_to_bf16(a).reshape(seq, nq, hd)

    for seq in prefills:
        want = oracle.qwen35_online_attention(q[:seq], k[:seq], v[:seq], seq=seq, past=0, scale=scale)
        assert_close(load("prefill", seq, seq), want.float(), f"prefill {seq}")
    for d in depths:
        want = oracle.qwen35_online_attention(q[:1], k[:d + 1], v[:d + 1], seq=1, past=d, scale=scale)
        assert_close(load("decode", 1, d + 1), want.float(), f"decode depth {d}")
        assert_close(load("decode_gated", 1, d + 1), oracle.mul_sigmoid_inplace(want, g[:1]).float(), f"gated depth {d}")


PROGRAM = r"""
#include "arcaine_attention.hpp"
#include <cstdio>
#include <exception>
#include <vector>
// A canvas step and a masked layer (head dim 256) over scratch that holds nothing: a borrowed region of no bytes, and an
// owned one that would have to grow while its stream is captured.  Exit 0: the same values as with room, each time.
int main() {
    const int seq = 256, kv = 1400, nq = 8, nkv = 4, hd = 256;
    auto filled = [](size_t n, unsigned s, float by) {
        std::vector<uint16_t> h(n);
        for (auto& x : h) {
            s = s * 1664525u + 1013904223u;
            const float f = (float)((int)((s >> 16) & 1023u) - 512) / 1024.0f * by;
            unsigned u;
            __builtin_memcpy(&u, &f, 4);
            x = (uint16_t)(u >> 16);
        }
        void* d = nullptr;
        cudaMalloc(&d, n * 2);
        cudaMemcpy(d, h.data(), n * 2, cudaMemcpyHostToDevice);
        return (uint16_t*)d;
    };
    const uint16_t *q = filled((size_t)seq * nq * hd, 1, 0.2f), *k = filled((size_t)kv * nkv * hd, 2, 1.f), *v = filled((size_t)kv * nkv * hd, 3, 1.f);
    uint16_t* out = filled((size_t)seq * nq * hd, 4, 0.f);
    float* mask = nullptr;
    cudaMalloc((void**)&mask, sizeof(float) * seq * kv);
    cudaStream_t stream;
    cudaStreamCreate(&stream);
    arcaine::CudaEngine eng{0, stream};
    arcaine::fill_causal_mask(stream, mask, seq, kv, kv - seq, INT_MAX);
    auto read = [&] {
        cudaStreamSynchronize(stream);
        std::vector<uint16_t> h((size_t)seq * nq * hd);
        cudaMemcpy(h.data(), out, h.size() * 2, cudaMemcpyDeviceToHost);
        cudaMemset(out, 0, h.size() * 2);
        std::vector<float> f(h.size());
        for (size_t i = 0; i < h.size(); ++i) {
            const unsigned u = (unsigned)h[i] << 16;
            __builtin_memcpy(&f[i], &u, 4);
        }
        return f;
    };
    auto differ = [](const std::vector<float>& a, const std::vector<float>& b) {
        double d = 0, n = 0;
        for (size_t i = 0; i < a.size(); ++i) d += (double)(a[i] - b[i]) * (a[i] - b[i]), n += (double)a[i] * a[i];
        return !(n > 0 && d <= 1e-4 * n);  // (rel. L2 1e-2)
    };
    try {
        for (int masked = 0; masked < 2; ++masked) {
            auto call = [&](arcaine::SdpaWorkspace& ws) {
                arcaine::gqa_attention_sdpa(eng, q, seq, nq, hd, k, v, kv, nkv, masked ? mask : nullptr, masked, out, ws);
            };
            arcaine::SdpaWorkspace room, none(nullptr, 0), grows;
            call(room);
            const auto want = read();
            if (room.capacity() == 0) return 2;
            call(none);
            if (differ(want, read())) return 3;
            cudaGraph_t graph;
            cudaGraphExec_t exec;
            cudaStreamBeginCapture(stream, cudaStreamCaptureModeGlobal);
            call(grows);
            if (cudaStreamEndCapture(stream, &graph) != cudaSuccess || cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) return 4;
            cudaGraphLaunch(exec, stream);
            if (differ(want, read())) return 5;
            cudaGraphExecDestroy(exec);
            cudaGraphDestroy(graph);
        }
    } catch (const std::exception& e) {
        std::printf("%s\n", e.what());
        return 6;
    }
    return 0;
}
"""


def test_calls_of_head_dim_256_run_over_scratch_without_room(tmp_path):
    from arcaine_b200 import build
    src, exe, pkg = tmp_path / "room.cpp", tmp_path / "room", os.path.dirname(BIN)
    src.write_text(PROGRAM)
    cuda = os.path.dirname(os.path.dirname(build._nvcc()))
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-o", str(exe), str(src), "-I" + os.path.join(pkg, "csrc"), "-I" + os.path.join(cuda, "include"),
                           "-L" + pkg, "-larc_sdpa", "-L" + os.path.join(cuda, "lib64"), "-lcudart", "-Wl,-rpath," + pkg])
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, (res.returncode, res.stdout, res.stderr)
