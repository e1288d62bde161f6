"""Scratch memory belongs to one call: calls in flight at the same time, from threads or on streams of their own, do not meet in it."""
import contextlib
import threading

import pytest
import torch


@pytest.fixture
def lbl(native_lib):
    from ipex_llm_b200.transformers import low_bit_linear
    return low_bit_linear


@pytest.mark.parametrize("entry", ["matmul", "mlp", "one token of experts"])
def test_calls_that_overlap_have_scratch_of_their_own(lbl, monkeypatch, entry):
    """the kernels' place is taken by a recorder that runs a second call, from another thread, inside the first one's"""
    ranges = []

    def recorder(position):
        def call(*args):
            at, size = args[position].value if hasattr(args[position], "value") else args[position], args[position + 1]
            ranges.append((at, at + size))
            if len(ranges) == 1:
                t = threading.Thread(target=run)
                t.start()
                t.join()
        return call
    monkeypatch.setattr(lbl.ggml, "lowbit_matmul_cuda", recorder(11))
    monkeypatch.setattr(lbl.ggml, "lowbit_mlp_cuda", recorder(11))
    monkeypatch.setattr(lbl.ggml, "lowbit_moe_cuda", recorder(18))
    monkeypatch.setattr(lbl, "_raw_stream", lambda d: 0)
    monkeypatch.setattr(lbl, "_stream_ptr", lambda d: 0)
    monkeypatch.setattr(lbl, "_on_device", lambda d: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    w, x = torch.zeros(4096 * 256, dtype=torch.uint8), torch.zeros(100, 256)
    table = torch.zeros(4, dtype=torch.int64)

    def run():
        if entry == "matmul":
            lbl.lowbit_matmul(x, w, (512, 256), lbl.SYM_INT4)
        elif entry == "mlp":
            lbl.mlp_forward(x, w, w, 100, 256, 512, lbl.SILU, lbl.SYM_INT4)
        else:
            lbl.moe_forward_vec(x[:1], table[None, :2], torch.zeros(1, 2), table, table, table, 256, 512, lbl.SYM_INT4)
    run()
    (a, b), (c, d) = ranges
    assert b > a and d > c and (b <= c or d <= a)


@pytest.mark.gpu
def test_streams_do_not_meet_in_scratch(lbl, cuda_device):
    """a K-split MLP and a 32-bit matmul -- partial sums and activation planes between two launches -- on four streams at once"""
    weights = [lbl.FP4Params(torch.randn(2048, 4096, device=cuda_device) * 0.02, qtype=lbl.SYM_INT4).to(cuda_device).data for _ in range(2)]
    xs = [torch.randn(100, 4096, device=cuda_device) for _ in range(4)]

    def run(x):
        return (lbl.mlp_forward(x.half(), *weights, 100, 4096, 2048, lbl.SILU, lbl.SYM_INT4), lbl.lowbit_matmul(x, weights[0], (2048, 4096), lbl.SYM_INT4))
    want = [run(x) for x in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    got = []
    for _ in range(30):
        for x, s in zip(xs, streams):
            with torch.cuda.stream(s):
                got.append(run(x))
    torch.cuda.synchronize()
    for i, (a, b) in enumerate(got):
        assert torch.equal(a, want[i % 4][0]) and torch.equal(b, want[i % 4][1])


def test_decode_attention_has_scratch_of_its_own(native_lib, monkeypatch):
    from ipex_llm_b200.transformers import kv
    ranges = []

    def call(q, k, v, mask, causal, scale, out, ws, stream):
        ranges.append((ws.data_ptr(), ws.data_ptr() + ws.numel()))
        if len(ranges) == 1:
            t = threading.Thread(target=run)
            t.start()
            t.join()
    monkeypatch.setattr(kv.ggml, "lowbit_sdp_fp8", call)
    monkeypatch.setattr(kv, "_stream", lambda d: 0)
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    cache = torch.zeros(2, 4, 1000, 128, dtype=torch.uint8)

    def run():
        kv.sdp_fp8(torch.zeros(2, 8, 1, 128), cache, cache, None, 0.1)
    run()
    (a, b), (c, d) = ranges
    assert b > a and d > c and (b <= c or d <= a)


@pytest.mark.gpu
def test_decode_attention_on_several_streams(native_lib, cuda_device):
    from ipex_llm_b200.transformers import kv
    cache = [torch.randn(2, 4, 3000, 128, device=cuda_device).to(torch.float8_e5m2).view(torch.uint8) for _ in range(2)]
    qs = [torch.randn(2, 16, 1, 128, device=cuda_device).half() for _ in range(4)]
    want = [kv.sdp_fp8(q, *cache, None, 0.1) for q in qs]
    streams = [torch.cuda.Stream() for _ in qs]
    torch.cuda.synchronize()
    got = []
    for _ in range(50):
        for q, s in zip(qs, streams):
            with torch.cuda.stream(s):
                got.append(kv.sdp_fp8(q, *cache, None, 0.1))
    torch.cuda.synchronize()
    assert all(torch.equal(o, want[i % 4]) for i, o in enumerate(got))
