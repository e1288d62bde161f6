"""Launches that overlap their starts keep the stream's order: what the kernel in front writes is read, weights too, and what stands
behind may overwrite the inputs at once.

A kernel of torch never releases its dependents early, so that behind one a launch starts when it has ended.  The chains have nothing of
torch between their calls: each reads what an early releasing kernel is still writing, or writes what one is still reading, while the host
runs ahead behind a pause.  test_in_the_stream_s_order adds copies around a call and the reuse of its scratch by the next.  Results are bit
for bit those of the same calls with the device waited for after each."""
import random

import pytest
import torch

pytestmark = pytest.mark.gpu


def qid(name):
    from ipex_llm_b200.transformers.low_bit_linear import ggml_tensor_qtype
    return ggml_tensor_qtype[name]


def matmul(dev, g, rows, qtype, dtype, n=2048, k=2048):
    from ipex_llm_b200.transformers import low_bit_linear as lbl
    ws = [lbl.FP4Params(torch.randn(n, k, generator=g, device=dev) * 0.02, qtype=qid(qtype)).to(dev).data for _ in range(2)]
    xs = [torch.randn(rows, k, generator=g, device=dev).to(dtype) for _ in range(2)]
    return [ws, xs], lambda w, x: lbl.lowbit_matmul(x, w, (n, k), qid(qtype))


def mlp(dev, g, rows, qtype, dtype, h=1024, i=2048):
    from ipex_llm_b200.transformers import low_bit_linear as lbl
    def one(n, k): return [lbl.FP4Params(torch.randn(n, k, generator=g, device=dev) * 0.02, qtype=qid(qtype)).to(dev).data for _ in range(2)]       # noqa: E704
    return [one(i, h), one(i, h), [torch.randn(rows, h, generator=g, device=dev).to(dtype) for _ in range(2)]], \
        lambda gate, up, x: lbl.mlp_forward(x, gate, up, rows, h, i, lbl.SILU, qid(qtype))


def grad(dev, g, rows, qtype, dtype, n=2048, k=1024):
    from ipex_llm_b200.transformers import low_bit_linear as lbl
    w = lbl.FP4Params(torch.randn(n, k, generator=g, device=dev) * 0.02, qtype=qid(qtype)).to(dev)
    xs = [torch.randn(rows, k, generator=g, device=dev).to(dtype) for _ in range(2)]
    gs = [torch.randn(rows, n, generator=g, device=dev).to(dtype) for _ in range(2)]

    def call(x, go):
        x = x.detach().requires_grad_(True)
        return torch.autograd.grad(lbl.MatMulLowBit.apply(x, w, n), x, go)[0]
    return [xs, gs], call


def attention(dev, g, batch, new, held, dtype):
    from ipex_llm_b200.transformers import kv
    q = [torch.randn(batch, 8, new, 128, generator=g, device=dev).to(dtype) for _ in range(2)]
    cache = [[torch.randn(batch, 2, new + held, 128, generator=g, device=dev).to(torch.float8_e5m2).view(torch.uint8) for _ in range(2)] for _ in range(2)]
    return [q, *cache], lambda q, k, v: kv.scaled_dot_product_attention(q, k, v, None, new > 1, 128 ** -0.5)


def delta(dev, g, tokens, dtype):
    from ipex_llm_b200.transformers.models import mixer_ops as ops
    G, H, D, V = 2, 4, 128, 64
    conv = [torch.randn(1, tokens, 2 * G * D + H * V, generator=g, device=dev).to(dtype) for _ in range(2)]
    proj = [torch.randn(1, tokens, 2 * H, generator=g, device=dev).to(dtype) for _ in range(2)]
    a_log, bias = torch.randn(H, generator=g, device=dev).to(dtype), torch.randn(H, generator=g, device=dev).to(dtype)
    states = [torch.randn(1, H, D, V, generator=g, device=dev) for _ in range(2)]
    pad = torch.zeros(1, dtype=torch.int32, device=dev)

    def call(conv, proj, state):
        o = ops.gated_delta_rule(conv, G, H, D, V, proj, 0, H, a_log, bias, state, 0, pad)
        return torch.cat([o.flatten(), state.flatten()])
    return [conv, proj, states], call


CALLS = {
    "row": lambda d, g: matmul(d, g, 1, "sym_int4", torch.float16), "rows_12": lambda d, g: matmul(d, g, 12, "fp8_e4m3", torch.bfloat16),
    "row_fp32": lambda d, g: matmul(d, g, 2, "nf4", torch.float32), "rows_40": lambda d, g: matmul(d, g, 40, "asym_int4", torch.float16),
    "prompt": lambda d, g: matmul(d, g, 300, "sym_int4", torch.bfloat16), "prompt_split": lambda d, g: matmul(d, g, 130, "fp6", torch.float16, 512, 8192),
    "prompt_fp32": lambda d, g: matmul(d, g, 100, "sym_int4", torch.float32), "mlp_3": lambda d, g: mlp(d, g, 3, "sym_int4", torch.float16),
    "mlp_30": lambda d, g: mlp(d, g, 30, "fp8_e5m2", torch.bfloat16), "mlp_300": lambda d, g: mlp(d, g, 300, "sym_int4", torch.float16),
    "gradient": lambda d, g: grad(d, g, 200, "sym_int4", torch.bfloat16), "decode_attention": lambda d, g: attention(d, g, 2, 1, 900, torch.float16),
    "prompt_attention": lambda d, g: attention(d, g, 1, 300, 0, torch.bfloat16), "delta_rule": lambda d, g: delta(d, g, 200, torch.bfloat16),
}


@pytest.mark.parametrize("side_stream", [False, True])
@pytest.mark.parametrize("name", list(CALLS))
def test_in_the_stream_s_order(cuda_device, name, side_stream):
    g = torch.Generator(device=cuda_device).manual_seed(7)
    pairs, call = CALLS[name](cuda_device, g)
    stream = torch.cuda.Stream() if side_stream else torch.cuda.current_stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        want = []
        for i in range(2):
            inputs = [p[i].clone() for p in pairs]
            torch.cuda.synchronize()
            want.append(call(*inputs).clone())
            torch.cuda.synchronize()
        assert not torch.equal(want[0], want[1])
        inputs, got = [p[0].clone() for p in pairs], []
        for i in range(12):
            torch.cuda._sleep(100000)
            for t, p in zip(inputs, pairs):
                t.copy_(p[i % 2])
            y = call(*inputs)
            again = call(*inputs) if name != "delta_rule" else None              # (the state has moved on)
            for t in inputs:
                t.zero_()
            got.append((y.clone(), again))
        torch.cuda.synchronize()
    for i, (y, again) in enumerate(got):
        assert torch.equal(y, want[i % 2]) and (again is None or torch.equal(again, want[i % 2])), i


def test_captured_calls_replay(cuda_device):
    g = torch.Generator(device=cuda_device).manual_seed(8)
    for name in ("rows_12", "rows_40", "prompt", "decode_attention", "prompt_attention"):
        pairs, call = CALLS[name](cuda_device, g)
        inputs = [p[0].clone() for p in pairs]
        want = [call(*[p[i] for p in pairs]).clone() for i in range(2)]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = call(*inputs)
            z = call(*inputs)
        for i in range(4):
            for t, p in zip(inputs, pairs):
                t.copy_(p[i % 2])
            graph.replay()
            assert torch.equal(y, want[i % 2]) and torch.equal(z, want[i % 2])


def packed(dev, g, n, k, qtype):
    from ipex_llm_b200.transformers import low_bit_linear as lbl
    return lbl.FP4Params(torch.randn(n, k, generator=g, device=dev) * k ** -0.5, qtype=qid(qtype)).to(dev).data


@pytest.mark.parametrize("rows,qtype,dtype", [(1, "sym_int4", torch.float16), (1, "nf4", torch.float32), (12, "fp8_e4m3", torch.bfloat16), (17, "fp6", torch.float16),
                                              (40, "asym_int4", torch.float16), (64, "nf4", torch.bfloat16), (33, "nf4", torch.float32), (100, "sym_int4", torch.float32),
                                              (100, "asym_int4", torch.float32), (130, "fp8_e5m2", torch.float16), (300, "sym_int4", torch.bfloat16), (1100, "fp6", torch.float16)])
@pytest.mark.parametrize("n", [1024, 2048])
def test_a_chain_of_matmuls_in_two_buffers(cuda_device, rows, qtype, dtype, n):
    """each call reads what the last one wrote, and writes over what that one read"""
    from ipex_llm_b200.transformers import low_bit_linear as lbl
    g = torch.Generator(device=cuda_device).manual_seed(rows)
    ws = [packed(cuda_device, g, n, n, qtype) for _ in range(3)]
    x = torch.randn(rows, n, generator=g, device=cuda_device).to(dtype)
    finals = []
    for waits in (True, False, False, False):
        pair = [x.clone(), torch.zeros_like(x)]
        torch.cuda._sleep(1000000)
        for i in range(16):
            lbl.lowbit_matmul(pair[i % 2], ws[i % 3], (n, n), qid(qtype), out=pair[(i + 1) % 2])
            if waits:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        finals.append([t.clone() for t in pair])
    assert float(finals[0][0].abs().max()) > 1e-3
    assert all(torch.equal(a, b) for f in finals[1:] for a, b in zip(f, finals[0]))


def links(dev, g):
    """name -> a call of several launches from the rows of one buffer to those of another, [300, 1024] fp16 both"""
    from ipex_llm_b200.transformers import kv, low_bit_linear as lbl
    from ipex_llm_b200.transformers.models import mixer_ops as ops
    W = 1024
    square = {q: packed(dev, g, W, W, q) for q in ("sym_int4", "asym_int4", "nf4", "fp8_e4m3", "fp6")}
    up, gate, down = packed(dev, g, 2048, W, "sym_int4"), packed(dev, g, 2048, W, "sym_int4"), packed(dev, g, W, 2048, "sym_int4")
    state, narrow = torch.randn(1, 4, 128, 128, generator=g, device=dev), packed(dev, g, W, 512, "asym_int4")
    a_log, bias = torch.randn(4, generator=g, device=dev).half(), torch.randn(4, generator=g, device=dev).half()
    proj, pad = torch.randn(1, 300, 8, generator=g, device=dev).half(), torch.zeros(1, dtype=torch.int32, device=dev)
    keys, values = (torch.randn(2, 2, 900, 128, generator=g, device=dev).to(torch.float8_e5m2).view(torch.uint8) for _ in range(2))
    ids, weight = torch.randint(0, 3, (300, 2), generator=g, device=dev), torch.rand(300, 2, generator=g, device=dev).half()
    tables = [torch.full((3,), t.data_ptr(), dtype=torch.int64, device=dev) for t in (gate, up, down)]
    kept = (gate, up, down)

    def matmul(rows, q):
        return lambda x, y: [lbl.lowbit_matmul(x[:rows], square[q], (W, W), qid(q), out=y[:rows])]

    def mlp(rows):
        def call(x, y):
            h = lbl.mlp_forward(x[:rows], gate, up, rows, W, 2048, lbl.SILU, qid("sym_int4"))
            return [lbl.lowbit_matmul(h, down, (W, 2048), qid("sym_int4"), out=y[:rows])]
        return call

    def decode(x, y):
        o = kv.scaled_dot_product_attention(x[:2].view(2, 8, 1, 128), keys, values, None, False, 128 ** -0.5)
        return [lbl.lowbit_matmul(o.transpose(1, 2).reshape(2, W), square["sym_int4"], (W, W), qid("sym_int4"), out=y[:2])]

    def prompt(x, y):
        o = kv.sdp_fp8_prefill(x.view(1, 300, 8, 128).transpose(1, 2), keys[:1], values[:1], None, 128 ** -0.5, True)
        return [lbl.lowbit_matmul(o.transpose(1, 2).view(300, W), square["fp6"], (W, W), qid("fp6"), out=y)]

    def prompt_to_40(x, y):                       # a kernel that takes tensor memory behind one that lets it start early
        o = kv.sdp_fp8_prefill(x.view(1, 300, 8, 128).transpose(1, 2), keys[:1], values[:1], None, 128 ** -0.5, True)
        return [lbl.lowbit_matmul(o.transpose(1, 2).view(300, W)[:40], square["asym_int4"], (W, W), qid("asym_int4"), out=y[:40])]

    def recurrence(x, y):                         # 32-bit outputs into a 32-bit prompt, twice
        s = state.clone()
        o = ops.gated_delta_rule(x.view(1, 300, W), 2, 4, 128, 128, proj, 0, 4, a_log, bias, s, 0, pad)
        h = lbl.lowbit_matmul(o.view(300, 512), narrow, (W, 512), qid("asym_int4"))
        return [s, lbl.lowbit_matmul(h, square["nf4"], (W, W), qid("nf4")), lbl.lowbit_matmul(x, square["sym_int4"], (W, W), qid("sym_int4"), out=y)]

    def gradient(x, y):
        return [lbl.lowbit_matmul(lbl.lowbit_matmul_grad(x[:200], square["sym_int4"], (W, W), qid("sym_int4")), square["fp8_e4m3"], (W, W), qid("fp8_e4m3"), out=y[:200])]

    def experts(x, y, kept=kept):
        return [lbl.lowbit_matmul(lbl.moe_forward_tokens(x, ids, weight, *tables, W, 2048, qid("sym_int4")), square["sym_int4"], (W, W), qid("sym_int4"), out=y)]

    return {"row": matmul(1, "sym_int4"), "rows 12": matmul(12, "fp8_e4m3"), "rows 40": matmul(40, "asym_int4"), "rows 60": matmul(60, "nf4"),
            "prompt 130": matmul(130, "fp6"), "prompt 300": matmul(300, "sym_int4"), "mlp 3": mlp(3), "mlp 30": mlp(30), "mlp 300": mlp(300),
            "decode attention": decode, "prompt attention": prompt, "prompt attention, 40 rows": prompt_to_40, "recurrence": recurrence, "gradient": gradient,
            "experts": experts}


@pytest.mark.parametrize("seed", range(12))
def test_a_chain_of_different_calls(cuda_device, seed):
    """every kind of call behind every other, in several orders"""
    g = torch.Generator(device=cuda_device).manual_seed(11)
    calls = links(cuda_device, g)
    x = torch.randn(300, 1024, generator=g, device=cuda_device).half()
    names = list(calls)
    random.Random(seed).shuffle(names)
    runs = []
    for waits in (True, False, False):
        pair, out = [x.clone(), x.clone()], []
        torch.cuda._sleep(4000000)
        for i, name in enumerate(names + names):
            for t in calls[name](pair[i % 2], pair[(i + 1) % 2])[:-1]:
                out.append(t)
            if waits:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        runs.append(out + pair)
    assert all(bool(t.isfinite().all()) for t in runs[0]) and float(runs[0][-1].float().std()) > 1e-4
    assert all(torch.equal(a, b) for r in runs[1:] for a, b in zip(r, runs[0])), names


@pytest.mark.parametrize("rows,qtype,dtype", [(1, "sym_int4", torch.float16), (12, "fp8_e4m3", torch.bfloat16), (40, "asym_int4", torch.float16),
                                              (100, "sym_int4", torch.float32), (100, "asym_int4", torch.float32), (300, "fp6", torch.float16)])
def test_weights_that_are_written_two_launches_ahead(cuda_device, rows, qtype, dtype):
    """a copy writes the weights, an early releasing kernel stands between it and the call that reads them"""
    from ipex_llm_b200.transformers import kv, low_bit_linear as lbl
    g = torch.Generator(device=cuda_device).manual_seed(5)
    ws = [packed(cuda_device, g, 2048, 1024, qtype) for _ in range(2)]
    x = torch.randn(rows, 1024, generator=g, device=cuda_device).to(dtype)
    q = torch.randn(1, 8, 40, 128, generator=g, device=cuda_device).half()
    k, v = (torch.randn(1, 2, 40, 128, generator=g, device=cuda_device).to(torch.float8_e5m2).view(torch.uint8) for _ in range(2))
    want = [lbl.lowbit_matmul(x, w, (2048, 1024), qid(qtype)) for w in ws]
    w, got = ws[0].clone(), []
    torch.cuda.synchronize()
    torch.cuda._sleep(1000000)
    for i in range(12):
        w.copy_(ws[i % 2])
        kv.sdp_fp8_prefill(q, k, v, None, 0.1, True)
        got.append(lbl.lowbit_matmul(x, w, (2048, 1024), qid(qtype)))
    torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1]) and all(torch.equal(y, want[i % 2]) for i, y in enumerate(got))


@pytest.mark.parametrize("rows,qtype,dtype", [(1, "sym_int4", torch.float16), (12, "fp8_e4m3", torch.bfloat16), (40, "asym_int4", torch.float16),
                                              (100, "sym_int4", torch.float32), (300, "fp6", torch.float16)])
@pytest.mark.parametrize("writer", [1, 40, 300])
def test_weights_that_the_launch_in_front_writes(cuda_device, rows, qtype, dtype, writer):
    """a matmul's results, whatever numbers they are as codes and scales, are the next one's packed weights"""
    from ipex_llm_b200.transformers import low_bit_linear as lbl
    g = torch.Generator(device=cuda_device).manual_seed(6)
    size = packed(cuda_device, g, 1024, 1024, qtype).numel()
    wide = -(-size // (2 * writer * 128)) * 128
    makers = [packed(cuda_device, g, wide, 256, "fp8_e4m3") for _ in range(2)]
    source, x = torch.randn(writer, 256, generator=g, device=cuda_device).half(), torch.randn(rows, 1024, generator=g, device=cuda_device).to(dtype)
    runs = []
    for waits in (True, False, False):
        held, out = torch.zeros(writer, wide, dtype=torch.float16, device=cuda_device), []
        torch.cuda.synchronize()
        torch.cuda._sleep(1000000)
        for i in range(12):
            lbl.lowbit_matmul(source, makers[i % 2], (wide, 256), qid("fp8_e4m3"), out=held)
            if waits:
                torch.cuda.synchronize()
            out.append(lbl.lowbit_matmul(x, held.view(-1).view(torch.uint8)[:size], (1024, 1024), qid(qtype)))
            if waits:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        runs.append([t.view(torch.uint8) for t in out])
    assert not torch.equal(runs[0][0], runs[0][1])
    assert all(torch.equal(a, b) for r in runs[1:] for a, b in zip(r, runs[0]))
