"""Launches that overlap their starts keep the stream's order: what the kernel in front writes is read, weights too, and what stands
behind may overwrite the inputs at once.

Every call stands between a copy that brings its inputs (behind a pause, so that the call is scheduled long before them) and copies that
overwrite them; the result is bit for bit that of the same call with the device waited for around it."""
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
