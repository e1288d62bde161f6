"""The bounded waits of the prompt kernels (csrc/tc_common.cuh): one that runs out ends its kernel, which first waits for the copies and
MMAs that it has under way; the next call reports it, and the one after is right."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def limit(native_lib, cuda_device):
    """sets the limit, in SM clocks, of this thread's launches; below zero half of a launch's copies never come, and the waits for them run out"""
    yield native_lib._lib.lowbit_debug_set_wait_limit
    native_lib._lib.lowbit_debug_set_wait_limit(0)


def rows(dev, m, k, dtype):
    return torch.randn(m, k, generator=torch.Generator(device=dev).manual_seed(m), device=dev).to(dtype)


def packed(lbl, dev, n, k, qtype="sym_int4", seed=0):
    w = torch.randn(n, k, generator=torch.Generator(device=dev).manual_seed(seed), device=dev) * 0.02
    return lbl.FP4Params(w, qtype=lbl.ggml_tensor_qtype[qtype]).to(dev).data


def calls(lbl, kv, dev):
    w, u, down = packed(lbl, dev, 2048, 4096), packed(lbl, dev, 2048, 4096, seed=1), packed(lbl, dev, 256, 384, seed=2)
    nf4, big = packed(lbl, dev, 384, 1024, "nf4"), packed(lbl, dev, 4096, 1024)
    gate, up = packed(lbl, dev, 384, 256, seed=3), packed(lbl, dev, 384, 256, seed=4)
    x16, x32, xb = rows(dev, 100, 4096, torch.float16), rows(dev, 100, 4096, torch.float32), rows(dev, 700, 1024, torch.bfloat16)
    table = lambda t: torch.full((2,), t.data_ptr(), dtype=torch.int64, device=dev)                                 # noqa: E731
    ids, weight, xe = torch.arange(600, device=dev).view(300, 2) % 2, torch.full((300, 2), 0.5, device=dev), rows(dev, 300, 256, torch.float16)
    tables = [table(t) for t in (gate, up, down)]
    q = rows(dev, 4 * 400, 128, torch.float16).view(1, 400, 4, 128).transpose(1, 2)
    k, v = (rows(dev, 400 + i, 128, torch.float32).to(torch.float8_e5m2).view(torch.uint8)[None, None, :400].expand(1, 4, 400, 128).contiguous()
            for i in range(2))
    wide = q.expand(40, 4, 400, 128)
    wide_k, wide_v = (t.expand(40, 4, 400, 128) for t in (k, v))
    return {"split matmul": lambda: lbl.lowbit_matmul(x16, w, (2048, 4096), lbl.SYM_INT4),
            "matmul of many tiles": lambda: lbl.lowbit_matmul(xb, big, (4096, 1024), lbl.SYM_INT4),
            "matmul through a table": lambda: lbl.lowbit_matmul(xb, nf4, (384, 1024), lbl.NF4),
            "mlp": lambda: lbl.mlp_forward(x16, w, u, 100, 4096, 2048, lbl.SILU, lbl.SYM_INT4),
            "experts": lambda held=(gate, up, down): lbl.moe_forward_tokens(xe, ids, weight, *tables, 256, 384, lbl.SYM_INT4),
            "fp32 matmul": lambda: lbl.lowbit_matmul(x32, w, (2048, 4096), lbl.SYM_INT4),
            "attention": lambda: kv.sdp_fp8_prefill(q, k, v, None, 0.1, True),
            "attention of many rows": lambda: kv.sdp_fp8_prefill(wide, wide_k, wide_v, None, 0.1, False)}


@pytest.mark.parametrize("clocks", [20, 100000])
@pytest.mark.parametrize("name", ["split matmul", "matmul of many tiles", "matmul through a table", "mlp", "experts", "fp32 matmul", "attention",
                                  "attention of many rows"])
def test_a_wait_that_runs_out_is_reported_once(native_lib, cuda_device, limit, name, clocks):
    from ipex_llm_b200.transformers import kv, low_bit_linear as lbl
    call = calls(lbl, kv, cuda_device)[name]
    want = call()
    assert not native_lib.lowbit_gemm_wait_expired()
    limit(-clocks)
    reported = False
    try:
        call()
    except native_lib.LowBitNativeError as e:                 # its own second launch may already see it
        assert "ran out" in str(e)
        reported = True
    limit(0)
    if native_lib.lowbit_gemm_wait_expired():
        with pytest.raises(native_lib.LowBitNativeError, match="ran out"):
            call()
        reported = True
    assert reported
    assert not native_lib.lowbit_gemm_wait_expired()
    assert torch.equal(call(), want)


@pytest.mark.parametrize("clocks", [1, 300, 1500, 6000, 30000])
@pytest.mark.parametrize("name", ["split matmul", "matmul of many tiles", "experts", "fp32 matmul", "attention of many rows"])
def test_wherever_a_wait_runs_out_the_next_call_is_right(native_lib, cuda_device, limit, name, clocks):
    """limits of the order of the kernels' own waits: they run out in the middle of the work, or not at all"""
    from ipex_llm_b200.transformers import kv, low_bit_linear as lbl
    call = calls(lbl, kv, cuda_device)[name]
    want = call()
    for _ in range(5):
        limit(clocks)
        try:
            call()
        except native_lib.LowBitNativeError as e:
            assert "ran out" in str(e)
        limit(0)
        if native_lib.lowbit_gemm_wait_expired():
            with pytest.raises(native_lib.LowBitNativeError, match="ran out"):
                call()
            torch.cuda.synchronize()
        assert torch.equal(call(), want)


@pytest.fixture
def delta_limit(cuda_device):
    """sets the limit of this thread's delta-rule launches; below zero only a block's first chunk comes"""
    from ipex_llm_b200.ggml.model import mixers_cpp
    yield mixers_cpp.lib().mixers_debug_set_wait_limit
    mixers_cpp.lib().mixers_debug_set_wait_limit(0)


def delta_call(dev, dtype, dim, tokens=300):
    from ipex_llm_b200.transformers.models import mixer_ops as ops
    B, G, H, V = 2, 2, 4, 40
    conv, proj = rows(dev, B * tokens, 2 * G * dim + H * V, dtype).view(B, tokens, -1), rows(dev, B * tokens, 2 * H, dtype).view(B, tokens, -1)
    a_log, bias, state = rows(dev, 1, H, dtype)[0], rows(dev, 2, H, dtype)[0], rows(dev, B * H * dim, V, torch.float32).view(B, H, dim, V)
    pad = torch.tensor([0, 50], dtype=torch.int32, device=dev)

    def call():
        s = state.clone()
        o = ops.gated_delta_rule(conv, G, H, dim, V, proj, 0, H, a_log, bias, s, 0, pad)
        return torch.cat([o.flatten(), s.flatten()])
    return call


@pytest.mark.parametrize("clocks", [-20, -100000, 1, 300, 1500, 6000])
@pytest.mark.parametrize("dtype,dim", [(torch.float32, 128), (torch.bfloat16, 128), (torch.float16, 64)])       # two chunks in shared memory, and three
def test_a_delta_rule_wait_that_runs_out_is_reported_once(delta_limit, cuda_device, dtype, dim, clocks):
    """chunks that never come, and limits of the order of the kernel's own waits (which run out in the middle of the work, or not at all)"""
    from ipex_llm_b200.ggml.model import mixers_cpp
    call, expired = delta_call(cuda_device, dtype, dim), mixers_cpp.lib().mixers_wait_expired
    want = call()
    assert expired() == 0
    for _ in range(5):
        delta_limit(clocks)
        got = call()
        delta_limit(0)
        if expired():
            with pytest.raises(mixers_cpp.MixersNativeError, match="702"):
                call()
        else:
            assert clocks > 0 and torch.equal(got, want)
        assert expired() == 0 and torch.equal(call(), want)
