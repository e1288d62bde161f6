"""``LowBitExperts`` (transformers/models/mixtral.py): which route a call takes, and that each gives what the loop over the experts'
modules gives."""
import threading

import pytest
import torch

E, H, I = 4, 256, 384


class Fused(torch.nn.Module):
    """the layout a checkpoint's experts have before conversion"""

    def __init__(self, dev, seed=0, experts=E):
        super().__init__()
        g = torch.Generator(device=dev).manual_seed(seed)
        draw = lambda *s: torch.nn.Parameter(torch.empty(*s, device=dev).normal_(0.0, 0.05, generator=g), requires_grad=False)      # noqa: E731
        self.gate_up_proj, self.down_proj, self.act_fn = draw(experts, 2 * I, H), draw(experts, H, I), torch.nn.SiLU()


def layer(dev, qtype="sym_int4", seed=0, experts=E):
    from ipex_llm_b200.transformers.low_bit_linear import ggml_tensor_qtype
    from ipex_llm_b200.transformers.models.mixtral import LowBitExperts
    return LowBitExperts.from_fused(Fused(dev, seed, experts).eval(), ggml_tensor_qtype[qtype])


def plain_layer(seed=0, experts=E):
    """on the CPU, where the packed bytes are not needed: weights with addresses of their own"""
    from ipex_llm_b200.transformers.low_bit_linear import FP4Params, ggml_tensor_qtype
    from ipex_llm_b200.transformers.models.mixtral import LowBitExperts
    with torch.device("meta"):
        m = LowBitExperts(experts, H, I, ggml_tensor_qtype["sym_int4"], torch.nn.SiLU())
    for mods, (n, k) in ((m.gate_proj, (I, H)), (m.up_proj, (I, H)), (m.down_proj, (H, I))):
        for lin in mods:
            lin._parameters["weight"] = FP4Params(torch.zeros(n * k // 64 * 34, dtype=torch.uint8), quantized=True, _shape=(n, k), qtype=lin.qtype)
    return m.eval()


def replace(mods, e):
    """a re-quantised expert: other bytes at another address"""
    from ipex_llm_b200.transformers.low_bit_linear import FP4Params
    old = mods[e].weight
    mods[e]._parameters["weight"] = FP4Params(old.data.flip(0).contiguous() if old.data.device.type == "cpu" else old.data.clone(), quantized=True,
                                              _shape=old._shape, qtype=old.qtype)


@pytest.mark.parametrize("name", ["gate_proj", "up_proj", "down_proj"])
@pytest.mark.parametrize("e", range(E))
def test_the_address_tables_follow_every_expert(name, e):
    m = plain_layer()
    m._address_tables(torch.device("cpu"))
    replace(getattr(m, name), e)
    for table, mods in zip(m._address_tables(torch.device("cpu")), (m.gate_proj, m.up_proj, m.down_proj)):
        assert table.tolist() == [lin.weight.data_ptr() for lin in mods]


@pytest.mark.parametrize("part", ["gate_up", "down"])
@pytest.mark.parametrize("e", range(3))
def test_the_address_tables_of_plain_matrices_follow_every_expert(part, e):
    from ipex_llm_b200.transformers.models import experts

    class One(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.gate_up, self.down, self.ff = torch.nn.Linear(16, 16, bias=False), torch.nn.Linear(8, 16, bias=False), 8
    mlp = torch.nn.Module()
    mlp.experts, mlp.shared, mlp._tables, cpu = torch.nn.ModuleList([One() for _ in range(3)]), None, None, torch.device("cpu")
    experts.address_tables(mlp, torch.float32, cpu)
    held = getattr(mlp.experts[e], part).weight
    getattr(mlp.experts[e], part).weight = torch.nn.Parameter(held.detach().clone())
    first, down = experts.address_tables(mlp, torch.float32, cpu)[:2]
    assert first.tolist() == [x.gate_up.weight.data_ptr() for x in mlp.experts] and down.tolist() == [x.down.weight.data_ptr() for x in mlp.experts]


def routing(dev, rows, top_k=2, seed=1, experts=E):
    g = torch.Generator(device=dev).manual_seed(seed)
    w, idx = torch.softmax(torch.randn(rows, experts, generator=g, device=dev), -1).topk(top_k, dim=-1)
    return idx, w / w.sum(-1, keepdim=True)


def loop(m, x, idx, w):
    """the statement: every expert's modules over its rows, in 32 bits around them"""
    out = torch.zeros(x.shape, dtype=torch.float32, device=x.device)
    for e in range(m.num_experts):
        r, s = torch.where(idx == e)
        if len(r):
            a = torch.nn.functional.silu(m.gate_proj[e](x[r]).float()) * m.up_proj[e](x[r]).float()
            out.index_add_(0, r, m.down_proj[e](a.to(x.dtype)).float() * w[r, s, None].float())
    return out


# the loop rounds gate and up to the activation dtype (u each, the activation's slope below 1.13), the hidden row and the expert's
# output on both sides: fewer than eight roundings of u = 2^-11 / 2^-8 each, taken relative to the largest |output|
TOL = {torch.float16: 8 * 2.0 ** -11, torch.bfloat16: 8 * 2.0 ** -8}


def same(m, x, idx, w):
    got, want = m(x, idx, w).float(), loop(m, x, idx, w)
    assert float((got - want).abs().max()) <= TOL[x.dtype] * float(want.abs().max())
    return got


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 100])
def test_a_replaced_expert_is_the_one_that_runs(native_lib, cuda_device, rows):
    m, other = layer(cuda_device), layer(cuda_device, seed=5)
    x = torch.randn(rows, H, device=cuda_device).half()
    idx, w = routing(cuda_device, rows)
    idx[0, 0], idx[0, 1] = 2, 1
    before = same(m, x, idx, w)
    old = m.up_proj[2].weight                                                       # kept: its memory is not handed out again
    m.up_proj[2]._parameters["weight"] = other.up_proj[2].weight
    assert float((same(m, x, idx, w) - before)[0].abs().max()) > 0 and old is not m.up_proj[2].weight


class Wrapper(torch.nn.Module):
    """an expert that scales what a linear gives, and passes its attributes through"""

    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    def __getattr__(self, name):
        try:
            return super().__getattr__(name)
        except AttributeError:
            return getattr(super().__getattr__("inner"), name)

    def forward(self, x):
        return 2 * self.inner(x)


def odd_linear(lin):
    new = torch.nn.Linear(lin.in_len, lin.out_len, bias=False, dtype=torch.float16)
    return new.requires_grad_(False)


def hooked(lin):
    lin.register_forward_hook(lambda mod, args, out: 3 * out)
    return lin


def pre_hooked(lin):
    lin.register_forward_pre_hook(lambda mod, args: (0.5 * args[0],))
    return lin


def own_forward(lin):
    plain = lin.forward
    lin.forward = lambda x: -plain(x)
    return lin


def with_bias(lin):
    lin._parameters["bias"] = torch.nn.Parameter(torch.ones(lin.out_len, dtype=torch.float16, device=lin.weight.device), requires_grad=False)
    return lin


def subclass(lin):
    class Another(type(lin)):
        def forward(self, x):
            return 4 * super().forward(x)
    lin.__class__ = Another
    return lin


ODD = [odd_linear, Wrapper, hooked, pre_hooked, own_forward, with_bias, subclass]


@pytest.mark.parametrize("native", [True, False])
def test_only_plain_experts_are_read_by_their_addresses(monkeypatch, native):
    from ipex_llm_b200.transformers import low_bit_linear as lbl
    if not native:
        monkeypatch.setattr(lbl, "_host", False)
    cpu = torch.device("cpu")
    m = plain_layer()
    want = [lin.weight.data_ptr() for mods in (m.gate_proj, m.up_proj, m.down_proj) for lin in mods]
    assert torch.frombuffer(bytearray(m._plain_addresses(cpu)), dtype=torch.int64).tolist() == want and (not native or lbl._host)
    odd = list(ODD) + [lambda lin: setattr(lin, "qtype", lbl.NF4) or lin, lambda lin: setattr(lin, "act_order", True) or lin, lambda lin: lin.train(),
                       lambda lin: setattr(lin, "mp_group", object()) or lin, lambda lin: setattr(lin.weight, "quantized", False) or lin,
                       lambda lin: setattr(lin, "in_len", lin.in_len + 64) or lin, lambda lin: lin._parameters.pop("weight") is None or lin]
    for i, change in enumerate(odd):
        m = plain_layer()
        mods = (m.gate_proj, m.up_proj, m.down_proj)[i % 3]
        mods[i % E] = change(mods[i % E])
        assert m._plain_addresses(cpu) is None, i
    m = plain_layer()
    m.up_proj = m.up_proj[:3]
    assert m._plain_addresses(cpu) is None
    hook = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    try:
        assert plain_layer()._plain_addresses(cpu) is None
    finally:
        hook.remove()


@pytest.mark.gpu
@pytest.mark.parametrize("change", ODD)
@pytest.mark.parametrize("name,e", [("gate_proj", 0), ("up_proj", 2), ("down_proj", 3)])
def test_an_expert_that_is_not_plain_runs_itself(native_lib, cuda_device, change, name, e):
    m = layer(cuda_device)
    mods = getattr(m, name)
    mods[e] = change(mods[e]).to(cuda_device)
    x = torch.randn(90, H, device=cuda_device).half()
    idx, w = routing(cuda_device, 90)
    idx[:, 0] = torch.where(idx[:, 1] == e, (e + 1) % E, e)
    same(m, x, idx, w)


@pytest.mark.gpu
def test_an_expert_of_another_format_runs_itself(native_lib, cuda_device):
    m = layer(cuda_device)
    m.up_proj[1] = layer(cuda_device, "fp8_e4m3", seed=7).up_proj[1]
    same(m, torch.randn(90, H, device=cuda_device).half(), *routing(cuda_device, 90))


@pytest.mark.gpu
@pytest.mark.parametrize("qtype", ["sym_int4", "asym_int4", "nf4", "fp8_e4m3", "fp8_e5m2", "fp6"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows", [(0, 1, 8, 9, 16, 17, 300, 2), (3, 16, 0, 0, 1, 5, 0, 7), (17, 33, 64, 65, 256, 257, 40, 18)])
def test_few_rows_keep_exact_weights(native_lib, cuda_device, qtype, dtype, rows):
    """up to 16 rows an expert's products are the GEMV's, bit for bit: weights as code x scale, not rounded to the activation dtype"""
    from ipex_llm_b200.transformers import low_bit_linear as lbl
    m = layer(cuda_device, qtype, experts=len(rows))
    idx = torch.cat([torch.full((n, 1), e, device=cuda_device) for e, n in enumerate(rows)])
    idx = idx[torch.randperm(len(idx), device=cuda_device)]
    x = torch.randn(len(idx), H, device=cuda_device).to(dtype)
    got = same(m, x, idx, torch.ones(len(idx), 1, device=cuda_device))
    for e, n in enumerate(rows):
        if 1 <= n <= 16:
            r = torch.where(idx[:, 0] == e)[0]
            h = lbl.mlp_forward(x[r], m.gate_proj[e].weight.data, m.up_proj[e].weight.data, n, H, I, lbl.SILU, m.qtype)
            assert torch.equal(got[r].to(dtype), lbl.lowbit_matmul(h, m.down_proj[e].weight.data, (H, I), m.qtype))


@pytest.mark.gpu
def test_few_rows_from_several_threads_and_streams(native_lib, cuda_device):
    """the row counts that the host waits for are each call's own"""
    m = layer(cuda_device, experts=8)
    calls = [(torch.randn(rows, H, device=cuda_device).half(), *routing(cuda_device, rows, seed=rows, experts=8)) for rows in (5, 40, 90, 200)]
    want = [m(*c) for c in calls]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        with torch.no_grad(), torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                if not torch.equal(m(*calls[i]), want[i]):
                    wrong.append(i)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [5, 200])
@pytest.mark.parametrize("bad", [-1, E, 1 << 40])
def test_a_choice_outside_the_layer_is_an_error(native_lib, cuda_device, rows, bad):
    m = layer(cuda_device)
    x = torch.randn(rows, H, device=cuda_device).half()
    idx, w = routing(cuda_device, rows)
    wrong = idx.clone()
    wrong[rows // 2, 1] = bad
    with pytest.raises(RuntimeError, match="outside"):
        m(x, wrong, w)
    same(m, x, idx, w)                                                              # and the next call is none the worse


@pytest.mark.gpu
@pytest.mark.parametrize("rows,limit", [(700, 1 << 20), (333, 100000), (3, 1), (4097, 4 << 20)])
def test_long_prompts_run_in_portions(native_lib, cuda_device, monkeypatch, rows, limit):
    """scratch stays below its bound (or at one token's), whatever the prompt's length"""
    from ipex_llm_b200.transformers import low_bit_linear as lbl
    m = layer(cuda_device)
    x = torch.randn(rows, H, device=cuda_device).half()
    idx, w = routing(cuda_device, rows)
    monkeypatch.setattr(lbl, "MOE_MAX_SCRATCH", limit)
    m(x, idx, w)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    got = m(x, idx, w)
    one = native_lib.lowbit_moe_tokens_workspace_size(H, I, E, 1, 2)
    # a portion holds whole tokens, and every piece of it is rounded up to 256 bytes
    assert torch.cuda.max_memory_allocated() - before <= got.numel() * 2 + max(limit, one) + one + 4096
    same(m, x, idx, w)
    with pytest.raises(RuntimeError, match="outside"):
        m(x, torch.where(torch.arange(rows, device=cuda_device)[:, None] == 0, E, idx), w)


def test_the_kernels_take_one_device_and_the_loops_types_only(native_lib, monkeypatch):
    """an address of another device's memory would be read there; what the loop refuses, or serves in its own way, stays with it"""
    from ipex_llm_b200.transformers import low_bit_linear as lbl
    from ipex_llm_b200.transformers.models import mixtral
    m = plain_layer()
    monkeypatch.setattr(mixtral, "moe_tokens_supported", lambda *a: True)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    x, idx, w = torch.zeros(6, H, dtype=torch.float16), torch.zeros(6, 2, dtype=torch.int64), torch.zeros(6, 2)
    with torch.no_grad():
        assert m._many_tokens_ok(x, idx, w)
        for args in ((x, idx.to("meta"), w), (x, idx, w.to("meta")), (x.to("meta"), idx, w), (x, idx.int(), w), (x, idx[:5], w[:5]), (x, idx, w[:, :1]),
                     (x, idx, w.double())):
            assert not m._many_tokens_ok(*args)
    tables = [torch.zeros(E, dtype=torch.int64)] * 3
    with pytest.raises(RuntimeError, match="device"):
        lbl.moe_forward_tokens(x, idx, w, *tables, H, I, m.qtype)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 70])
def test_routing_on_the_host_is_refused(native_lib, cuda_device, rows):
    m = layer(cuda_device)
    x = torch.randn(rows, H, device=cuda_device).half()
    idx, w = routing(cuda_device, rows)
    for args in ((x, idx.cpu(), w), (x, idx, w.cpu()), (torch.cat([x, x]), torch.cat([idx, idx]).int(), torch.cat([w, w]))):
        with pytest.raises(RuntimeError):
            m(*args)
    part = m(torch.cat([x, x]), idx, w)                                             # rows without a choice come out zero
    assert not bool(part[rows:].any())
    same(m, x, idx, w)
