"""The gated delta rule 32 tokens at a time (csrc/mixers/delta_chunks.cu) against float64 and against the token-by-token kernel.

Bound: all arithmetic is 32-bit; a token's value passes through a handful of dot products of up to 128 terms and its chunk's
triangular system, whose entries are at most 1 for unit keys, so 2e-6 of the largest |value| leaves a factor of about ten over what
sums of that length show."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from ipex_llm_b200.transformers.models import mixer_ops
    return mixer_ops


def inputs(dev, B, S, G, H, D, V, dtype, seed=0, gate_std=1.0):
    g = torch.Generator(device=dev).manual_seed(seed + S)
    conv = torch.randn(B, S, 2 * G * D + H * V, generator=g, device=dev).to(dtype)
    proj = (torch.randn(B, S, 2 * H + 3, generator=g, device=dev) * gate_std).to(dtype)
    a_log, bias = (torch.randn(H, generator=g, device=dev) * 0.5 - 1).to(dtype), (torch.randn(H, generator=g, device=dev) * 0.5).to(dtype)
    state = torch.randn(B, H, D, V, generator=g, device=dev)
    return conv, proj, a_log, bias, state


def statement(conv, proj, a_log, bias, state, G, H, D, V, slot0, pad):
    B, S, _ = conv.shape
    c, p = conv.double(), proj.double()
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)                                       # noqa: E731
    q = (unit(c[..., :G * D].view(B, S, G, D)) * D ** -0.5).repeat_interleave(H // G, 2)
    k = unit(c[..., G * D:2 * G * D].view(B, S, G, D)).repeat_interleave(H // G, 2)
    v = c[..., 2 * G * D:].view(B, S, H, V)
    beta = torch.sigmoid(p[..., 1:1 + H])
    decay = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(p[..., 1 + H:1 + 2 * H] + bias.double()))
    M, o = state.double().clone(), torch.zeros(B, S, H, V, dtype=torch.float64, device=conv.device)
    for t in range(S):
        real = (slot0 + t >= pad).view(B, 1, 1, 1)
        N = M * decay[:, t, :, None, None]
        u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhdv,bhd->bhv", N, k[:, t]))
        N = N + k[:, t, :, :, None] * u[:, :, None, :]
        M = torch.where(real, N, M)
        o[:, t] = torch.where(real[..., 0], torch.einsum("bhdv,bhd->bhv", N, q[:, t]), 0.0)
    return o, M


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,S,G,H,D,V,pads", [(1, 64, 1, 1, 128, 16, (0,)), (2, 65, 1, 2, 64, 17, (0, 40)), (1, 95, 2, 2, 5, 9, (3,)), (3, 127, 1, 3, 70, 33, (0, 127, 64)),
                                              (1, 200, 2, 32, 128, 128, (0,)), (2, 96, 1, 1, 65, 256, (31, 33)), (1, 333, 4, 16, 128, 128, (0,))])
def test_against_float64_and_the_token_walk(ops, cuda_device, monkeypatch, dtype, B, S, G, H, D, V, pads):
    conv, proj, a_log, bias, state = inputs(cuda_device, B, S, G, H, D, V, dtype)
    pad = torch.tensor(pads, dtype=torch.int32, device=cuda_device)
    want_o, want_s = statement(conv, proj, a_log, bias, state, G, H, D, V, 0, pad)
    err = {}
    for route, least in (("chunks", 1), ("tokens", 1 << 30)):
        monkeypatch.setattr(ops, "DELTA_CHUNK_TOKENS", least)
        s = state.clone()
        o = ops.gated_delta_rule(conv, G, H, D, V, proj, 1, 1 + H, a_log, bias, s, 0, pad)
        assert float((o.double() - want_o).abs().max()) <= 2e-6 * max(1.0, float(want_o.abs().max()))
        assert float((s.double() - want_s).abs().max()) <= 2e-6 * max(1.0, float(want_s.abs().max()))
        err[route] = float((o.double() - want_o).norm() / want_o.norm())
    assert err["chunks"] <= 1.2 * err["tokens"] + 2.0 ** -24                       # as exact as the walk it replaces


def test_portions_and_hard_gates(ops, cuda_device):
    """a prompt in portions that end inside chunks; gates from 'forget all' to 'keep all' (decays that underflow, betas at 0 and 1)"""
    B, S, G, H, D, V = 2, 300, 1, 2, 128, 40
    conv, proj, a_log, bias, state = inputs(cuda_device, B, S, G, H, D, V, torch.float32, gate_std=40.0)
    a_log = a_log + 3.0                                                              # exp(-20 softplus): zero in 32 bits for half of the tokens
    proj[0, 70:75, 1 + H:1 + 2 * H] = 1e30
    pad = torch.tensor([0, 7], dtype=torch.int32, device=cuda_device)
    want_o, want_s = statement(conv, proj, a_log, bias, state, G, H, D, V, 0, pad)
    s, got, at = state.clone(), [], 0
    for n in (65, 100, 1, 134):
        got.append(ops.gated_delta_rule(conv[:, at:at + n].contiguous(), G, H, D, V, proj[:, at:at + n].contiguous(), 1, 1 + H, a_log, bias, s, at, pad))
        at += n
    assert float((torch.cat(got, 1).double() - want_o).abs().max()) <= 2e-6 * float(want_o.abs().max())
    assert float((s.double() - want_s).abs().max()) <= 2e-6 * float(want_s.abs().max())


def test_equal_keys(ops, cuda_device):
    """every key the same: the triangular system at its worst"""
    B, S, G, H, D, V = 1, 160, 1, 1, 64, 16
    conv, proj, a_log, bias, state = inputs(cuda_device, B, S, G, H, D, V, torch.float32)
    conv[..., D:2 * D] = conv[:, :1, D:2 * D]
    a_log = a_log - 9.0                                                              # hardly any decay
    pad = torch.zeros(B, dtype=torch.int32, device=cuda_device)
    want_o, want_s = statement(conv, proj, a_log, bias, state, G, H, D, V, 0, pad)
    o = ops.gated_delta_rule(conv, G, H, D, V, proj, 1, 1 + H, a_log, bias, state, 0, pad)
    assert float((o.double() - want_o).abs().max()) <= 2e-6 * float(want_o.abs().max())
    assert float((state.double() - want_s).abs().max()) <= 2e-6 * float(want_s.abs().max())


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_token_that_is_not_finite_stays_behind_the_earlier_ones(ops, cuda_device, bad):
    """values at token 77, in the middle of a chunk: the tokens before it come out as without it"""
    B, S, G, H, D, V = 1, 130, 1, 1, 128, 32
    conv, proj, a_log, bias, state = inputs(cuda_device, B, S, G, H, D, V, torch.float32)
    pad = torch.zeros(B, dtype=torch.int32, device=cuda_device)
    o = ops.gated_delta_rule(conv, G, H, D, V, proj, 1, 1 + H, a_log, bias, state.clone(), 0, pad)
    conv[0, 77, 2 * G * D + 3] = bad                                                 # one value column
    got = ops.gated_delta_rule(conv, G, H, D, V, proj, 1, 1 + H, a_log, bias, state.clone(), 0, pad)
    assert torch.equal(got[:, :77], o[:, :77]) and not bool(got[:, 77:, :, 3].isfinite().any())
    assert torch.equal(got[..., :3], o[..., :3]) and torch.equal(got[..., 4:], o[..., 4:])


def test_a_prompt_in_portions_of_its_scratch(ops, cuda_device):
    """one chunk of these heads takes 304 MB, so that the four chunks run one by one; padding ends in each of them"""
    B, S, G, H, D, V = 64, 100, 128, 128, 5, 9
    conv, proj, a_log, bias, state = inputs(cuda_device, B, S, G, H, D, V, torch.float32)
    pad = torch.arange(B, dtype=torch.int32, device=cuda_device) * 100 // 63
    want_o, want_s = statement(conv, proj, a_log, bias, state, G, H, D, V, 0, pad)
    o = ops.gated_delta_rule(conv, G, H, D, V, proj, 1, 1 + H, a_log, bias, state, 0, pad)
    assert float((o.double() - want_o).abs().max()) <= 2e-6 * max(1.0, float(want_o.abs().max()))
    assert float((state.double() - want_s).abs().max()) <= 2e-6 * max(1.0, float(want_s.abs().max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bad", [float("nan"), float("-inf")])
@pytest.mark.parametrize("what", ["query", "key", "value"])
def test_nothing_of_a_later_token_reaches_an_earlier_one(ops, cuda_device, dtype, bad, what):
    """a query, a key, a value that is no number, as a chunk's first token and inside one: the tokens before it come out bit for bit as
    without it; a query stays with its own token, a key reaches every column behind it"""
    B, S, G, H, D, V = 1, 100, 1, 5, 128, 40
    conv, proj, a_log, bias, state = inputs(cuda_device, B, S, G, H, D, V, dtype)
    pad = torch.zeros(B, dtype=torch.int32, device=cuda_device)
    o = ops.gated_delta_rule(conv, G, H, D, V, proj, 1, 1 + H, a_log, bias, state.clone(), 0, pad)
    for at in (32, 45):
        c = conv.clone()
        c[0, at, {"query": 5, "key": D + 5, "value": 2 * D + 2 * V + 7}[what]] = bad
        got = ops.gated_delta_rule(c, G, H, D, V, proj, 1, 1 + H, a_log, bias, state.clone(), 0, pad)
        assert torch.equal(got[:, :at], o[:, :at])
        if what == "query":
            assert not bool(got[:, at].isfinite().any()) and torch.equal(got[:, at + 1:], o[:, at + 1:])
        elif what == "key":
            assert not bool(got[:, at:].isfinite().any())
        else:
            assert not bool(got[:, at:, 2, 7].isfinite().any())
            got[:, at:, 2, 7] = o[:, at:, 2, 7]
            assert torch.equal(got, o)


@pytest.mark.parametrize("dtype,power", [(torch.float32, 55), (torch.float32, -55), (torch.bfloat16, 40), (torch.bfloat16, -40), (torch.float16, -6), (torch.float16, 11)])
def test_keys_and_queries_of_any_size(ops, cuda_device, dtype, power):
    """the unit vectors' factors are powers of two and a rest: keys and queries far from one, and tokens without any"""
    B, S, G, H, D, V = 1, 96, 2, 2, 96, 24
    conv, proj, a_log, bias, state = inputs(cuda_device, B, S, G, H, D, V, dtype)
    conv[..., :2 * G * D] *= 2.0 ** power
    conv[:, 40, :2 * G * D] = 0
    pad = torch.zeros(B, dtype=torch.int32, device=cuda_device)
    want_o, want_s = statement(conv, proj, a_log, bias, state, G, H, D, V, 0, pad)
    o = ops.gated_delta_rule(conv, G, H, D, V, proj, 1, 1 + H, a_log, bias, state, 0, pad)
    assert float((o.double() - want_o).abs().max()) <= 2e-6 * max(1.0, float(want_o.abs().max()))
    assert float((state.double() - want_s).abs().max()) <= 2e-6 * max(1.0, float(want_s.abs().max()))


@pytest.mark.parametrize("dtype,value", [(torch.float32, torch.finfo(torch.float32).max), (torch.float32, torch.finfo(torch.float32).min), (torch.float32, 3.397e38),
                                         (torch.float32, 1.1e38), (torch.bfloat16, torch.finfo(torch.bfloat16).min), (torch.bfloat16, torch.finfo(torch.bfloat16).max)])
def test_the_largest_values_stay_behind_their_token(ops, cuda_device, dtype, value):
    """values of the size of a mask's lowest, whose first bf16 plane may be an infinity: the tokens before one and the other columns come out
    bit for bit as without it, the column behind it as float64 has it"""
    B, S, G, H, D, V = 1, 100, 1, 5, 128, 40
    conv, proj, a_log, bias, state = inputs(cuda_device, B, S, G, H, D, V, dtype)
    pad = torch.zeros(B, dtype=torch.int32, device=cuda_device)
    plain = state.clone()
    o = ops.gated_delta_rule(conv, G, H, D, V, proj, 1, 1 + H, a_log, bias, plain, 0, pad)
    for at in (32, 45):
        c, s = conv.clone(), state.clone()
        c[0, at, 2 * D + 2 * V + 7] = value
        got = ops.gated_delta_rule(c, G, H, D, V, proj, 1, 1 + H, a_log, bias, s, 0, pad)
        assert torch.equal(got[:, :at], o[:, :at])
        want_o, want_s = statement(c, proj, a_log, bias, state, G, H, D, V, 0, pad)
        for t, want, free in ((got[:, at:], want_o[:, at:], o[:, at:]), (s.movedim(2, 1), want_s.movedim(2, 1), plain.movedim(2, 1))):
            column, w = t[:, :, 2, 7].double(), want[:, :, 2, 7]
            assert float((column - w).abs().max()) <= 2e-6 * max(1.0, float(w.abs().max()))
            t, free = t.clone(), free.clone()
            t[:, :, 2, 7] = free[:, :, 2, 7] = 0
            assert torch.equal(t, free)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("at", [32, 63, 71])
def test_the_largest_values_enter_the_state(ops, cuda_device, dtype, at):
    """a gate that takes the largest value whole into the state, which forgets next to nothing: finite and right in the chunks behind it"""
    B, S, G, H, D, V = 1, 200, 2, 4, 96, 24
    conv, proj, a_log, bias, state = inputs(cuda_device, B, S, G, H, D, V, dtype)
    a_log -= 8.0
    conv[0, at, 2 * G * D:] = torch.finfo(dtype).min
    proj[0, at, 1:1 + H] = 30.0
    pad = torch.zeros(B, dtype=torch.int32, device=cuda_device)
    want_o, want_s = statement(conv, proj, a_log, bias, state, G, H, D, V, 0, pad)
    o = ops.gated_delta_rule(conv, G, H, D, V, proj, 1, 1 + H, a_log, bias, state, 0, pad)
    assert float((o.double() - want_o).abs().max()) <= 2e-6 * float(want_o.abs().max())
    assert float((state.double() - want_s).abs().max()) <= 2e-6 * float(want_s.abs().max())


def test_the_largest_outputs(ops, cuda_device):
    """a state near the end of the range that is read and hardly changed: every partial product stays in the range as the outputs do"""
    B, S, G, H, D, V = 1, 96, 1, 2, 128, 24
    conv, proj, a_log, bias, state = inputs(cuda_device, B, S, G, H, D, V, torch.float32)
    conv[..., :D].abs_()
    conv[..., D:2 * D] -= conv[..., D:2 * D].mean(-1, keepdim=True)                # keys at right angles to the state's columns
    proj[..., 1:1 + H], a_log = -30.0, a_log - 8.0
    state.fill_(2e38)
    pad = torch.zeros(B, dtype=torch.int32, device=cuda_device)
    want_o, want_s = statement(conv, proj, a_log, bias, state, G, H, D, V, 0, pad)
    assert float(want_o.abs().max()) > 1.5e38
    o = ops.gated_delta_rule(conv, G, H, D, V, proj, 1, 1 + H, a_log, bias, state, 0, pad)
    assert float((o.double() - want_o).abs().max()) <= 2e-6 * float(want_o.abs().max())
    assert float((state.double() - want_s).abs().max()) <= 2e-6 * float(want_s.abs().max())
