"""Prompt attention over the e5m2 cache (csrc/sdp_prefill.cuh): edges of its 128-row and 128-key tiles, both CTA sizes, masks, rows
whose maximum keeps growing, against float64 on the same bytes.

Bound (that of the decode kernel's tests): queries and probabilities enter the products as fp16 (2^-11 each, probabilities relative to
the row's largest), sums in 32 bits: 1e-3 of the largest |output| for fp16 results, 8e-3 for bf16 (2^-8 of an element for the
result's own rounding)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = {torch.float16: 1e-3, torch.bfloat16: 8e-3}


@pytest.fixture(scope="module")
def kv(native_lib, cuda_device):
    from ipex_llm_b200.transformers import kv as module
    yield module
    assert not native_lib.lowbit_gemm_wait_expired()


def inputs(dev, B, Hq, Hkv, S, L, dtype, growth=0.0, seed=0):
    g = torch.Generator(device=dev).manual_seed(seed + S + L)
    q = torch.randn(B, S, Hq, 128, generator=g, device=dev).to(dtype).transpose(1, 2)
    k, v = (torch.randn(B, Hkv, L + 5, 128, generator=g, device=dev) for _ in range(2))
    if growth:                                                 # every key tile holds larger scores than the one before
        k = k * (1 + growth * torch.arange(L + 5, device=dev)[:, None])
    k, v = (t.to(torch.float8_e5m2).view(torch.uint8)[:, :, :L] for t in (k, v))          # views of a longer cache
    return q, k, v


def statement(q, k, v, mask, causal, scale):
    B, H, S, _ = q.shape
    L = k.shape[2]
    k, v = (t.contiguous().view(torch.float8_e5m2).double().repeat_interleave(H // t.shape[1], 1) for t in (k, v))
    s = q.double() @ k.transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(torch.ones(S, L, dtype=torch.bool, device=q.device).triu(L - S + 1), -math.inf)
    if mask is not None:
        s = s + mask.double()
    p = torch.softmax(s, -1)
    return torch.where(torch.isnan(p), torch.zeros_like(p), p) @ v                        # a row without a visible key gives zeros


def check(kv, q, k, v, mask, causal, scale=128 ** -0.5):
    got = kv.sdp_fp8_prefill(q, k, v, mask, scale, causal).double()
    want = statement(q, k, v, mask, causal, scale)
    assert float((got - want).abs().max()) <= TOL[q.dtype] * float(want.abs().max())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,Hq,Hkv,S,L", [(1, 1, 1, 1, 1), (1, 2, 1, 33, 33), (1, 2, 2, 127, 128), (2, 4, 2, 128, 128), (1, 4, 1, 129, 300), (1, 3, 3, 255, 256),
                                          (1, 2, 1, 257, 1000), (2, 80, 8, 129, 129), (5, 32, 8, 256, 256), (5, 32, 32, 257, 385), (1, 32, 8, 1300, 1300)])
@pytest.mark.parametrize("causal", [True, False])
def test_tiles(kv, cuda_device, dtype, B, Hq, Hkv, S, L, causal):
    check(kv, *inputs(cuda_device, B, Hq, Hkv, S, L, dtype), None, causal)


@pytest.mark.parametrize("S,L,heads", [(200, 700, 2), (300, 513, 80)])
def test_growing_maxima_rescale_what_was_summed(kv, cuda_device, S, L, heads):
    q, k, v = inputs(cuda_device, 1, heads, heads, S, L, torch.float16, growth=0.02)
    for scale in (128 ** -0.5, 1.0):                          # scores up to thousands: the softmax picks single keys
        check(kv, q, k, v, None, True, scale)


@pytest.mark.parametrize("S,L,Hq", [(70, 300, 2), (258, 258, 160)])
@pytest.mark.parametrize("kind", ["padding", "lowest", "rows without keys", "random"])
def test_masks(kv, cuda_device, S, L, Hq, kind):
    q, k, v = inputs(cuda_device, 2, Hq, Hq // 2, S, L, torch.float16)
    g = torch.Generator(device=cuda_device).manual_seed(S)
    m = torch.zeros(2, 1, S, L, device=cuda_device)
    if kind == "padding":
        m[1, :, :, :131] = -math.inf
    elif kind == "lowest":                                    # finite, so a row of nothing else is the plain average
        m = m.half()
        m[0, :, :, ::3] = torch.finfo(torch.float16).min
        m[1, :, 5] = torch.finfo(torch.float16).min
    elif kind == "rows without keys":
        m[0, :, ::7] = -math.inf
    else:
        m = torch.randn(2, 1, S, L, generator=g, device=cuda_device)
    check(kv, q, k, v, m.expand(2, Hq, S, L), False)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("S,L,Hq", [(70, 300, 2), (300, 512, 80)])
def test_the_denominator_fits_what_the_product_sums(kv, native_lib, cuda_device, dtype, S, L, Hq):
    """Values of one everywhere: an output is the sum of the probabilities that the product takes over the denominator, and one again.
    What is left are 32-bit sums: L / 8 steps of the tensor cores, each dropping up to 2^-22 of the sum, and L / 4 additions of 2^-24.
    Probabilities that are rounded for the one and not for the other leave 1e-4."""
    q, k, v = inputs(cuda_device, 1, Hq, Hq, S, L, dtype)
    v = torch.ones(v.shape, device=cuda_device).to(torch.float8_e5m2).view(torch.uint8)
    out = torch.empty(1, Hq, S, 128, device=cuda_device)
    for scale in (128 ** -0.5, 0.3):
        native_lib.lowbit_sdp_fp8_prefill(q, k, v, None, True, scale, out, torch.cuda.current_stream().cuda_stream)
        assert float((out - 1).abs().max()) <= L / 8 * 2.0 ** -22 + L / 4 * 2.0 ** -24


@pytest.mark.parametrize("S,L,Hq,Hkv,causal", [(40, 200, 2, 1, True), (129, 129, 4, 2, True), (300, 1077, 8, 2, True), (700, 700, 80, 8, True), (260, 900, 2, 2, False)])
@pytest.mark.parametrize("scale", [0.02, 128 ** -0.5, 0.3, 1.0])
def test_the_probabilities_are_not_rounded_to_16_bits(kv, native_lib, cuda_device, S, L, Hq, Hkv, causal, scale):
    """32-bit results: the sums' error, not fp16's 2^-12 of every probability (1e-4 here, with the largest one exact or not).  A score's
    eight steps drop up to 2^-23 of it each, which is that much of its probability; so do the L / 8 steps of P . V of the result."""
    q, k, v = inputs(cuda_device, 1, Hq, Hkv, S, L, torch.float16)
    out = torch.empty(1, Hq, S, 128, device=cuda_device)
    native_lib.lowbit_sdp_fp8_prefill(q, k, v, None, causal, scale, out, torch.cuda.current_stream().cuda_stream)
    want = statement(q, k, v, None, causal, scale)
    keys = k.contiguous().view(torch.float8_e5m2).double().repeat_interleave(Hq // Hkv, 1)
    largest = float((q.double() @ keys.transpose(-1, -2)).abs().max()) * scale
    assert float((out.double() - want).norm() / want.norm()) <= (8 * largest + L / 8 + 4) * 2.0 ** -23
