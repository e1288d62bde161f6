"""The product with the transposed packed weight behind MatMulLowBit's backward (gemm_pair.cu, GRAD) against dequantise-and-multiply."""
import threading

import pytest
import torch
import torch.autograd.forward_ad as fw

pytestmark = pytest.mark.gpu
QTYPES = ["sym_int4", "asym_int4", "nf4", "fp8_e4m3", "fp8_e5m2", "fp6"]


@pytest.fixture
def lbl(native_lib):
    from ipex_llm_b200.transformers import low_bit_linear
    return low_bit_linear


def weight(lbl, dev, n, k, qtype, std=0.02):
    w = torch.randn(n, k, device=dev, generator=torch.Generator(device=dev).manual_seed(n + k)) * std
    return lbl.FP4Params(w, qtype=lbl.ggml_tensor_qtype[qtype]).to(dev)


@pytest.mark.parametrize("qtype", QTYPES)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_a_unit_gradient_reads_the_dequantised_rows(lbl, cuda_device, qtype, dtype):
    """the weights in the product are the bits that dequantising gives, minima and table included"""
    p = weight(lbl, cuda_device, 192, 384, qtype)
    want = lbl.dequantize_device_layout(p.data, (192, 384), p.qtype, dtype=dtype)
    got = lbl.lowbit_matmul_grad(torch.eye(192, device=cuda_device, dtype=dtype), p.data, (192, 384), p.qtype)
    if qtype == "asym_int4" and dtype == torch.float16:                # one fma there, a product and a sum here: the last bit of few
        assert float((got != want).float().mean()) < 2e-3 and bool(((got - want).abs() <= 2.0 ** -10 * want.abs() + 2.0 ** -24).all())
    else:
        assert torch.equal(got, want)


@pytest.mark.parametrize("m,n,k", [(1, 64, 128), (17, 128, 384), (65, 192, 128), (100, 4096, 1024), (257, 320, 640), (129, 704, 4224), (513, 2048, 256)])
@pytest.mark.parametrize("qtype,dtype", [(q, d) for q in QTYPES for d in (torch.float16, torch.bfloat16)])
def test_gradient_edges(lbl, native_lib, cuda_device, qtype, dtype, m, n, k):
    """odd numbers of 64-row groups and of feature pairs, ragged tokens, split and whole row ranges.  Bound: 32-bit sums (2e-6 of sum|g w|)
    of weights that are exact here, the result rounded once"""
    p = weight(lbl, cuda_device, n, k, qtype)
    g = torch.randn(m, n, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(m)).to(dtype)
    w = lbl.dequantize_device_layout(p.data, (n, k), p.qtype, dtype=dtype).double()
    want, mag = g.double() @ w, g.double().abs() @ w.abs()
    last = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    slack = 2.0 ** -11 if qtype == "asym_int4" and dtype == torch.float16 else 0.0         # see above: few weights differ in their last bit
    bound = last * want.abs() + (2e-6 + 2e-3 * slack) * mag + slack * (g.double().abs().amax() * w.abs().amax()) * 4 + 2.0 ** -24
    got = lbl.lowbit_matmul_grad(g, p.data, (n, k), p.qtype)
    assert bool(((got.double() - want).abs() <= bound).all())
    assert torch.equal(lbl.lowbit_matmul_grad(g.t().contiguous().t(), p.data, (n, k), p.qtype), got)          # another stride
    odd = torch.empty(m * n + 1, device=cuda_device, dtype=dtype)[1:].view(m, n)
    odd.copy_(g)
    assert torch.equal(lbl.lowbit_matmul_grad(odd, p.data, (n, k), p.qtype), got)                             # off a 16-byte boundary
    whole = torch.empty_like(got)                                                                             # no scratch: rows not split
    native_lib.lowbit_matmul_grad_cuda(p.data.data_ptr(), p.qtype, n, k, g.data_ptr(), lbl._TORCH_TO_DT[dtype], m, whole.data_ptr(), None, 0,
                                       torch.cuda.current_stream().cuda_stream)
    assert bool(((whole.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("m,n,k", [(1100, 576, 8320), (1500, 576, 8320), (2500, 320, 4224)])
@pytest.mark.parametrize("qtype,dtype", [("sym_int4", torch.float16), ("nf4", torch.bfloat16), ("fp8_e4m3", torch.bfloat16), ("asym_int4", torch.float16)])
def test_gradient_over_several_units_a_cluster(lbl, native_lib, cuda_device, qtype, dtype, m, n, k):
    """rings, parities and the second accumulator carried from unit to unit, an epilogue beside the next unit's products, tiles of 192 to 256
    tokens with a ragged last one"""
    units = (k // 128 + 1) // 2 * -(-m // 256)                         # at least: no tile holds more than 256 tokens
    assert units > 2 * (torch.cuda.get_device_properties(cuda_device).multi_processor_count // 2)
    test_gradient_edges(lbl, native_lib, cuda_device, qtype, dtype, m, n, k)


def test_backward_takes_it_or_the_general_path(lbl, cuda_device, monkeypatch):
    """expanded and 3-dimensional half gradients in one launch; 32-bit ones, a derivative of the gradient in either direction, batched, negated
    and zero ones, those under an autocast to another type and other shapes by dequantising, with the same values"""
    calls = []
    real = lbl.lowbit_matmul_grad
    monkeypatch.setattr(lbl, "lowbit_matmul_grad", lambda *a: calls.append(1) or real(*a))
    p = weight(lbl, cuda_device, 256, 384, "sym_int4")
    wd = {d: lbl.dequantize_device_layout(p.data, (256, 384), p.qtype, dtype=d).double() for d in (torch.float16, torch.float32)}
    for dtype, taken in ((torch.float16, 1), (torch.float32, 0)):
        x = torch.randn(2, 30, 384, device=cuda_device).to(dtype).requires_grad_(True)
        y = lbl.MatMulLowBit.apply(x, p, 256)
        calls.clear()
        y.sum().backward()
        assert len(calls) == taken
        assert torch.allclose(x.grad.double(), wd[dtype].sum(0).expand_as(x), rtol=2e-3, atol=2e-3)
    x = torch.randn(5, 384, device=cuda_device).half().requires_grad_(True)
    y = lbl.MatMulLowBit.apply(x, p, 256)
    g = torch.randn(5, 256, device=cuda_device).half().requires_grad_(True)
    calls.clear()
    (gx,) = torch.autograd.grad(y, x, g, create_graph=True, retain_graph=True)
    (gg,) = torch.autograd.grad(gx.float().sum(), g)
    assert not calls and torch.allclose(gg.double(), wd[torch.float16].sum(1).expand_as(gg), rtol=2e-3, atol=2e-3)
    (batched,) = torch.autograd.grad(y, x, torch.stack([g.detach(), 2 * g.detach()]), is_grads_batched=True)
    assert not calls and torch.allclose(batched[0].double(), g.detach().double() @ wd[torch.float16], rtol=2e-3, atol=2e-3)
    tangent = torch.randn(5, 256, device=cuda_device).half()
    with fw.dual_level():                                               # a tangent of the gradient is carried on
        (gd,) = torch.autograd.grad(y, x, fw.make_dual(g.detach(), tangent), retain_graph=True)
        primal, moved = fw.unpack_dual(gd)
        assert not calls and moved is not None
        assert torch.allclose(primal.double(), g.detach().double() @ wd[torch.float16], rtol=2e-3, atol=2e-3)
        assert torch.allclose(moved.double(), tangent.double() @ wd[torch.float16], rtol=2e-3, atol=2e-3)
    for lazy, want in ((torch._neg_view(g.detach()), -g.detach().double()),       # the sign and the zeros are not in memory
                       (torch._efficientzerotensor((5, 256), dtype=torch.float16, device=cuda_device), torch.zeros(5, 256, device=cuda_device).double())):
        (gl,) = torch.autograd.grad(y, x, lazy, retain_graph=True)
        assert not calls and torch.allclose(gl.double(), want @ wd[torch.float16], rtol=2e-3, atol=2e-3)
    with torch.autocast("cuda", dtype=torch.bfloat16):                  # the product in bf16, as autocast has matmul do it
        (ga,) = torch.autograd.grad(y, x, g.detach(), retain_graph=True)
        assert not calls and torch.equal(ga, torch.matmul(g.detach(), wd[torch.float16].half()).half())
    (gp,) = torch.autograd.grad(y, x, g.detach(), retain_graph=True)    # ... and a plain one is the kernel's again
    assert len(calls) == 1 and torch.allclose(gp.double(), g.detach().double() @ wd[torch.float16], rtol=2e-3, atol=2e-3)
    calls.clear()
    q = weight(lbl, cuda_device, 100, 192, "sym_int4")                  # rows behind the last 64, columns no multiple of 128
    x = torch.randn(70, 192, device=cuda_device).half().requires_grad_(True)
    lbl.MatMulLowBit.apply(x, q, 100).sum().backward()
    assert not calls and x.grad is not None
    with pytest.raises(RuntimeError):
        real(torch.zeros(4, 100, device=cuda_device).half(), q.data, (100, 192), q.qtype)


def test_a_thread_whose_first_call_it_is(lbl, cuda_device):
    """autograd runs backward in threads of its own, which may have made no call into CUDA yet"""
    p = weight(lbl, cuda_device, 256, 384, "sym_int4")
    g = torch.randn(70, 256, device=cuda_device).half()
    want, got = lbl.lowbit_matmul_grad(g, p.data, (256, 384), p.qtype), []
    t = threading.Thread(target=lambda: got.append(lbl.lowbit_matmul_grad(g, p.data, (256, 384), p.qtype)))
    t.start()
    t.join()
    assert got and torch.equal(got[0], want)
