"""The native host side of one linear (csrc/host/linear_host.cpp): when it is built and loaded, and what serves where it cannot be."""
import os
import subprocess
import sys
import sysconfig
import threading
import time

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def lbl(native_lib):
    from ipex_llm_b200.transformers import low_bit_linear
    return low_bit_linear


def test_importing_the_package_neither_builds_nor_loads_it():
    code = ("import ipex_llm_b200.build_native as b\n"
            "def no(*a, **k): raise AssertionError('built on import')\n"
            "b.build_host = no\n"
            "import ipex_llm_b200.transformers.models.mixtral\n"
            "assert 'b200_host' not in open('/proc/self/maps').read()\n")
    subprocess.run([sys.executable, "-c", code], cwd=ROOT, check=True)


def test_the_gradients_scratch_is_asked_for_on_the_weights_device(lbl, monkeypatch):
    """the number of SMs decides the splits: each device its own answer, whichever device is the current one"""
    current = [0]

    class Guard:
        def __init__(self, device):
            self.device = device.index

        def __enter__(self):
            self.before, current[0] = current[0], self.device

        def __exit__(self, *exc):
            current[0] = self.before

    monkeypatch.setattr(torch.cuda, "current_device", lambda: current[0])
    monkeypatch.setattr(torch.cuda, "device", Guard)
    monkeypatch.setattr(lbl.ggml, "lowbit_matmul_grad_workspace_size", lambda n, k, m: 1000 + current[0])
    lbl._grad_plan.cache_clear()
    try:
        sizes = [lbl._grad_plan(torch.device("cuda", i), lbl.SYM_INT4, 4096, 4096, 100) for i in (0, 1, 0)]
    finally:
        lbl._grad_plan.cache_clear()
    assert sizes == [1000, 1001, 1000] and current == [0]


@pytest.mark.parametrize("n,k,taken,left", [(11008, 4096, (16, 512, 1024), (1280, 4000)), (8192, 8192, (16, 512, 1024), (3000, 4000)),
                                            (4096, 11008, (16, 512, 1280), (4000,)), (2048, 8192, (16, 512), (2000, 3000)),
                                            (1024, 1024, (1, 1024), ()), (14336, 14336, (16, 1024), (3000,))])
def test_nf4_gradients_are_taken_where_that_is_quicker(lbl, n, k, taken, left):
    """both sides of the line for matrices whose times stand at the rule (148 SMs); the other formats always, shapes it has no kernel for never"""
    faster = lbl.ggml.lowbit_matmul_grad_faster
    assert [m for m in taken if not faster(lbl.NF4, n, k, m)] == [] and [m for m in left if faster(lbl.NF4, n, k, m)] == []
    assert all(faster(q, n, k, m) for q in (lbl.SYM_INT4, lbl.ASYM_INT4, lbl.ggml_tensor_qtype["fp6"], lbl.ggml_tensor_qtype["fp8_e4m3"]) for m in taken + left)
    assert not any(faster(q, a, b, 64) for q in (lbl.SYM_INT4, lbl.NF4) for a, b in ((n + 32, k), (n, k + 64))) and not faster(lbl.NF4, n, k, 0)


def test_the_file_is_named_by_what_it_is_bound_to():
    from ipex_llm_b200 import build_native
    name = os.path.basename(build_native.build_host())
    assert sysconfig.get_config_var("SOABI") in name and torch.__version__ in name


def test_where_it_cannot_be_built_the_python_statements_serve(lbl, monkeypatch):
    from ipex_llm_b200 import build_native

    def fails():
        raise RuntimeError("no compiler")
    monkeypatch.setattr(build_native, "build_host", fails)
    monkeypatch.setattr(lbl, "_host", None)
    with pytest.warns(UserWarning, match="no compiler"):
        assert lbl._load_host() is False
    assert lbl._load_host() is False                                               # asked for once


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 16, 40, 130])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
def test_both_give_the_same_bits(lbl, cuda_device, monkeypatch, rows, dtype):
    lin = lbl.LowBitLinear(512, 384, lbl.SYM_INT4, bias=True).to(cuda_device).eval()
    lin.bias.data = lin.bias.data.to(dtype)
    x = torch.randn(2, rows, 512, device=cuda_device).to(dtype)
    with torch.no_grad():
        native = lin(x)
        assert lbl._host
        monkeypatch.setattr(lbl, "_host", False)
        assert torch.equal(lin(x), native)


@pytest.mark.gpu
def test_other_threads_run_while_a_launch_waits(lbl, cuda_device):
    """more launches than the device's queue holds, behind a second of a busy stream: the calls wait, other threads do not"""
    lin = lbl.LowBitLinear(128, 128, lbl.SYM_INT4, bias=False).to(cuda_device).eval()
    x = torch.randn(1, 128, device=cuda_device).half()
    longest, stop = [0.0], threading.Event()

    def clock():
        last = time.monotonic()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.monotonic()
            longest[0], last = max(longest[0], now - last), now
    with torch.no_grad():
        lin(x)
        torch.cuda.synchronize()
        torch.cuda._sleep(2000000000)                                               # cycles
        ticking = threading.Thread(target=clock)
        ticking.start()
        try:
            for _ in range(4000):
                lin(x)
            torch.cuda.synchronize()
        finally:
            stop.set()
            ticking.join()
    assert longest[0] < 0.5


def _views(device, B, Hq, Hkv, S, L, D, dtype, order="shd"):
    """queries as the models hand them over (or laid out as named), keys and values as views of a longer cache"""
    gen = torch.Generator(device=device).manual_seed(B * L + S)
    q = torch.randn(B, S, Hq, D, device=device, generator=gen).to(dtype).transpose(1, 2)
    if order == "hsd":
        q = q.contiguous()
    elif order == "dense last dimension elsewhere":
        q = q.transpose(2, 3).contiguous().transpose(2, 3)
    elif order == "part of a wider row":
        q = torch.cat([q, q], -1)[..., :D]
    k, v = (torch.randn(B, Hkv, L + 40, D, device=device, generator=gen).to(torch.float8_e5m2).view(torch.uint8)[:, :, :L] for _ in range(2))
    return q, k, v


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 4, 4, 1, 1, 128), (3, 8, 2, 1, 130, 128), (8, 32, 8, 1, 700, 128), (1, 8, 1, 1, 9000, 128), (2, 8, 8, 3, 257, 128),
                                   (1, 32, 8, 8, 500, 128), (1, 12, 2, 32, 96, 128), (2, 8, 2, 1, 300, 64), (1, 4, 2, 5, 70, 96), (1, 4, 4, 33, 33, 128),
                                   (2, 8, 2, 200, 301, 128), (1, 4, 2, 40, 60, 64), (1, 4, 4, 50, 50, 80)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("order", ["shd", "hsd", "dense last dimension elsewhere", "part of a wider row"])
def test_attention_gives_the_same_bits_and_layout_either_way(lbl, cuda_device, monkeypatch, shape, dtype, order):
    """one native call, or the Python statements that it stands for (which serve the shapes it leaves to them)"""
    from ipex_llm_b200.transformers import kv
    B, Hq, Hkv, S, L, D = shape
    q, k, v = _views(cuda_device, *shape, dtype, order)
    for causal in (False, True):
        for scale in (None, 0.5):
            native = kv.scaled_dot_product_attention(q, k, v, None, causal, scale)
            assert lbl._host
            with monkeypatch.context() as m:
                m.setattr(lbl, "_host", False)
                want = kv.scaled_dot_product_attention(q, k, v, None, causal, scale)
            assert native.dtype == want.dtype and native.stride() == want.stride() and torch.equal(native, want)


@pytest.mark.gpu
def test_attention_refuses_and_leaves_alone_what_it_did(lbl, cuda_device, monkeypatch):
    """misaligned keys of a few tokens: the kernel's error either way; a batch, type or device that does not fit is not the native call's"""
    from ipex_llm_b200.transformers import kv
    q, k, v = _views(cuda_device, 1, 4, 2, 1, 64, 128, torch.float16)
    odd = torch.zeros(k.numel() + 1, dtype=torch.uint8, device=cuda_device)[1:].view(1, 2, 64, 128)
    host = lbl._load_host()
    assert host
    for serving in (host, False):
        monkeypatch.setattr(lbl, "_host", serving)
        with pytest.raises(RuntimeError):
            kv.scaled_dot_product_attention(q, odd, v, None, False)
    assert host.attention(q.double(), k, v, False, 1.0, True) is None
    assert host.attention(q, k[:, :, :63], v, False, 1.0, True) is None
    assert host.attention(torch.cat([q, q]), k, v, False, 1.0, True) is None
    assert host.attention(q, k.cpu(), v, False, 1.0, True) is None
    assert host.attention(q.expand(1, 4, 40, 128), torch.cat([k, k], 2), torch.cat([v, v], 2), True, 1.0, False) is None      # prompts switched off
