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
