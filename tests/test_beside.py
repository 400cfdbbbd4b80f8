"""Weight gradients that start beside the launch in front of them: only where that launch is not the zeroing of their own output.  The library is
a stand-in that records its calls."""
import contextlib

import pytest
import torch

from gradient_compression_b200.ops import conv, gemm


@pytest.fixture
def calls(monkeypatch):
    seen = []

    class Library:
        def __getattr__(self, name):
            return lambda *args: seen.append((name, args[-1])) or 0

    monkeypatch.setattr(gemm.nat, "cuda", Library)
    monkeypatch.setattr(gemm.nat, "stream_ptr", lambda: None)
    monkeypatch.setattr(gemm, "tn_supported", lambda *_: True)
    monkeypatch.setattr(torch.cuda, "device", lambda _: contextlib.nullcontext())
    return seen


@pytest.mark.parametrize("beside", [False, True])
@pytest.mark.parametrize("out,accumulate", [(False, False), (True, False), (True, True)])
def test_product_waits_for_the_zeroing_of_its_output(calls, out, accumulate, beside):
    a, b = torch.ones(64, 32), torch.ones(64, 32)
    gemm.gemm_tn_tf32(a, b, out=torch.ones(32, 32) if out else None, accumulate=accumulate, beside=beside)
    assert calls == [("gc_cuda_gemm_tn_tf32", int(beside and accumulate))]


@pytest.mark.parametrize("beside", [False, True])
@pytest.mark.parametrize("out", [False, True])
def test_convolution_waits_for_the_zeroing_of_its_output(calls, out, beside):
    dy, x = torch.ones(1, 32, 4, 4), torch.ones(1, 32, 4, 4)
    conv.conv_wgrad(dy, x, 3, 1, 1, out=torch.ones(32, 288) if out else None, beside=beside)
    assert calls == [("gc_cuda_conv_wgrad", int(beside and out))]
