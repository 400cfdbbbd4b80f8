"""What libtorch throws inside the extension module's calls reaches Python as an exception."""
import pytest
import torch


@pytest.mark.filterwarnings("ignore:Accessing the data pointer")
@pytest.mark.skipif(torch.cuda.is_available(), reason="relies on the CUDA runtime having no device to answer for")
def test_exceptions_do_not_end_the_process():
    from torch._subclasses.fake_tensor import FakeTensorMode

    from gradient_compression_b200.ops import _native as nat

    ext = nat.ext()
    with FakeTensorMode():                      # tensors that say they are on a GPU: the first call that asks for one throws
        x, w = torch.empty(64, device="cuda"), torch.empty(10, 64, device="cuda")
        f = torch.empty(2, 64, 4, 4, device="cuda").contiguous(memory_format=torch.channels_last)
        for call in (lambda: ext.classify(f, w, None), lambda: ext.absmax(x, None)):
            with pytest.raises(RuntimeError):
                call()
    assert ext.absmax(torch.zeros(3), None) is None


@pytest.mark.gpu
def test_out_of_memory_is_raised():
    from gradient_compression_b200 import ops

    x = torch.randn(1 << 24, device="cuda")
    norm = ops.absmax(x)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (8 << 20)) / total)
        with pytest.raises(torch.OutOfMemoryError):
            ops.quantize_levels(x, norm, 255)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert int(ops.quantize_levels(x, norm, 255).abs().max()) == 255
