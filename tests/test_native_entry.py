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


@pytest.mark.gpu
def test_other_threads_run_while_a_launch_waits():
    """A thousand launches behind a busy stream fill its queue, and the next one waits: not with the interpreter lock held."""
    import threading
    import time

    from gradient_compression_b200 import ops

    x, norm = torch.randn(64, device="cuda"), torch.ones(1, device="cuda")
    out = torch.empty(64, dtype=torch.int8, device="cuda")
    ops.quantize_levels(x, norm, 7, out=out)
    torch.cuda.synchronize()
    longest, stop = [0.0], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            longest[0], last = max(longest[0], now - last), now

    thread = threading.Thread(target=tick)
    thread.start()
    torch.cuda._sleep(1_000_000_000)                # about half a second
    start = time.perf_counter()
    for _ in range(4000):
        ops.quantize_levels(x, norm, 7, out=out)
    took = time.perf_counter() - start
    stop.set()
    thread.join()
    torch.cuda.synchronize()
    assert took > 0.2, "the queue never filled up"
    assert longest[0] < 0.8 * took          # (with the lock held: all but the last few milliseconds)


@pytest.mark.gpu
@pytest.mark.parametrize("number", [float, int, __import__("numpy").float64, __import__("numpy").int32, torch.tensor])
def test_scales_and_seeds_of_any_number_type(number):
    from gradient_compression_b200 import ops

    x, norm = torch.randn(1000, device="cuda"), torch.full((1,), 3.0, device="cuda")
    want = ops.quantize_levels(x.cpu(), 3.0, 7, 5, 9, 2)
    got = ops.quantize_levels(x, norm, number(7), number(5), number(9), number(2), dtype=torch.int8)
    assert got.dtype == torch.int8 and torch.equal(got.cpu().to(torch.int32), want)
    assert torch.equal(ops.dequantize_levels(got, norm, number(7), number(2)).cpu(), ops.dequantize_levels(want, 3.0, 7, 2))
    q, mask = ops.quantize_fit(x, norm, number(7), number(3), number(5), number(9), number(2))
    assert torch.equal(q.cpu(), want) and torch.equal(mask.cpu(), (want.abs() <= 3).to(torch.int8))
    assert torch.equal(ops.quantize_levels(x, norm, 7, 5, 9, 2, dtype=torch.uint8).view(torch.int8), got)        # a container of one byte


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_results_that_do_not_fit_are_refused(device):
    from gradient_compression_b200 import ops

    x, norm = torch.randn(1000, device=device), torch.full((1,), 3.0, device=device)
    q = ops.quantize_levels(x, norm, 7, out=torch.empty(1001, dtype=torch.int32, device=device))[:1000].contiguous()
    with pytest.raises(ValueError):
        ops.quantize_levels(x, norm, 7, out=torch.empty(999, dtype=torch.int32, device=device))
    with pytest.raises(ValueError):
        ops.dequantize_levels(q, norm, 7, out=torch.empty(999, device=device))
    with pytest.raises(ValueError):
        ops.absmax(x, torch.empty(0, device=device))
    assert torch.equal(ops.dequantize_levels(q, norm, 7, out=torch.empty(1000, device=device)), ops.dequantize_levels(q, norm, 7))
