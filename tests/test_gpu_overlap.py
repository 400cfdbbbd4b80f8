"""Kernels that start while their predecessor on the stream is still running: a layer's weight gradient beside its input gradient, behind a
batch norm's backward that writes what both read, in front of a consumer of both; eager and replayed from a graph.  Exact on small integers."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from gradient_compression_b200.ops import conv, gemm  # noqa: E402


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("n,h,cin,cout,r", [(1, 8, 64, 64, 1), (2, 8, 64, 96, 3), (40, 16, 64, 128, 3), (128, 32, 64, 64, 1), (70, 4, 512, 256, 3)])
def test_gradients_side_by_side(n, h, cin, cout, r, captured):
    g = torch.Generator().manual_seed(n)
    ints = lambda *shape: torch.randint(-2, 3, shape, generator=g).float().cuda().contiguous(memory_format=torch.channels_last)  # noqa: E731
    x, w, src = ints(n, cin, h, h), ints(cout, cin, r, r), ints(n, cout, h, h)
    dy, dx, dw = torch.zeros_like(src), torch.empty_like(x), torch.zeros(cout, r * r * cin, device="cuda")
    ballast = torch.zeros(32 << 20, device="cuda")
    lib, flag = conv.nat.cuda(), gemm._error_flag(torch.device("cuda", 0)).data_ptr()
    out = []

    def chain():
        dy.zero_()
        dw.zero_()
        ballast.add_(1.0)                    # the writer of dy starts late
        dy.copy_(src)
        conv.nat.check(lib.gc_cuda_conv_dgrad(dy.data_ptr(), w.data_ptr(), dx.data_ptr(), n, h, h, cin, cout, r, r // 2, 0, flag, conv.nat.stream_ptr()), "dgrad")
        if r == 1:
            gemm.gemm_tn_tf32(conv._as_2d(dy), conv._as_2d(x), out=dw, accumulate=True, beside=True)
        else:
            conv.conv_wgrad(dy, x, r, 1, r // 2, out=dw, beside=True)
        return dx.clone(), dw.clone()

    if captured:
        chain()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = chain()
        for _ in range(4):
            graph.replay()
            out.append([t.clone() for t in got])
    else:
        out = [chain() for _ in range(4)]
    gemm.check()
    ref = torch.ops.aten.convolution_backward(src.double(), x.double(), w.double(), None, [1, 1], [r // 2] * 2, [1, 1], False, [0, 0], 1, [True, True, False])
    for a, b in out:
        assert torch.equal(a, ref[0].float())
        assert torch.equal(b.view(cout, r, r, cin), ref[1].permute(0, 2, 3, 1).float())
