"""Kernels that start while their predecessor on the stream is still running: a layer's weight gradient beside its input gradient, behind a
batch norm's backward that writes what both read, in front of a consumer of both; eager and replayed from a graph.  Exact on small integers."""
import os
import subprocess
import sys

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


def ints(gen, *shape):
    t = torch.randint(-2, 3, shape, generator=gen).float().cuda()
    return t.contiguous(memory_format=torch.channels_last) if t.dim() == 4 else t


def results(chain, captured):
    """What `chain` returns in four runs, eager or replayed."""
    if not captured:
        return [chain() for _ in range(4)]
    chain()
    torch.cuda.synchronize()
    graph, out = torch.cuda.CUDAGraph(), []
    with torch.cuda.graph(graph):
        got = chain()
    for _ in range(4):
        graph.replay()
        out.append([t.clone() for t in got])
    return out


def gradients(dy, x, w, stride, pad):
    return torch.ops.aten.convolution_backward(dy.double(), x.double(), w.double(), None, [stride] * 2, [pad] * 2, [1, 1], False, [0, 0], 1, [True, True, False])


def call(name, *args):
    lib, flag = conv.nat.cuda(), gemm._error_flag(torch.device("cuda", 0)).data_ptr()
    conv.nat.check(getattr(lib, name)(*[a.data_ptr() if torch.is_tensor(a) else a for a in args], flag, conv.nat.stream_ptr()), name)


def weight_gradient(dy, x, r, stride, dw):
    if r == 1 and stride == 1:
        gemm.gemm_tn_tf32(conv._as_2d(dy), conv._as_2d(x), out=dw, accumulate=True, beside=True)
    else:
        conv.conv_wgrad(dy, x, r, stride, r // 2, out=dw, beside=True)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("n,h,cin,cout,r", [(2, 16, 64, 64, 3), (33, 16, 64, 128, 3), (31, 8, 256, 512, 3), (40, 16, 64, 128, 1), (2, 8, 128, 96, 1)])
def test_beside_the_input_gradient_of_a_stride_2_layer(n, h, cin, cout, r, captured):
    gen = torch.Generator().manual_seed(n)
    x, w, src = ints(gen, n, cin, h, h), ints(gen, cout, cin, r, r), ints(gen, n, cout, h // 2, h // 2)
    dy, dx, dw, ballast = torch.zeros_like(src), torch.empty_like(x), torch.zeros(cout, r * r * cin, device="cuda"), torch.zeros(32 << 20, device="cuda")

    def chain():
        dy.zero_()
        dw.zero_()
        dx.fill_(float("nan"))
        ballast.add_(1.0)
        dy.copy_(src)
        call("gc_cuda_conv_dgrad_s2", dy, w, dx, n, h, h, cin, cout, r, r // 2)
        weight_gradient(dy, x, r, 2, dw)
        return dx.clone(), dw.clone()

    want = gradients(src, x, w, 2, r // 2)
    for a, b in results(chain, captured):
        assert torch.equal(a, want[0].float())
        assert torch.equal(b.view(cout, r, r, cin), want[1].permute(0, 2, 3, 1).float())
    gemm.check()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("n,h,cin,mid,cout,r,stride", [(20, 16, 64, 64, 128, 3, 2), (31, 8, 256, 128, 512, 1, 1), (40, 16, 64, 128, 256, 1, 1), (2, 8, 128, 64, 64, 3, 2)])
def test_behind_the_addition_of_a_shortcut(n, h, cin, mid, cout, r, stride, captured):
    """A block's first convolution and its strided 1x1 shortcut: the first one's input gradient, the shortcut's added onto it, the first one's
    weight gradient beside that addition."""
    gen = torch.Generator().manual_seed(n)
    x, w, ws = ints(gen, n, cin, h, h), ints(gen, mid, cin, r, r), ints(gen, cout, cin, 1, 1)
    src, dys = ints(gen, n, mid, h // stride, h // stride), ints(gen, n, cout, h // 2, h // 2)
    dy, dx, dw, ballast = torch.zeros_like(src), torch.empty_like(x), torch.zeros(mid, r * r * cin, device="cuda"), torch.zeros(32 << 20, device="cuda")

    def chain():
        dy.zero_()
        dw.zero_()
        dx.fill_(float("nan"))
        ballast.add_(1.0)
        dy.copy_(src)
        if stride == 2:
            call("gc_cuda_conv_dgrad_s2", dy, w, dx, n, h, h, cin, mid, r, r // 2)
        else:
            call("gc_cuda_conv_dgrad", dy, w, dx, n, h, h, cin, mid, r, r // 2, 0)
        call("gc_cuda_conv_dgrad_s2_add", dys, ws, dx, n, h, h, cin, cout, 1, 0, 1)
        weight_gradient(dy, x, r, stride, dw)
        return dx.clone(), dw.clone()

    want, short = gradients(src, x, w, stride, r // 2), gradients(dys, x, ws, 2, 0)
    for a, b in results(chain, captured):
        assert torch.equal(a, (want[0] + short[0]).float())
        assert torch.equal(b.view(mid, r, r, cin), want[1].permute(0, 2, 3, 1).float())
    gemm.check()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("splits", [2, 3])
@pytest.mark.parametrize("n,h,cin,cout,r", [(2, 8, 64, 512, 3), (24, 4, 512, 512, 3), (31, 8, 256, 512, 1)])
def test_behind_a_split_input_gradient(n, h, cin, cout, r, splits, captured):
    """The output is zeroed by a kernel in front of the product, which the product itself waits for."""
    gen = torch.Generator().manual_seed(n)
    x, w, src = ints(gen, n, cin, h, h), ints(gen, cout, cin, r, r), ints(gen, n, cout, h, h)
    dy, dx, dw, ballast = torch.zeros_like(src), torch.empty_like(x), torch.zeros(cout, r * r * cin, device="cuda"), torch.zeros(32 << 20, device="cuda")

    def chain():
        dy.zero_()
        dw.zero_()
        dx.fill_(float("nan"))
        ballast.add_(1.0)
        dy.copy_(src)
        call("gc_cuda_conv_dgrad", dy, w, dx, n, h, h, cin, cout, r, r // 2, 0)
        weight_gradient(dy, x, r, 1, dw)
        return dx.clone(), dw.clone()

    gemm.configure_split(splits)
    try:
        got = results(chain, captured)
    finally:
        gemm.configure_split(0)
    want = gradients(src, x, w, 1, r // 2)
    for a, b in got:
        assert torch.equal(a, want[0].float())
        assert torch.equal(b.view(cout, r, r, cin), want[1].permute(0, 2, 3, 1).float())
    gemm.check()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("n,positions,c,k", [(1, 1, 4, 1), (31, 16, 512, 10), (128, 16, 2048, 10), (130, 1, 100, 32)])
def test_the_two_gradients_of_the_head(n, positions, c, k, captured):
    gen = torch.Generator().manual_seed(n)
    src, pooled, w, g = ints(gen, n, k), ints(gen, n, c), ints(gen, k, c), torch.full((1,), 2.0, device="cuda")
    dl, dx, dw, db = torch.zeros_like(src), torch.empty(n, positions, c, device="cuda"), torch.empty(k, c, device="cuda"), torch.empty(k, device="cuda")
    ballast = torch.zeros(32 << 20, device="cuda")

    def chain():
        dl.zero_()
        ballast.add_(1.0)
        dl.copy_(src)
        conv.nat.check(conv.nat.cuda().gc_cuda_head_backward(dl.data_ptr(), pooled.data_ptr(), w.data_ptr(), g.data_ptr(), n, positions, c, k, dx.data_ptr(), dw.data_ptr(),
                                                             db.data_ptr(), conv.nat.stream_ptr()), "head_backward")
        return dx.clone(), dw.clone(), db.clone()

    for a, b, d in results(chain, captured):
        assert torch.equal(a, (2.0 * (src.double() @ w.double()) / positions).float()[:, None].expand(-1, positions, -1))
        assert torch.equal(b, (2.0 * (src.double().t() @ pooled.double())).float())
        assert torch.equal(d, (2.0 * src.double().sum(0)).float())


@pytest.mark.skipif(os.environ.get("GCB200_PDL") == "0", reason="this is that process")
def test_everything_without_programmatic_launches():
    """The same chains, and the other kernels that take part, launched the ordinary way (the switch is read once a process)."""
    here = os.path.dirname(os.path.abspath(__file__))
    files = [os.path.join(here, f) for f in ("test_gpu_overlap.py", "test_gpu_small_kernels.py", "test_gpu_solo.py", "test_gpu_step.py")]
    run = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", *files, "-k", "overlap or head or gather or topk_lists or powersgd or agree_at_first_steps"],
                         cwd=os.path.dirname(here), env=dict(os.environ, GCB200_PDL="0"), capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout[-3000:]
