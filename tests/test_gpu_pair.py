"""CTA pairs of the persistent tensor-core kernel (256-row tiles) against the single-CTA tiles of the same width, whose contraction
order they share, and against an fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from gradient_compression_b200.ops import conv, gemm  # noqa: E402


@pytest.fixture
def paired():
    def use(tile, pairs, splits=1):
        gemm.configure("auto", tile)
        gemm.configure_pair(pairs)
        gemm.configure_split(splits)
    yield use
    use(0, 0, 0)


def both(paired, tile, call, splits=1):
    out = []
    for pairs in (1, 2):
        paired(tile, pairs, splits)
        out.append(call().clone())
    return out


def close(a, b, tol=3e-3):
    assert float((a.double() - b.double()).norm() / b.double().norm()) < tol


@pytest.mark.parametrize("tile", [64, 128, 256])
@pytest.mark.parametrize("m,n,k", [(129, 20, 4), (256, 64, 32), (257, 68, 100), (640, 260, 96), (19000, 256, 64), (40000, 128, 160)])
def test_gemm(paired, tile, m, n, k):
    """Second CTA with one row, none of its rows, ragged columns, one and several tiles per pair."""
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a, b = torch.randn(m, k, device="cuda", generator=g), torch.randn(n, k, device="cuda", generator=g)
    bias = torch.randn(n, device="cuda", generator=g)
    one, two = both(paired, tile, lambda: gemm.gemm_tf32(a, b, bias))
    assert torch.equal(one, two)
    close(two, a @ b.t() + bias)
    base = torch.randn(m, n, device="cuda", generator=g)
    one, two = both(paired, tile, lambda: gemm.gemm_tf32(a, b, out=base.clone(), accumulate=True))
    assert torch.equal(one, two)


@pytest.mark.parametrize("tile", [64, 128, 256])
def test_split_and_sums(paired, tile):
    g = torch.Generator(device="cuda").manual_seed(3)
    a, b = torch.randn(700, 1024, device="cuda", generator=g), torch.randn(96, 1024, device="cuda", generator=g)
    one, two = both(paired, tile, lambda: gemm.gemm_tf32(a, b), splits=3)
    close(two, one, 1e-5)
    paired(tile, 2)
    rows = gemm.m_tiles(700)
    partials = torch.full((rows, 2, 96), float("nan"), device="cuda")
    y = gemm.gemm_tf32(a, b, col_partials=partials)
    close(partials[:, 0].double().sum(0), y.double().sum(0), 1e-5)
    close(partials[:, 1].double().sum(0), (y.double() ** 2).sum(0), 1e-5)


@pytest.mark.parametrize("tile", [64, 128, 256])
@pytest.mark.parametrize("n,h,cin,cout,stride", [(1, 16, 32, 64, 1), (3, 16, 64, 96, 1), (18, 8, 64, 128, 2), (70, 16, 32, 64, 1), (20, 4, 96, 64, 1)])
def test_conv(paired, tile, n, h, cin, cout, stride):
    """Forward and input gradient (filter read in place), one image to several tiles per pair; exact on small integers."""
    lib, st = conv.nat.cuda(), conv.nat.stream_ptr()
    flag = gemm._error_flag(torch.device("cuda", 0)).data_ptr()
    g = torch.Generator().manual_seed(n + h)
    ints = lambda *shape: torch.randint(-3, 4, shape, generator=g).float().cuda().contiguous(memory_format=torch.channels_last)  # noqa: E731
    x, w, dy = ints(n, cin, h, h), ints(cout, cin, 3, 3), ints(n, cout, h // stride, h // stride)
    assert lib.gc_cuda_conv_fwd_supported(n, h, h, cin, cout, 3, stride, 1)
    paired(tile, 2)
    assert torch.equal(conv.conv_forward(x, w, None, stride, 1), torch.nn.functional.conv2d(x.double(), w.double(), None, stride, 1).float())
    dx = torch.empty_like(x)
    if stride == 1:
        conv.nat.check(lib.gc_cuda_conv_dgrad(dy.data_ptr(), w.data_ptr(), dx.data_ptr(), n, h, h, cin, cout, 3, 1, 0, flag, st), "dgrad")
    elif lib.gc_cuda_conv_dgrad_s2_supported(n, h, h, cin, cout, 3, 1):
        conv.nat.check(lib.gc_cuda_conv_dgrad_s2(dy.data_ptr(), w.data_ptr(), dx.data_ptr(), n, h, h, cin, cout, 3, 1, flag, st), "dgrad_s2")
    else:
        return
    ref = torch.ops.aten.convolution_backward(dy.double(), x.double(), w.double(), None, [stride] * 2, [1, 1], [1, 1], False, [0, 0], 1,
                                              [True, False, False])[0].float()
    gemm.check()
    assert torch.equal(dx, ref)


@pytest.mark.parametrize("tile", [128, 256])
@pytest.mark.parametrize("p,mo,no", [(1, 160, 32), (33, 256, 96), (1000, 384, 288), (70000, 512, 160), (40, 2048, 512)])
def test_weight_gradient_matrix(paired, tile, p, mo, no):
    """Second CTA with 32 rows, all or none of its rows; ragged columns; fewer positions than a stage; exact on small integers."""
    g = torch.Generator(device="cuda").manual_seed(p + mo)
    a, b = (torch.randint(-2, 3, (p, d), device="cuda", generator=g).float() for d in (mo, no))
    paired(tile, 2)
    out = gemm.gemm_tn_tf32(a, b, out=torch.ones(mo, no, device="cuda"), accumulate=True)
    gemm.check()
    assert torch.equal(out, (a.double().t() @ b.double() + 1).float())


@pytest.mark.parametrize("n,h,cin,cout,stride", [(2, 8, 128, 160, 1), (5, 8, 256, 256, 2), (3, 16, 256, 384, 1), (40, 4, 512, 512, 1)])
def test_weight_gradient_conv(paired, n, h, cin, cout, stride):
    g = torch.Generator().manual_seed(n + h)
    ints = lambda *shape: torch.randint(-3, 4, shape, generator=g).float().cuda().contiguous(memory_format=torch.channels_last)  # noqa: E731
    x, dy = ints(n, cin, h, h), ints(n, cout, h // stride, h // stride)
    paired(0, 2)
    if not conv.nat.cuda().gc_cuda_conv_wgrad_supported(n, h, h, cin, cout, 3, stride, 1):
        pytest.skip("not a tensor-core shape")
    dw = conv.conv_wgrad(dy, x, 3, stride, 1)
    gemm.check()
    w = torch.zeros(cout, cin, 3, 3, device="cuda", dtype=torch.float64)
    ref = torch.ops.aten.convolution_backward(dy.double(), x.double(), w, None, [stride] * 2, [1, 1], [1, 1], False, [0, 0], 1, [False, True, False])[1]
    assert torch.equal(dw.view(cout, 3, 3, cin), ref.permute(0, 2, 3, 1).float())


@pytest.mark.parametrize("pairs", [1, 2])
@pytest.mark.parametrize("r", [1, 3])
def test_strided_input_gradient_onto_an_existing_one(paired, r, pairs):
    n, h, cin, cout = 6, 16, 64, 96
    g = torch.Generator().manual_seed(r)
    ints = lambda *shape: torch.randint(-3, 4, shape, generator=g).float().cuda().contiguous(memory_format=torch.channels_last)  # noqa: E731
    x, w, dy, dx = ints(n, cin, h, h), ints(cout, cin, r, r), ints(n, cout, h // 2, h // 2), ints(n, cin, h, h)
    ref = torch.ops.aten.convolution_backward(dy.double(), x.double(), w.double(), None, [2, 2], [r // 2] * 2, [1, 1], False, [0, 0], 1,
                                              [True, False, False])[0].float() + dx
    paired(0, pairs)
    lib, flag = conv.nat.cuda(), gemm._error_flag(torch.device("cuda", 0)).data_ptr()
    conv.nat.check(lib.gc_cuda_conv_dgrad_s2_add(dy.data_ptr(), w.data_ptr(), dx.data_ptr(), n, h, h, cin, cout, r, r // 2, 1, flag, conv.nat.stream_ptr()), "add")
    gemm.check()
    assert torch.equal(dx, ref)
