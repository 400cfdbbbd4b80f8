"""Input gradients of stride-2 convolutions, the four parity classes of input pixels in one launch: tiles of part of an image, of one image and of several, tiles
beyond the batch, columns that end inside a tile, more tiles than workers; filters the kernel does not cover are refused."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from gradient_compression_b200.ops import conv, gemm  # noqa: E402

# (N, H, W, Cin, Cout, R); the one of 36 channels has no whole chunks of 32 and takes a launch per class, R = 2 has one tap in every class
SHAPES = [(1, 32, 32, 64, 32, 3), (3, 16, 16, 160, 64, 3), (2, 8, 64, 32, 32, 3), (37, 4, 4, 96, 64, 3), (5, 8, 8, 64, 96, 3), (150, 16, 16, 288, 32, 3), (3, 8, 8, 36, 32, 3),
          (9, 16, 8, 64, 32, 2)]


@pytest.fixture
def setting():
    def use(tile=0, pairs=0):
        gemm.configure("auto", tile)
        gemm.configure_pair(pairs)
    yield use
    use()


@pytest.mark.parametrize("tile,pairs", [(0, 0), (64, 1), (128, 1), (256, 1), (64, 2), (128, 2), (256, 2)])
@pytest.mark.parametrize("n,h,w,cin,cout,r", SHAPES)
def test_exact_on_small_integers(setting, n, h, w, cin, cout, r, tile, pairs):
    g = torch.Generator().manual_seed(n + h)
    pad = r // 2 if r & 1 else 0
    ints = lambda *shape: torch.randint(-3, 4, shape, generator=g).float().cuda().contiguous(memory_format=torch.channels_last)  # noqa: E731
    x, wt, dy, base = ints(n, cin, h, w), ints(cout, cin, r, r), ints(n, cout, h // 2, w // 2), ints(n, cin, h, w)
    lib, st, flag = conv.nat.cuda(), conv.nat.stream_ptr(), gemm._error_flag(torch.device("cuda", 0)).data_ptr()
    assert lib.gc_cuda_conv_dgrad_s2_supported(n, h, w, cin, cout, r, pad)
    setting(tile, pairs)
    back = torch.ops.aten.convolution_backward(dy.double(), x.double(), wt.double(), None, [2, 2], [pad, pad], [1, 1], False, [0, 0], 1, [True, False, False])[0]
    for accumulate in (0, 1):
        dx = base.clone(memory_format=torch.channels_last)
        conv.nat.check(lib.gc_cuda_conv_dgrad_s2_add(dy.data_ptr(), wt.data_ptr(), dx.data_ptr(), n, h, w, cin, cout, r, pad, accumulate, flag, st), "dgrad_s2")
        gemm.check()
        assert torch.equal(dx, (back + accumulate * base.double()).float())
