"""Input gradients of 3x3 convolutions whose filter columns share one load of the pixels, against float64: tiles of one image and of
several, the last one partly beyond the batch, split contractions, sums onto an existing gradient."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from gradient_compression_b200.ops import conv, gemm  # noqa: E402

# (N, H, W, Cin, Cout): tiles of 4 rows of 32, 8 of 16, 2 of 64 and 16 of 8 pixels with a row above and below; whole images of 8x8, 4x4, 2x2, 8x4; ragged last tiles
SHAPES = [(2, 32, 32, 64, 32), (3, 16, 16, 32, 64), (1, 64, 64, 32, 32), (2, 32, 8, 96, 32), (3, 8, 8, 160, 96), (17, 4, 4, 128, 64), (37, 2, 2, 64, 64), (5, 8, 4, 64, 32),
          (3, 8, 8, 36, 32)]      # the last one's filter is no whole chunks of 32 columns: a load per tap


@pytest.fixture
def setting():
    def use(tile=0, pairs=0, splits=0):
        gemm.configure("auto", tile)
        gemm.configure_pair(pairs)
        gemm.configure_split(splits)
    yield use
    use()


@pytest.mark.parametrize("tile,pairs,splits", [(0, 0, 0), (64, 1, 1), (128, 1, 2), (64, 2, 3), (128, 2, 1)])
@pytest.mark.parametrize("n,h,w,cin,cout", SHAPES)
def test_exact_on_small_integers(setting, n, h, w, cin, cout, tile, pairs, splits):
    g = torch.Generator().manual_seed(n + h)
    ints = lambda *shape: torch.randint(-3, 4, shape, generator=g).float().cuda().contiguous(memory_format=torch.channels_last)  # noqa: E731
    x, wt, dy, base = ints(n, cin, h, w), ints(cout, cin, 3, 3), ints(n, cout, h, w), ints(n, cin, h, w)
    lib, st, flag = conv.nat.cuda(), conv.nat.stream_ptr(), gemm._error_flag(torch.device("cuda", 0)).data_ptr()
    setting(tile, pairs, splits)
    back = torch.ops.aten.convolution_backward(dy.double(), x.double(), wt.double(), None, [1, 1], [1, 1], [1, 1], False, [0, 0], 1, [True, False, False])[0]
    for accumulate in (0, 1):
        dx = base.clone(memory_format=torch.channels_last)
        conv.nat.check(lib.gc_cuda_conv_dgrad(dy.data_ptr(), wt.data_ptr(), dx.data_ptr(), n, h, w, cin, cout, 3, 1, accumulate, flag, st), "dgrad")
        assert torch.equal(dx, (back + accumulate * base.double()).float())
    gemm.check()
