"""Edges of the stem's gather (columns that do not divide a block, padding columns, images of odd sizes) and of the head's gradients (samples around the eight that
a warp loads together, channels beyond the last block)."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

from gradient_compression_b200.ops import conv, head  # noqa: E402


@pytest.mark.parametrize("n,h,w,cin,r,kp", [(2, 5, 7, 3, 3, 32), (1, 4, 4, 1, 5, 28), (3, 6, 5, 2, 3, 128), (150, 9, 11, 3, 1, 4), (1, 1, 1, 3, 3, 32)])
def test_gather(n, h, w, cin, r, kp):
    g = torch.Generator().manual_seed(n + h)
    x = torch.randn(n, cin, h, w, generator=g).cuda().contiguous(memory_format=torch.channels_last)
    wt = torch.randn(8, cin, r, r, generator=g).cuda().contiguous(memory_format=torch.channels_last)
    a, wpad = torch.full((n * h * w, kp), 7.0, device="cuda"), torch.full((8, kp), 7.0, device="cuda")
    lib = conv.nat.cuda()
    conv.nat.check(lib.gc_cuda_im2col_small(x.data_ptr(), a.data_ptr(), n, h, w, cin, r, r // 2, kp, wt.data_ptr(), wpad.data_ptr(), 8, conv.nat.stream_ptr()), "gather")
    k = r * r * cin
    rows = F.unfold(x, r, padding=r // 2).view(n, cin, r * r, h * w).permute(0, 3, 2, 1).reshape(n * h * w, k)
    assert torch.equal(a, F.pad(rows, (0, kp - k))) and torch.equal(wpad, F.pad(wt.permute(0, 2, 3, 1).reshape(8, k), (0, kp - k)))


@pytest.mark.parametrize("n", [1, 7, 8, 9, 63, 64, 65, 200])
@pytest.mark.parametrize("c", [4, 36, 512])
def test_head_gradients(n, c):
    g = torch.Generator().manual_seed(n * c)
    x = torch.randn(n, c, 2, 2, generator=g).cuda().contiguous(memory_format=torch.channels_last).requires_grad_()
    lin, y = torch.nn.Linear(c, 10).cuda(), torch.randint(0, 10, (n,), generator=g).cuda()
    loss, _, metrics = head.head_loss(x, lin, y)
    got = torch.autograd.grad(loss, [x, lin.weight, lin.bias])
    assert torch.equal(loss.detach(), metrics[0])
    xr, wr, br = x.detach().double().requires_grad_(), lin.weight.detach().double().requires_grad_(), lin.bias.detach().double().requires_grad_()
    want = torch.autograd.grad(F.cross_entropy(F.linear(xr.mean((2, 3)), wr, br), y), [xr, wr, br])
    for a, b in zip(got, want):      # sums of up to 512 fp32 products, exponentials to 2 ulp: 1e-5 of the largest
        assert float((a.double() - b).abs().max()) <= 1e-5 * float(b.abs().max())
