"""Stride-2 filters whose parity classes have taps in front of their own pixel (4x4 with padding 1, 5x5 with padding 2) are not this library's: refused
at the C entry, and a layer's gradients are torch's."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from gradient_compression_b200.ops import conv  # noqa: E402


@pytest.mark.parametrize("r,pad,taken", [(1, 0, 1), (2, 0, 1), (3, 1, 1), (4, 1, 0), (5, 2, 0)])
def test_entry(r, pad, taken):
    assert conv.nat.cuda().gc_cuda_conv_dgrad_s2_supported(4, 16, 16, 64, 64, r, pad) == taken


def test_gradients_of_a_5x5_layer():
    torch.manual_seed(1)
    conv5 = torch.nn.Conv2d(64, 64, 5, 2, 2, bias=False).cuda().to(memory_format=torch.channels_last)
    bn = torch.nn.BatchNorm2d(64).cuda()
    x = torch.randn(32, 64, 16, 16, device="cuda").contiguous(memory_format=torch.channels_last).requires_grad_()
    dy = torch.randn(32, 64, 8, 8, device="cuda")
    got, = torch.autograd.grad(conv.conv_bn_act(conv5, bn, x), x, dy.contiguous(memory_format=torch.channels_last))
    want, = torch.autograd.grad(torch.relu(torch.nn.functional.batch_norm(torch.nn.functional.conv2d(x.double(), conv5.weight.double(), None, 2, 2), None, None, bn.weight.double(),
                                                                           bn.bias.double(), True, 0.1, bn.eps)), x, dy.double())
    # TF32 products (2^-11 relative) and ReLUs that switch at a rounded zero: a per cent; a missing row of taps is a quarter of the gradient
    assert (got.double() - want.double()).norm() / want.double().norm() < 0.05
