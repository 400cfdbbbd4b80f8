"""Batch norm in one launch per direction against plain PyTorch in fp32."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

# rows per block below, at and above the lanes of a block; one block per channel group; more groups than runs; a ragged last run
SHAPES = [(1, 32, 2, 2), (2, 32, 8, 16), (3, 64, 16, 16), (5, 96, 10, 14), (128, 2048, 2, 2), (31, 512, 4, 4), (7, 4096, 4, 2), (64, 64, 32, 32),
          (400, 32, 32, 32)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", ["relu", "residual", "plain", "pool"])
@pytest.mark.parametrize("partials", [False, True])
def test_one_launch_forward_and_backward(shape, kind, partials):
    from gradient_compression_b200.ops import bn as B

    n, c, h, w = shape
    pool, relu, m = kind == "pool", kind != "plain", n * h * w
    if not B.fused_ok(m // 4 if pool else m, c):
        pytest.skip("more channel groups than blocks")
    gen = torch.Generator(device="cuda").manual_seed(n + c)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    x = (rand(n, c, h, w) * 2 + rand(1, c, 1, 1) * 3).contiguous(memory_format=torch.channels_last)
    gamma, beta, rm, rv = rand(c), rand(c), rand(c), rand(c).abs()
    res = rand(n, c, h, w).contiguous(memory_format=torch.channels_last) if kind == "residual" else None
    parts = None
    if partials:                    # what a convolution kernel leaves: sums and sums of squares of runs of rows
        rows = x.permute(0, 2, 3, 1).reshape(m, c)
        cut = [rows[i::5] for i in range(5) if i < m]
        parts = torch.stack([torch.stack([t.sum(0), t.square().sum(0)]) for t in cut]).contiguous()
    stats, y = torch.empty(2 * c, device="cuda"), torch.empty_like(x[:, :, ::2, ::2] if pool else x, memory_format=torch.channels_last)
    rm2, rv2 = rm.clone(), rv.clone()
    B.fused_forward(x, pool, parts, gamma, beta, res, relu, rm2, rv2, 0.1, 1e-5, stats, y)

    xr = x.double().requires_grad_()
    g, b = gamma.double().requires_grad_(), beta.double().requires_grad_()
    rr = res.double().requires_grad_() if res is not None else None
    rmr, rvr = rm.double(), rv.double()
    out = F.batch_norm(xr, rmr, rvr, g, b, True, 0.1, 1e-5) if m > 1 else None
    out = out + rr if rr is not None else out
    out = F.relu(out) if relu else out
    out = F.max_pool2d(out, 2, 2) if pool else out
    torch.testing.assert_close(y.double(), out.detach(), rtol=2e-5, atol=2e-5)
    torch.testing.assert_close(rm2.double(), rmr, rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(rv2.double(), rvr, rtol=1e-4, atol=1e-5)

    dy = rand(*y.shape).contiguous(memory_format=torch.channels_last)
    sums, dx = torch.empty(2 * c, device="cuda"), torch.empty_like(x)
    dres = torch.empty_like(x) if res is not None else None
    B.fused_backward(dy, x, y if res is not None else None, pool, stats, gamma, beta, relu, sums, dx, dres)
    # masks and window winners are found from fp32 values: where the reference decides otherwise on rounding noise, one channel moves
    out.backward(dy.double())

    def off(got, want, tol):
        return ((got.double() - want).abs() > tol * float(want.abs().max())).double().mean()

    assert off(dx, xr.grad, 1e-4) < 3e-3
    assert off(sums[:c], b.grad, 1e-4) <= max(3e-3, 1.0 / c) and off(sums[c:], g.grad, 1e-4) <= max(3e-3, 1.0 / c)
    if dres is not None:
        assert off(dres, rr.grad, 1e-6) < 1e-4


@pytest.mark.parametrize("kind", ["relu", "residual", "plain", "pool"])
@pytest.mark.parametrize("rows", [7, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1025])
def test_rows_of_a_thread(rows, kind):
    """One, two and three rows per thread of the fullest block, threads without a row: the backward keeps up to two rows (one pooled one), the forward's first
    four are loaded in front of the statistics.  (Not two rows in all: normalised they are 1 and -1 whatever x is, and the gradient is what eps / variance, some
    1e-5, leaves of terms that cancel: no more than a digit above their rounding.)"""
    test_one_launch_forward_and_backward((1, 64, 2, 2 * rows) if kind == "pool" else (1, 64, 1, rows), kind, True)
