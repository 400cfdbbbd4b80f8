"""Launch plan of the one-launch batch norm on chips of any size (host arithmetic, no GPU)."""
import pytest


@pytest.mark.parametrize("sms", [1, 20, 74, 132, 147, 148, 149, 160, 264, 1000])
def test_blocks_fit_the_scratch_on_any_chip(sms):
    from gradient_compression_b200.ops import _native as nat

    lib = nat.cuda()
    room = lib.gc_cuda_bn_fused_scratch_bytes() // (2 * 4 + 64 * 4)          # per block two counts and 64 partial sums
    for c in (32, 64, 96, 160, 256, 1024, 2048, 4096, 4736, 4768, 8192):
        for m in (1, 255, 256, 257, 4096, 49999, 131072, 10 ** 8):
            blocks = lib.gc_cuda_bn_fused_blocks(m, c, sms)
            assert 0 <= blocks <= min(sms, room), (m, c, blocks)
            assert (blocks > 0) == (c // 32 <= min(sms, room))
            if blocks:
                groups = c // 32
                assert blocks == groups or (blocks % groups == 0 and blocks // groups * 256 <= m + 255)
    assert lib.gc_cuda_bn_fused_blocks(10 ** 6, 64, 148) == 148 and lib.gc_cuda_bn_fused_blocks(0, 64, 148) == lib.gc_cuda_bn_fused_blocks(64, 48, 148) == 0
