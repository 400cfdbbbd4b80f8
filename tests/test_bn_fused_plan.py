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


@pytest.mark.parametrize("sms", [1, 74, 148, 149, 1000])
def test_pooled_runs_have_a_row_for_every_lane(sms):
    """A row is a pooled one with its four pixels: runs of 128 rows, one per lane of a block, where blocks allow it."""
    from gradient_compression_b200.ops import _native as nat

    lib = nat.cuda()
    room = lib.gc_cuda_bn_fused_scratch_bytes() // (2 * 4 + 64 * 4)
    for c in (32, 64, 96, 256, 512, 4736, 4768):
        for m in (1, 127, 128, 129, 255, 256, 257, 2048, 7936, 32768, 10 ** 8):
            groups, blocks = c // 32, lib.gc_cuda_bn_fused_pool_blocks(m, c, sms)
            assert (blocks > 0) == (groups <= min(sms, room))
            if blocks:
                runs, most = blocks // groups, max(min(sms, room) // groups, 1)
                per = -(-m // min(most, -(-m // 128)))                       # rows a run, as few as blocks allow and 128 at least
                assert blocks % groups == 0 and runs == -(-m // per) <= most and runs * 128 < m + 128
    assert lib.gc_cuda_bn_fused_pool_blocks(128 * 148, 32, 148) == 148 and lib.gc_cuda_bn_fused_blocks(128 * 148, 32, 148) == 74
    assert lib.gc_cuda_bn_fused_pool_blocks(0, 64, 148) == lib.gc_cuda_bn_fused_pool_blocks(64, 48, 148) == 0
