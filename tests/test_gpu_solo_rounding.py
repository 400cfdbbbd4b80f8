"""Second pass of the single-worker QSGD reduces, bit for bit against the CPU: levels at and around integers, elements of the norm's own size,
poisoned and subnormal gradients on vectors that fit the chip's shared memory and on longer ones, every relation between the two scales."""
import pytest
import torch

from gradient_compression_b200 import make_reducer

pytestmark = pytest.mark.gpu

CONFIGS = [("QSGDMaxNormReducer", {"quantization_level": 1}), ("QSGDMaxNormReducer", {"quantization_level": 8}), ("QSGDMaxNormReducer", {"quantization_level": 16}),
           ("QSGDMaxNormTwoScaleReducer", {"quantization_level": 2, "higher_quantization_level": 6}),
           ("QSGDMaxNormTwoScaleReducer", {"quantization_level": 6, "higher_quantization_level": 10}),
           ("QSGDMaxNormTwoScaleReducer", {"quantization_level": 6, "higher_quantization_level": 6})]
RANDK = [("GlobalRandKMaxNormReducer", {"K": 3000, "quantization_level": 8}),
         ("GlobalRandKMaxNormTwoScaleReducer", {"K": 3000, "quantization_level": 6, "higher_quantization_level": 10})]
NAN = float("nan")


def compare(name, config, host):
    cpu, gpu = (make_reducer(name, d, None, dict(config, seed=5)) for d in ("cpu", "cuda"))
    for _ in range(2):
        want, got = [torch.empty_like(t) for t in host], [torch.empty_like(t).cuda() for t in host]
        cpu.reduce([t.clone() for t in host], want)
        gpu.reduce([t.cuda() for t in host], got)
        for w, g in zip(want, got):
            # the same bits, NaN as NaN
            assert torch.equal(torch.nan_to_num(w, nan=7.0).view(torch.int32), torch.nan_to_num(g.cpu(), nan=7.0).view(torch.int32))


@pytest.mark.parametrize("n", [4096 * 3 + 5, 148 * 4096 * 14 + 9])
@pytest.mark.parametrize("name,config", CONFIGS)
def test_around_levels(name, config, n):
    gen = torch.Generator().manual_seed(n)
    s = 2 ** config.get("higher_quantization_level", config["quantization_level"]) - 1
    norm = 0.7310586
    k = torch.randint(0, s + 1, (n,), generator=gen).float()
    off = torch.randint(-2, 3, (n,), generator=gen)              # a few units in the last place away from a level
    x = k * (norm / s)
    x = (x.view(torch.int32) + off.where(x > 0, torch.zeros_like(off)).int()).view(torch.float32).clamp(max=norm)
    x = torch.where(torch.rand(n, generator=gen) < 0.5, x, -x)
    x[1::5] = torch.randn(x[1::5].numel(), generator=gen) * 1e-3
    x[2] = -norm
    compare(name, config, [x])


@pytest.mark.parametrize("value", [0.0, NAN, -NAN, float("inf"), -float("inf"), 1e-36, 3e-39, 1e-44])
@pytest.mark.parametrize("name,config", CONFIGS[1:2] + CONFIGS[3:])
def test_special_values(name, config, value):
    small = [torch.full((6,), value), torch.tensor([-1e-3, 0.5, value, -0.25, -value])]
    compare(name, config, small)
    if value != value or abs(value) < 1e-30 or value in (float("inf"), -float("inf")):
        long = torch.randn(148 * 4096 * 14 + 3, generator=torch.Generator().manual_seed(2)) * (1e-37 if abs(value) < 1e-30 else 1.0)
        long[::100003] = value
        compare(name, config, [long])


@pytest.mark.parametrize("n", [4096 * 3 + 5, 148 * 4096 * 14 + 9])
@pytest.mark.parametrize("norm", [1e-34, 1e-36, 1e-37, 1e-44])
@pytest.mark.parametrize("name,config", CONFIGS + RANDK)
def test_zeros_of_both_signs_at_tiny_norms(name, config, norm, n):
    """Where levels / norm overflows, zero times infinity is given the last level, and the sign of a zero does not count; where the value of a level
    underflows to zero (1e-44 and more than thirteen levels), negative elements become -0.0."""
    x = torch.rand(n, generator=torch.Generator().manual_seed(n)) * (2 * norm) - norm
    x[::7], x[3::7], x[1] = 0.0, -0.0, -norm
    compare(name, config, [x])


@pytest.mark.parametrize("sizes", [[1], [4095], [4097], [8193], [12288], [16383], [16384], [16385], [1, 4090, 3, 4000], [5, 0, 7], [4096, 1, 2, 3], [1, 4097, 1, 2]])
@pytest.mark.parametrize("name,config", CONFIGS)
def test_one_block(name, config, sizes):
    """Up to four tiles of 4096 elements have a kernel of their own; a tensor that starts inside a tile begins another."""
    gen = torch.Generator().manual_seed(sum(sizes))
    compare(name, config, [torch.randn(n, generator=gen) for n in sizes])
