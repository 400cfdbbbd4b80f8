"""Inference head (pooling + linear) and batch metrics of logits against torch."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c,hw,k,bias", [(1, 4, 1, 1, True), (33, 512, 1, 10, True), (7, 516, 4, 32, False), (300, 2048, 4, 10, True), (5, 4096, 2, 5, True)])
def test_classify(n, c, hw, k, bias):
    from gradient_compression_b200.models.layers import head
    from gradient_compression_b200.ops.head import classify

    g = torch.Generator(device="cuda").manual_seed(n + c)
    x = torch.randn(n, c, hw, hw, device="cuda", generator=g).contiguous(memory_format=torch.channels_last)
    linear = torch.nn.Linear(c, k, bias=bias).cuda()
    assert classify(x, linear) is None                      # a gradient may be wanted
    with torch.no_grad():
        y = classify(x, linear)
        ref = F.linear(x.double().mean((2, 3)), linear.weight.double(), linear.bias.double() if bias else None)
        assert y.is_contiguous() and torch.allclose(y.double(), ref, rtol=1e-5, atol=1e-5)
        assert torch.equal(head(x, hw, linear), y)
        wide = torch.nn.Linear(c, 40).cuda()                # more classes than the kernel takes
        assert classify(x, wide) is None and head(x, hw, wide).shape == (n, 40)


@pytest.mark.parametrize("n,k", [(1, 5), (31, 10), (257, 10), (1500, 100), (70, 1024)])
def test_logit_metrics(n, k):
    from gradient_compression_b200.ops.head import logit_metrics

    g = torch.Generator(device="cuda").manual_seed(n + k)
    z = torch.randn(n, k, device="cuda", generator=g) * 5
    labels = torch.randint(0, k, (n,), device="cuda", generator=g)
    for ignore in (0, n // 3):
        labels[:ignore] = -100
        ce, top1, top5 = logit_metrics(z, labels)
        hit = z.topk(5, 1, True, True)[1].eq(labels.view(-1, 1))
        assert torch.allclose(ce.double(), F.cross_entropy(z.double(), labels), rtol=1e-6)
        assert float(top1) == float(hit[:, 0].float().sum() / n) and float(top5) == float(hit.float().sum() / n)
    labels[-1] = 0
    z[-1, 1] = float("nan")
    assert torch.isnan(logit_metrics(z, labels)[0])
    assert logit_metrics(z[:, :4].contiguous(), labels) is None and logit_metrics(z.half(), labels) is None


@pytest.mark.parametrize("name", ["ResNet18", "VGG11"])
@pytest.mark.parametrize("what", ["forward hook", "pruned"])
def test_a_classifier_with_hooks_is_called(name, what):
    import torch.nn.utils.prune as prune

    from gradient_compression_b200 import models

    torch.manual_seed(2)
    model = getattr(models, name)().cuda().to(memory_format=torch.channels_last)
    linear = model.linear if name == "ResNet18" else model.classifier
    x, labels, seen = torch.randn(6, 3, 32, 32, device="cuda").contiguous(memory_format=torch.channels_last), torch.arange(6, device="cuda"), []
    with torch.no_grad():
        model(x)
        plain = model.eval()(x)
    if what == "pruned":
        prune.custom_from_mask(linear, "weight", torch.ones_like(linear.weight))
        with torch.no_grad():
            linear.weight_orig.mul_(2.0)
    else:
        linear.register_forward_hook(lambda m, i, o: seen.append(m) or 2.0 * o)
    with torch.no_grad():
        got = model(x)
        want = 2.0 * plain - (linear.bias if what == "pruned" else 0.0)
    assert torch.allclose(got, want, rtol=1e-4, atol=1e-4 * float(want.abs().max()))
    assert seen == [linear] * (what != "pruned")
    loss, logits, _ = model.train().forward_loss(x, labels)
    loss.backward()
    assert torch.isfinite(loss) and (len(seen) == 2 if what == "forward hook" else float(linear.weight_orig.grad.abs().max()) > 0)


@pytest.mark.parametrize("n,k,kernel", [(1, 5, True), (20000, 10, True), (4096, 16, True), (4097, 16, False), (1024, 64, True), (1025, 64, False),
                                        (256, 256, True), (257, 256, False), (16, 257, False), (30, 1000, False)])
def test_metrics_of_a_batch_on_both_sides_of_the_line(n, k, kernel):
    from gradient_compression_b200.ops import _native as nat
    from gradient_compression_b200.train import CIFAR

    task = CIFAR("cuda", None, "LeNet", data="synthetic", synthetic_train_size=1, synthetic_test_size=1)
    g = torch.Generator(device="cuda").manual_seed(n + k)
    z, labels = torch.randn(n, k, device="cuda", generator=g) * 3, torch.randint(0, k, (n,), device="cuda", generator=g)
    before = nat.launches()
    got = task.evaluate_predictions(z, labels)
    assert nat.launches() - before == kernel
    hit = z.topk(5, 1, True, True)[1].eq(labels.view(-1, 1))
    assert torch.allclose(got["cross_entropy_loss"].double(), F.cross_entropy(z.double(), labels), rtol=1e-6)
    assert float(got["top1_accuracy"]) == float(hit[:, 0].float().sum() / n) and float(got["top5_accuracy"]) == float(hit.float().sum() / n)
