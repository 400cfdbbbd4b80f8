"""Inference layers (convolution, batch norm of running statistics, residual, ReLU, pool in one go) against PyTorch in fp64."""
import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

#          n, cin, h, cout, r, stride, pad
LAYERS = [(3, 3, 32, 64, 3, 1, 1),           # stem
          (1, 64, 8, 64, 1, 1, 0), (5, 64, 16, 256, 1, 1, 0), (2, 36, 8, 100, 1, 1, 0), (1, 20, 4, 36, 1, 1, 0),
          (2, 64, 32, 64, 3, 1, 1), (3, 128, 16, 256, 3, 2, 1), (1, 256, 8, 512, 1, 2, 0),
          (2, 512, 4, 512, 3, 1, 1),         # few tiles, long contraction: split over the SMs
          (130, 64, 2, 96, 3, 1, 1),
          (2, 32, 6, 32, 3, 1, 1)]           # a map the tilings exclude


@pytest.mark.parametrize("layer", LAYERS)
@pytest.mark.parametrize("kind", ["relu", "residual", "plain", "bias", "pool"])
def test_layer(layer, kind):
    from gradient_compression_b200.ops import conv_bn_act

    n, cin, h, cout, r, stride, pad = layer
    torch.manual_seed(cout + r)
    conv = nn.Conv2d(cin, cout, r, stride, pad, bias=kind == "bias").cuda().to(memory_format=torch.channels_last)
    bn = nn.BatchNorm2d(cout).cuda().eval()
    with torch.no_grad():
        for t in (bn.weight, bn.bias, bn.running_mean):
            t.normal_()
        bn.running_var.uniform_(0.3, 3.0)
        x = torch.randn(n, cin, h, h, device="cuda").contiguous(memory_format=torch.channels_last)
        ho = (h + 2 * pad - r) // stride + 1
        res = torch.randn(n, cout, ho, ho, device="cuda").contiguous(memory_format=torch.channels_last) if kind == "residual" else None
        got = conv_bn_act(conv, bn, x, residual=res, relu=kind != "plain", pool=kind == "pool")
        want = F.conv2d(x.double(), conv.weight.double(), conv.bias.double() if conv.bias is not None else None, stride, pad)
        want = F.batch_norm(want, bn.running_mean.double(), bn.running_var.double(), bn.weight.double(), bn.bias.double(), False, 0.0, bn.eps)
        want = want + res.double() if res is not None else want
        want = F.relu(want) if kind != "plain" else want
        want = F.max_pool2d(want, 2, 2) if kind == "pool" else want
        assert got.shape == want.shape and got.is_contiguous(memory_format=torch.channels_last)
        err = (got.double() - want).abs()
        assert float(err.max()) < 0.03 * float(want.abs().max()) and float(err.norm() / want.norm()) < 2e-3


@pytest.mark.parametrize("name", ["ResNet18", "ResNet50", "VGG11", "MobileNetV2", "densenet_cifar"])
def test_model_matches_the_layers_one_by_one(name):
    from gradient_compression_b200 import models
    from gradient_compression_b200.ops import _native as nat

    torch.manual_seed(1)
    model = getattr(models, name)().cuda().to(memory_format=torch.channels_last)
    x = torch.randn(20, 3, 32, 32, device="cuda").contiguous(memory_format=torch.channels_last)
    with torch.no_grad():
        model(x)
        model.eval()
        got, before = model(x), nat.launches()
        # layers with hooks are called as the torch modules they are: cuDNN convolutions, torch batch norms and classifier
        handles = [m.register_forward_hook(lambda *_: None) for m in model.modules() if isinstance(m, (nn.Conv2d, nn.BatchNorm2d, nn.Linear))]
        want = model(x)
        assert nat.launches() == before
        for h in handles:
            h.remove()
        model(x)
        assert (nat.launches() > before) == (name != "densenet_cifar")        # (none of its widths divides a block of the kernels)
    assert float((got - want).norm() / want.norm()) < 2e-2


def _layer(cin=64, cout=64, r=3):
    torch.manual_seed(3)
    conv = nn.Conv2d(cin, cout, r, 1, r // 2).cuda().to(memory_format=torch.channels_last)
    bn = nn.BatchNorm2d(cout).cuda().eval()
    with torch.no_grad():
        bn.weight.normal_()
        bn.running_var.uniform_(0.3, 3.0)
    return conv, bn, torch.randn(4, cin, 8, 8, device="cuda").contiguous(memory_format=torch.channels_last)


def _want(conv_w, conv_b, bn, bn_w, x):
    y = F.conv2d(x.double(), conv_w.double(), conv_b.double(), 1, conv_w.shape[2] // 2)
    return F.relu(F.batch_norm(y, bn.running_mean.double(), bn.running_var.double(), bn_w.double(), bn.bias.double(), False, 0.0, bn.eps))


@pytest.mark.filterwarnings("ignore:.*weight_norm.*")
@pytest.mark.parametrize("r", [1, 3])
@pytest.mark.parametrize("how", ["conv weight pruned", "conv bias pruned", "bn weight pruned", "weight_norm"])
def test_computed_parameters(how, r):
    """Layers whose weight is computed from another parameter: not registered under its own name any more."""
    import torch.nn.utils as U
    import torch.nn.utils.prune as prune

    from gradient_compression_b200.ops import conv_bn_act

    conv, bn, x = _layer(r=r)
    if how == "weight_norm":
        U.weight_norm(conv)
    else:
        module, name = bn if "bn" in how else conv, "bias" if "bias" in how else "weight"
        prune.custom_from_mask(module, name, (torch.rand_like(getattr(module, name)) < 0.5).float())
    with torch.no_grad():
        got = conv_bn_act(conv, bn, x)
        want = _want(conv.weight, conv.bias, bn, bn.weight, x)
    assert float((got.double() - want).norm() / want.norm()) < 2e-3


@pytest.mark.filterwarnings("ignore:.*weight_norm.*")
@pytest.mark.parametrize("training", [False, True])
@pytest.mark.parametrize("how", ["conv pruned", "bn pruned", "weight_norm", "spectral_norm"])
def test_recomputed_weights(how, training):
    """The weight is recomputed from what it is made of at every call, in inference and in training (two steps)."""
    import torch.nn.utils as U
    import torch.nn.utils.prune as prune

    from gradient_compression_b200.ops import conv_bn_act

    conv, bn, x = _layer()
    if "pruned" in how:
        prune.custom_from_mask(bn if "bn" in how else conv, "weight", (torch.rand_like((bn if "bn" in how else conv).weight) < 0.5).float())
    else:
        getattr(U, how)(conv)
    conv.train(training), bn.train(training)
    for _ in range(2):
        with torch.set_grad_enabled(training):
            got = conv_bn_act(conv, bn, x)
        with torch.no_grad():
            y = F.conv2d(x.double(), conv.weight.double(), conv.bias.double(), 1, 1)        # the weight of that call
            y = F.batch_norm(y, bn.running_mean.double(), bn.running_var.double(), bn.weight.double(), bn.bias.double(), training, 0.0, bn.eps)
            want = F.relu(y)
        assert float((got.detach().double() - want).norm() / want.norm()) < 2e-3
        changed = [p for n, p in list(conv.named_parameters()) + list(bn.named_parameters()) if n in ("weight_orig", "weight_g")]
        if training:
            got.square().sum().backward()
            assert changed and all(p.grad is not None and float(p.grad.abs().max()) > 0 for p in changed)
            conv.zero_grad(), bn.zero_grad()
        with torch.no_grad():
            for p in changed:
                p.mul_(1.5)


@pytest.mark.parametrize("training", [False, True])
@pytest.mark.parametrize("kind", ["forward", "pre", "backward", "global"])
def test_hooks_run(kind, training):
    from gradient_compression_b200.ops import conv_bn_act

    conv, bn, x = _layer()
    bn.train(training)
    seen = []
    with torch.set_grad_enabled(training):
        plain = conv_bn_act(conv, bn, x)
        if kind == "global":
            handles = [nn.modules.module.register_module_forward_hook(lambda m, i, o: seen.append(m))]
        else:
            add = {"forward": "register_forward_hook", "pre": "register_forward_pre_hook", "backward": "register_full_backward_hook"}[kind]
            handles = [getattr(m, add)(lambda m, *_: seen.append(m)) for m in (conv, bn)]
        got = conv_bn_act(conv, bn, x)
        if training:
            got.sum().backward()
        for h in handles:
            h.remove()
        again = conv_bn_act(conv, bn, x)
    assert set(seen) == (set() if kind == "backward" and not training else {conv, bn})
    got, plain, again = got.detach(), plain.detach(), again.detach()
    assert float((got - plain).norm() / plain.norm()) < 2e-3 and torch.equal(again, plain)


@pytest.mark.parametrize("training", [False, True])
@pytest.mark.parametrize("mode,cin,r,stride", [("gemm", 64, 1, 1), ("conv", 64, 3, 1), ("conv", 64, 1, 2), ("stem", 3, 3, 1)])
def test_switches_act_in_inference_as_in_training(mode, cin, r, stride, training, monkeypatch):
    from gradient_compression_b200.ops import conv as C

    torch.manual_seed(4)
    conv = nn.Conv2d(cin, 64, r, stride, r // 2).cuda().to(memory_format=torch.channels_last).train(training)
    bn = nn.BatchNorm2d(64).cuda().train(training)
    x = torch.randn(2, cin, 8, 8, device="cuda").contiguous(memory_format=torch.channels_last)
    rows, calls, forward = 2 * (8 // stride) ** 2, [], nn.Conv2d.forward
    monkeypatch.setattr(nn.Conv2d, "forward", lambda m, i: calls.append(1) or forward(m, i))        # only cuDNN calls the module

    def on_cudnn(**switches):
        with monkeypatch.context() as m, torch.set_grad_enabled(training):
            for k, v in switches.items():
                m.setattr(C, k, v)
            del calls[:]
            C.conv_bn_act(conv, bn, x)
        return bool(calls)

    every = {"gemm", "conv", "stem", "dgrad_s2"}
    assert not on_cudnn() and not on_cudnn(PATHS={mode}) and not on_cudnn(MIN_ROWS=rows)
    assert on_cudnn(PATHS=every - {mode}) and on_cudnn(MIN_ROWS=rows + 1) and on_cudnn(ENABLED=False)


@pytest.mark.parametrize("name", ["ResNet18", "MobileNetV2"])
@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("transform", ["forward AD", "vmap", "trace"])
def test_transforms_the_kernels_know_nothing_of_are_refused(name, transform):
    """No tangent dropped, no result baked into a graph: the layers' general path refuses these."""
    import torch.autograd.forward_ad as fwad

    from gradient_compression_b200 import models

    torch.manual_seed(1)
    model = getattr(models, name)().cuda().to(memory_format=torch.channels_last).eval()
    x = torch.randn(2, 3, 32, 32, device="cuda").contiguous(memory_format=torch.channels_last)
    with torch.no_grad(), pytest.raises((RuntimeError, TypeError)):        # (NotImplementedError is a RuntimeError)
        if transform == "forward AD":
            with fwad.dual_level():
                model(fwad.make_dual(x, torch.ones_like(x)))
        elif transform == "vmap":
            torch.func.vmap(model)(x[:, None])
        else:
            traced = torch.jit.trace(model, x, check_trace=False)
            other = torch.randn_like(x)
            assert float((traced(other) - model(other)).norm()) < 1e-3 * float(model(other).norm())
            raise RuntimeError("traced, and follows its input")
    with torch.no_grad():
        assert torch.isfinite(model(x)).all()
