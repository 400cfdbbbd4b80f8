"""Fused batch-norm (+ residual add) (+ ReLU) for channels-last fp32 activations.

``bn_act(bn_module, x, residual=None, relu=True)`` computes ``relu(bn(x) + residual)`` -- the pattern
of every block of the zoo (reference: models/resnet.py:71-75, models/vgg.py:105-106) -- with the
kernels of ``csrc/gc_bn.cu`` on CUDA and with the equivalent torch ops on CPU.  The module stays a plain
``torch.nn.BatchNorm2d`` (same parameters, buffers and ``state_dict`` keys); only the arithmetic moves.
"""
from __future__ import annotations

import os
import weakref

import torch
import torch.nn.functional as F

from . import _native as nat

# Hooks registered for every module of the process (profilers, module trackers).
_PRE, _FORWARD, _BACKWARD_PRE, _BACKWARD = (getattr(torch.nn.modules.module, n) for n in (
    "_global_forward_pre_hooks", "_global_forward_hooks", "_global_backward_pre_hooks", "_global_backward_hooks"))


def hooked(a, b=None):
    """Whether calling the module ``a`` (or ``b``) runs more than its forward.  The kernels take a layer's parameters without calling
    it, so a layer with hooks is called as the module it is: pruning and the weight normalisations recompute the weight in one."""
    d, e = a.__dict__, (a if b is None else b).__dict__            # (a third of the time of as many attributes)
    return bool(d["_forward_pre_hooks"] or d["_forward_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"] or
                e["_forward_pre_hooks"] or e["_forward_hooks"] or e["_backward_hooks"] or e["_backward_pre_hooks"] or
                _PRE or _FORWARD or _BACKWARD_PRE or _BACKWARD)


# Gradient tensors this library allocated itself and handed to autograd for a residual input: nobody else holds
# them, so a later kernel may accumulate into them in place (``ops.conv.GradLink``).  Keyed by address, checked by
# object identity through a weak reference, so a freed and re-used address never matches.
_owned_grads = {}


# ``num_batches_tracked`` of the batch norms of a model that called ``defer_batch_counters``: incremented together by
# one multi-tensor launch when the model's forward returns, instead of one tiny launch per layer (53 for ResNet-50).
_pending_counters = {}


def count_batch(bn):
    t = bn.num_batches_tracked
    if getattr(bn, "_gcb200_deferred_counter", False) and t.is_cuda:
        e = _pending_counters.get(id(t))
        if e is None:
            _pending_counters[id(t)] = [t, 1]
        else:
            e[1] += 1
        if len(_pending_counters) > 4096:
            flush_batch_counters()
    else:
        t.add_(1)


def flush_batch_counters():
    if _pending_counters:
        entries = list(_pending_counters.values())
        _pending_counters.clear()
        if all(n == 1 for _, n in entries):
            torch._foreach_add_([t for t, _ in entries], 1)
        else:
            for t, n in entries:
                t.add_(n)


def _flush_hook(module, inputs, output):
    flush_batch_counters()


def defer_batch_counters(model):
    """Batch the ``num_batches_tracked`` increments of every batch norm under ``model`` into one launch at the end of
    ``model``'s forward."""
    for m in model.modules():
        if isinstance(m, torch.nn.modules.batchnorm._BatchNorm):
            m._gcb200_deferred_counter = True
    model.register_forward_hook(_flush_hook)
    return model


def own_grad(t):
    if len(_owned_grads) >= 256:
        for k in [k for k, r in _owned_grads.items() if r() is None]:
            del _owned_grads[k]
        if len(_owned_grads) >= 256:
            _owned_grads.clear()
    _owned_grads[t.data_ptr()] = weakref.ref(t)
    return t


def take_owned_grad(t):
    """True exactly once for a tensor registered with ``own_grad``."""
    r = _owned_grads.pop(t.data_ptr(), None)
    return r is not None and r() is t

_scratch = {}
# One launch per direction (csrc/gc_bn_fused.cu) where the channels come in groups of 32; off: separate reduction, finalize and apply.
FUSED = os.environ.get("GCB200_BN_FUSED", "1") == "1"
_fused_scratch = {}
FUSED_BWD_FINALIZE = os.environ.get("GCB200_BN_FUSED_BWD_FINALIZE", "0") == "1"


def _scratch_for(device, channels):
    key = (device.type, device.index)
    cur = _scratch.get(key)
    need = nat.cuda().gc_cuda_bn_scratch_bytes(int(channels))
    if cur is None or cur.numel() < need:
        cur = torch.empty(max(need, nat.cuda().gc_cuda_bn_scratch_bytes(2048)), dtype=torch.uint8, device=device)
        _scratch[key] = cur
    return cur


def fused_scratch(device):
    """Barrier counts and partial sums of the one-launch kernels: zeroed once, every launch leaves them ready for the next."""
    key = (device.type, device.index)
    cur = _fused_scratch.get(key)
    if cur is None:
        cur = _fused_scratch[key] = torch.zeros(nat.cuda().gc_cuda_bn_fused_scratch_bytes(), dtype=torch.uint8, device=device)
    return cur


def fused_ok(m, c):
    return FUSED and bool(nat.cuda().gc_cuda_bn_fused_supported(m, c))


def fused_forward(x, pool, partials, gamma, beta, residual, relu, running_mean, running_var, momentum, eps, stats, y):
    """Statistics (from the convolution's partial sums when given), running statistics and apply of ``x`` [N, C, H, W]."""
    from . import gemm

    n, c, h, w = x.shape
    nat.check(nat.cuda().gc_cuda_bn_fused_forward(
        x.data_ptr(), n, h, w, c, int(pool), nat.ptr(partials), partials.shape[0] if partials is not None else 0, gamma.data_ptr(), beta.data_ptr(),
        nat.ptr(residual), int(relu), nat.ptr(running_mean), nat.ptr(running_var), float(momentum), float(eps), stats.data_ptr(), y.data_ptr(),
        fused_scratch(x.device).data_ptr(), gemm._error_flag(x.device).data_ptr(), nat.stream_ptr()), "bn_fused_forward")


def fused_backward(dy, x, y, pool, stats, gamma, beta, relu, sums, dx, dres):
    from . import gemm

    n, c, h, w = x.shape
    nat.check(nat.cuda().gc_cuda_bn_fused_backward(
        dy.data_ptr(), x.data_ptr(), nat.ptr(y), n, h, w, c, int(pool), stats.data_ptr(), gamma.data_ptr(), beta.data_ptr(), int(relu), sums.data_ptr(),
        dx.data_ptr(), nat.ptr(dres), fused_scratch(x.device).data_ptr(), gemm._error_flag(x.device).data_ptr(), nat.stream_ptr()), "bn_fused_backward")


def _fin_ptr(device, channels):
    """Scratch that lets the backward reduction finish its sums inside its own launch (None: separate finalize)."""
    from . import gemm

    if not FUSED_BWD_FINALIZE or channels > gemm.FIN_MAX_CHANNELS:
        return None
    return gemm.fin_scratch(device).data_ptr()


def _cl(t):
    """``t`` in channels-last memory order, starting on a 16-byte boundary (the kernels read quads of channels)."""
    if not t.is_contiguous(memory_format=torch.channels_last):
        return t.contiguous(memory_format=torch.channels_last)
    return t if t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.channels_last)


def on_boundary(p):
    """The tensor ``p``, or a copy that autograd leads back to it, on a 16-byte boundary.  Parameters of a flat buffer (``FlatArena`` packs
    them back to back) need not start on one: behind a tensor whose size is no multiple of four none of them do."""
    return p if p.data_ptr() % 16 == 0 else p.clone(memory_format=torch.preserve_format)


def kernel_path_ok(x):
    if not (x.is_cuda and x.dtype == torch.float32 and x.dim() == 4):
        return False
    n, c, h, w = x.shape
    return bool(nat.cuda().gc_cuda_bn_supported(n * h * w, c))


class _FusedBNAct(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias, residual, running_mean, running_var, training, momentum, eps, relu):
        x = _cl(x)
        n, c, h, w = x.shape
        m = n * h * w
        lib, st = nat.cuda(), nat.stream_ptr()
        stats = torch.empty(2 * c, dtype=torch.float32, device=x.device)
        with torch.cuda.device(x.device):
            if training and fused_ok(m, c):
                y = torch.empty_like(x)
                fused_forward(x, False, None, weight, bias, _cl(residual) if residual is not None else None, relu, running_mean, running_var, momentum,
                              eps, stats, y)
                ctx.relu, ctx.has_res, ctx.training = bool(relu), residual is not None, True
                ctx.save_for_backward(x, weight, bias, stats, y if (residual is not None and relu) else None)
                return y
            if training:
                nat.check(lib.gc_cuda_bn_stats(x.data_ptr(), m, c, _scratch_for(x.device, c).data_ptr(), stats.data_ptr(),
                                               nat.ptr(running_mean), nat.ptr(running_var), float(momentum), float(eps),
                                               st), "bn_stats")
                nat.count_launch()
            else:
                stats[:c] = running_mean
                stats[c:] = torch.rsqrt(running_var + eps)
            res = _cl(residual) if residual is not None else None
            y = torch.empty_like(x)
            nat.check(lib.gc_cuda_bn_apply(x.data_ptr(), m, c, stats.data_ptr(), weight.data_ptr(), bias.data_ptr(),
                                           nat.ptr(res), int(relu), y.data_ptr(), st), "bn_apply")
        ctx.relu, ctx.has_res, ctx.training = bool(relu), residual is not None, bool(training)
        ctx.save_for_backward(x, weight, bias, stats, y if (residual is not None and relu) else None)
        return y

    @staticmethod
    def backward(ctx, dy):
        x, weight, bias, stats, y = ctx.saved_tensors
        dy = _cl(dy)
        n, c, h, w = x.shape
        m = n * h * w
        lib, st = nat.cuda(), nat.stream_ptr()
        if not ctx.training:
            raise RuntimeError("bn_act: backward through eval-mode statistics is not supported by the fused kernel")
        sums = torch.empty(2 * c, dtype=torch.float32, device=x.device)
        dx = torch.empty_like(x)
        dres = own_grad(torch.empty_like(x)) if (ctx.has_res and ctx.needs_input_grad[3]) else None
        if fused_ok(m, c):
            with torch.cuda.device(x.device):
                fused_backward(dy, x, y, False, stats, weight, bias, ctx.relu, sums, dx, dres)
            if ctx.has_res and dres is None and ctx.needs_input_grad[3]:
                dres = dy
            return dx, sums[c:], sums[:c], dres, None, None, None, None, None, None
        with torch.cuda.device(x.device):
            nat.check(lib.gc_cuda_bn_bwd_reduce(dy.data_ptr(), x.data_ptr(), nat.ptr(y), m, c, stats.data_ptr(),
                                                weight.data_ptr(), bias.data_ptr(), int(ctx.relu),
                                                _scratch_for(x.device, c).data_ptr(), sums.data_ptr(), _fin_ptr(x.device, c), st),
                      "bn_bwd_reduce")
            nat.count_launch()
            nat.check(lib.gc_cuda_bn_bwd_apply(dy.data_ptr(), x.data_ptr(), nat.ptr(y), m, c, stats.data_ptr(),
                                               weight.data_ptr(), bias.data_ptr(), sums.data_ptr(), int(ctx.relu),
                                               dx.data_ptr(), nat.ptr(dres), st), "bn_bwd_apply")
        if ctx.has_res and dres is None and ctx.needs_input_grad[3]:
            dres = dy
        return dx, sums[c:], sums[:c], dres, None, None, None, None, None, None


def _by_torch(bn, x):
    """``bn(x)``.  The library's channels-last kernels read quads too (its training batch norm raised a misaligned address on an activation
    between two boundaries), so it gets copies where ours would."""
    if x.is_cuda:
        x = on_boundary(x)
        moved = {n: on_boundary(p) for n, p in bn._parameters.items() if p is not None and p.data_ptr() % 16}
        if moved:
            return torch.func.functional_call(bn, moved, (x,))
    return bn(x)


def bn_act(bn, x, residual=None, relu=True):
    """``relu(bn(x) + residual)`` with ``bn`` a ``torch.nn.BatchNorm2d`` (affine, tracking running stats)."""
    training = bn.training or bn.running_mean is None
    plain = bn.affine and not hooked(bn)
    if not training and x.is_cuda and plain and not torch.is_grad_enabled():
        y = nat.ext().bn_eval(x, bn.weight, bn.bias, bn.running_mean, bn.running_var, bn.eps, residual, relu)
        if y is not None:
            nat.count_launch()
            return y
    use_kernel = plain and kernel_path_ok(x) and not (not training and torch.is_grad_enabled() and x.requires_grad)
    if not use_kernel:
        y = _by_torch(bn, x)
        if residual is not None:
            y = y + residual
        return F.relu(y) if relu else y
    momentum = 0.1 if bn.momentum is None else bn.momentum
    if training and bn.track_running_stats and bn.num_batches_tracked is not None:
        count_batch(bn)
    rm = bn.running_mean if bn.track_running_stats else None
    rv = bn.running_var if bn.track_running_stats else None
    return _FusedBNAct.apply(x, on_boundary(bn.weight), on_boundary(bn.bias), residual, rm, rv, training, momentum, bn.eps, relu)
