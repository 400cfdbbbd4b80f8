"""Single-worker reducers on lists of tensors as they are: bit for bit what the same reducer computes on the CPU."""
import pytest
import torch

from gradient_compression_b200 import make_reducer

pytestmark = pytest.mark.gpu

TILE = 4096        # elements of one tile of the segment kernels

SIZES = {
    "one": [1], "tail": [5], "tile": [TILE], "tile+1": [TILE + 1], "one-block": [4 * TILE], "two-blocks": [4 * TILE + 1],
    "kept": [148 * TILE * 2 + 77], "re-read": [148 * TILE * 13 + 3],                        # beyond the tiles kept in shared memory
    "many": [64, 3, 4097, 1, 10, 127, 36864, 2, 8191, 512 * 10], "odd starts": [1, TILE, 2, TILE, 3, TILE, 4 * TILE + 1],
    "most": [7] * 320, "too many": [7] * 321,
}


def _values(sizes, seed):
    gen = torch.Generator().manual_seed(seed)
    return [torch.randn(n, generator=gen) * 10.0 ** (-(i % 3)) for i, n in enumerate(sizes)]


def _on_gpu(host, layout):
    """flat: views of one buffer (neighbours merge); separate: an allocation each; shifted: none of them 16-byte aligned."""
    if layout == "flat":
        buf, out, off = torch.cat(host).cuda(), [], 0
        for t in host:
            out.append(buf[off: off + t.numel()])
            off += t.numel()
        return out
    if layout == "separate":
        return [t.cuda() for t in host]
    return [torch.cat([torch.zeros(1), t]).cuda()[1:] for t in host]


@pytest.mark.parametrize("layout", ["flat", "separate", "shifted"])
@pytest.mark.parametrize("sizes", list(SIZES))
@pytest.mark.parametrize("name,config", [("QSGDMaxNormReducer", {"quantization_level": 8}), ("QSGDMaxNormReducer", {"quantization_level": 1}),
                                         ("QSGDMaxNormTwoScaleReducer", {"quantization_level": 2, "higher_quantization_level": 6}),
                                         ("NoneAllReducer", {})])
def test_matches_the_cpu(name, config, sizes, layout):
    host = _values(SIZES[sizes], 3)
    send, outs = _on_gpu(host, layout), _on_gpu([torch.zeros_like(t) for t in host], layout)
    cpu, gpu = (make_reducer(name, d, None, dict(config, seed=11)) for d in ("cpu", "cuda"))
    for step in range(2):
        in_place = step == 1
        want = [torch.empty_like(t) for t in host]
        bits = cpu.reduce([t.clone() for t in host], want)
        got = send if in_place else outs
        assert gpu.reduce(send, got) == bits
        for w, g in zip(want, got):
            assert torch.equal(w, g.cpu())


@pytest.mark.parametrize("value", [0.0, float("nan"), float("inf"), -float("inf"), 1e-38])
def test_special_values(value):
    host = [torch.full((6,), value), torch.tensor([-1e-3, 0.5, value, -0.25])]
    cpu, gpu = (make_reducer("QSGDMaxNormReducer", d, None, {"quantization_level": 4, "seed": 1}) for d in ("cpu", "cuda"))
    want, got = [torch.empty_like(t) for t in host], [torch.empty_like(t).cuda() for t in host]
    cpu.reduce([t.clone() for t in host], want)
    gpu.reduce([t.cuda() for t in host], got)
    for w, g in zip(want, got):
        assert torch.equal(torch.nan_to_num(w, nan=7.0), torch.nan_to_num(g.cpu(), nan=7.0))


def test_overlapping_tensors_take_the_general_path():
    buf = torch.randn(64, device="cuda")
    send, outs = [buf[:32].clone(), buf[8:40]], [buf[8:40], buf[40:72] if buf.numel() > 72 else torch.zeros(32, device="cuda")]
    host = [t.cpu().clone() for t in send]
    want = [torch.empty_like(t) for t in host]
    cpu, gpu = (make_reducer("QSGDMaxNormReducer", d, None, {"quantization_level": 4, "seed": 1}) for d in ("cpu", "cuda"))
    cpu.reduce([t.clone() for t in host], want)
    gpu.reduce(send, outs)
    for w, g in zip(want, outs):
        assert torch.equal(w, g.cpu())


def _topk_values(kind, sizes):
    host = _values(sizes, 5)
    if kind == "zeros":             # more entries asked for than differ from zero
        return [torch.where(torch.arange(t.numel()) % 211 == 3, t, torch.zeros(())) for t in host]
    if kind == "constant":          # one bin holds everything: no room on the candidate lists
        return [torch.full_like(t, 0.25) for t in host]
    if kind == "tiny":              # subnormals: the lowest bin, with larger entries above it
        return [torch.where(torch.arange(t.numel()) % 301 == 7, t, t * 1e-39) for t in host]
    if kind == "close":             # one bin, all different
        return [1.0 + t * 1e-4 for t in host]
    return host


@pytest.mark.parametrize("layout", ["flat", "separate", "shifted"])
@pytest.mark.parametrize("sizes", ["one", "tile+1", "two-blocks", "kept", "many", "odd starts", "most", "too many"])
@pytest.mark.parametrize("kind", ["normal", "zeros", "constant", "tiny", "close"])
@pytest.mark.parametrize("name,config", [("TopKReducerRatio", {"compression": 0.01}), ("TopKReducer", {"K": 60}), ("GlobalTopKReducer", {"K": 500})])
def test_topk(name, config, kind, sizes, layout):
    host = _topk_values(kind, SIZES[sizes])
    red = make_reducer(name, "cuda", None, config)
    groups = host if name != "GlobalTopKReducer" else [torch.cat(host)]
    mem = [torch.zeros_like(t) for t in groups]
    for step in range(2):
        send = _on_gpu([t * (1 + step) for t in host], layout)
        outs = send if step else _on_gpu([torch.full_like(t, 9.0) for t in host], layout)
        assert red.reduce(send, outs) == sum(red._top_size(t.numel()) for t in groups) * (32 + red.position_bits)
        flat_out = torch.cat([t.cpu() for t in outs])
        got = flat_out.split([t.numel() for t in groups])
        now = red.state_dict()["memory"].cpu().split([t.numel() for t in groups])
        for t, o, e, e_before in zip(groups, got, now, mem):
            a = t * (1 + step) + e_before
            k = red._top_size(t.numel())
            assert torch.equal(o + e, a) and not ((o != 0) & (e != 0)).any()
            threshold = torch.topk(a.abs(), k)[0][-1]
            assert (o != 0).sum() == min(k, int((a != 0).sum()))
            assert (o[o != 0].abs() >= threshold).all() and (e.abs() <= threshold).all()
        mem = now


@pytest.mark.parametrize("kind", ["normal", "zeros", "constant", "tiny"])
@pytest.mark.parametrize("memory", [False, True])
def test_topk_lists(kind, memory):
    from gradient_compression_b200.ops.topk import TopKSelector

    host = _topk_values(kind, SIZES["many"] + [200003])
    a, segs, off = torch.cat(host), [], 0
    for t in host:
        segs.append((off, t.numel(), max(1, t.numel() // 50)))
        off += t.numel()
    sel = TopKSelector(segs, "cuda")
    for _ in range(2):
        e = torch.zeros(off, device="cuda") if memory else None
        idx, val = (t.cpu() for t in sel.select(a.cuda(), e))
        assert torch.equal(val, a[idx.long()]) and idx.unique().numel() == idx.numel()
        for (s, n, k), o in zip(sel.segments, sel.offsets):
            mine = idx[o: o + k].long()
            assert ((mine >= s) & (mine < s + n)).all()
            assert (a[mine].abs() >= torch.topk(a[s: s + n].abs(), k)[0][-1]).all()
        if memory:
            want = a.clone()
            want[idx.long()] = 0
            assert torch.equal(e.cpu(), want)


@pytest.mark.parametrize("layout", ["flat", "separate", "shifted"])
@pytest.mark.parametrize("rank", [1, 2, 3, 4])
@pytest.mark.parametrize("reuse", [False, True])
def test_powersgd(rank, reuse, layout):
    from gradient_compression_b200.reducers import RankKReducer

    # ragged rows, fewer rows or columns than the rank, more rows than one chunk, vectors in between
    shapes = [(64, 3, 3, 3), (64,), (1, 7), (130, 65), (2, 4096), (257, 128), (10,), (3, 1), (65, 64, 1, 1)]
    host = [t.view(s) for t, s in zip(_values([int(torch.Size(s).numel()) for s in shapes], 4), shapes)]
    cpu, gpu = (RankKReducer(d, None, rank=rank, seed=5, reuse_query=reuse) for d in ("cpu", "cuda"))
    for step in range(3):
        now = [t * (1 + 0.1 * step) for t in host]
        want = [torch.empty_like(t) for t in now]
        send = [t.view(s) for t, s in zip(_on_gpu([t.reshape(-1) for t in now], layout), shapes)]
        outs = send if step == 1 else [torch.empty_like(t) for t in send]
        assert gpu.reduce(send, outs) == cpu.reduce([t.clone() for t in now], want)
        for w, g in zip(want, outs):
            torch.testing.assert_close(g.cpu(), w, rtol=2e-4, atol=2e-4 * float(w.abs().max()))
        torch.testing.assert_close(gpu.state_dict()["_memory"].cpu(), cpu.state_dict()["_memory"], rtol=1e-3, atol=2e-4)
    assert reuse or gpu.state_dict()["step"] == cpu.state_dict()["step"] == 3


@pytest.mark.parametrize("layout", ["flat", "separate", "shifted"])
@pytest.mark.parametrize("sizes", ["one", "tile+1", "two-blocks", "kept", "many", "most", "too many"])
@pytest.mark.parametrize("unselected", ["local", "zero"])
@pytest.mark.parametrize("name,K,bits", [("GlobalRandKMaxNormReducer", 300, (8,)), ("GlobalRandKMaxNormReducer", 200000, (4,)),
                                         ("GlobalRandKMaxNormTwoScaleReducer", 1000, (2, 6))])
def test_randk(name, K, bits, unselected, sizes, layout):
    from gradient_compression_b200 import reducers as R

    host = _values(SIZES[sizes], 6)
    kw = dict(seed=7, K=K, unselected=unselected)
    kw.update(quantization_level=bits[0]) if len(bits) == 1 else kw.update(lower_quantization_level=bits[0], higher_quantization_level=bits[1])
    cpu, gpu = (getattr(R, name)(d, None, **kw) for d in ("cpu", "cuda"))
    for step in range(3):                   # windows run through the permutation and wrap around
        want = [torch.empty_like(t) for t in host]
        bits_cpu = cpu.reduce([t.clone() for t in host], want)
        send = _on_gpu(host, layout)
        outs = send if step == 1 else _on_gpu([torch.full_like(t, 9.0) for t in host], layout)
        assert gpu.reduce(send, outs) == bits_cpu
        for w, g in zip(want, outs):
            assert torch.equal(w, g.cpu())
    assert gpu.state_dict()["queue"]["position"] % sum(SIZES[sizes]) == cpu.state_dict()["queue"]["position"] % sum(SIZES[sizes])


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 4096, 148 * 8 * 1024 + 1])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("s", [1, 3, 127, 255, 65535, (1 << 22) - 1, 1 << 22])
def test_level_kernels(n, shift, s):
    from gradient_compression_b200 import ops

    host = _values([n + shift], 8)[0][shift:].contiguous()
    dev = torch.cat([torch.zeros(1), host]).cuda()[1:] if shift else host.cuda()
    norm = ops.absmax(host) * 0.75           # some values beyond the largest level
    for dtype in (torch.int8, torch.int16, torch.int32):
        want = ops.quantize_levels(host, norm, s, 5, 9, 2, dtype=torch.int32)
        got = ops.quantize_levels(dev, norm.cuda(), s, 5, 9, 2, dtype=dtype)
        assert torch.equal(got.cpu(), want.to(dtype))
        assert torch.equal(ops.dequantize_levels(got, norm.cuda(), s, 3).cpu(), ops.dequantize_levels(want.to(dtype).to(torch.int32), norm, s, 3))
        q, mask = ops.quantize_fit(dev, norm.cuda(), s, s // 4, 5, 9, 2, dtype=dtype)
        assert torch.equal(q.cpu(), want.to(dtype)) and torch.equal(mask.cpu(), (want.abs() <= s // 4).to(torch.int8))
        two = ops.dequantize_two(q, mask, norm.cuda(), s, s // 4 + 1, 2).cpu()
        fine, coarse = (ops.dequantize_levels(q.cpu().to(torch.int32), norm, l, 2) for l in (s, s // 4 + 1))
        assert torch.equal(two, torch.where(mask.cpu().bool(), fine, coarse))
    assert torch.equal(ops.absmax(dev).cpu(), ops.absmax(host))


@pytest.mark.parametrize("n,step", [(1000, 4), (4096, 8), (4097, 8), (200003, 400), (3000001, 4000)])
def test_topk_ties_go_to_the_first(n, step):
    """Rounded values: a dozen to a hundred entries share the threshold; the same ones are taken every time, by index."""
    from gradient_compression_b200.ops.topk import TopKSelector

    a = torch.round(torch.randn(n, generator=torch.Generator().manual_seed(n)) * step) / step
    k = n // 50
    sel = TopKSelector([(0, n, k)], "cuda")
    want = torch.sort(a.abs(), descending=True, stable=True)[1][:k].sort()[0]
    for _ in range(3):
        assert torch.equal(sel.select(a.cuda(), None)[0].cpu().long().sort()[0], want)


@pytest.mark.parametrize("rank", [3, 4])
@pytest.mark.parametrize("n,m", [(40, 4), (33, 36), (64, 132), (70, 1060), (17, 4104)])
def test_powersgd_rows_that_end_inside_a_block_of_columns(rank, n, m):
    from gradient_compression_b200.reducers import RankKReducer

    host = _values([n * m], 9)[0].view(n, m)
    cpu, gpu = (RankKReducer(d, None, rank=rank, seed=5) for d in ("cpu", "cuda"))
    for step in range(2):
        want, got = torch.empty_like(host), torch.empty(n, m, device="cuda")
        cpu.reduce([host.clone()], [want])
        gpu.reduce([host.cuda()], [got])
        torch.testing.assert_close(got.cpu(), want, rtol=2e-4, atol=2e-4 * float(want.abs().max()))
        torch.testing.assert_close(gpu.state_dict()["_memory"].cpu(), cpu.state_dict()["_memory"], rtol=1e-3, atol=2e-4)


@pytest.mark.parametrize("name,config", [("QSGDMaxNormReducer", {"quantization_level": 8}), ("NoneAllReducer", {}), ("GlobalRandKMaxNormReducer", {"K": 10}),
                                         ("QSGDMaxNormTwoScaleReducer", {"quantization_level": 2, "higher_quantization_level": 6}),
                                         ("TopKReducerRatio", {"compression": 0.1}), ("RankKReducer", {"rank": 2})])
def test_tensors_of_another_gpu_than_the_arenas_are_refused(name, config):
    """The arena is made to say that it lives on the next GPU: nothing is launched, the general path reports it."""
    import ctypes

    from gradient_compression_b200.ops import _native as nat

    red = make_reducer(name, "cuda", None, dict(config, seed=3))
    x = torch.randn(64, 32, device="cuda")
    first = torch.empty_like(x)
    red.reduce([x], [first])
    ctx = red._fused.ops.arena.ctxs[0]
    device = ctypes.c_int.from_address(ctx.handle.value + 8)               # CommCtx {world, rank, device, ...}
    assert nat.cuda().gc_comm_device(ctx.handle) == device.value == ctx.device_index == x.device.index
    out, before = torch.full_like(x, 5.0), nat.launches()
    try:
        device.value += 1
        ctx.device_index += 1
        assert red._solo_reduce([x], [out]) is None
        if name.startswith(("QSGD", "None")):                   # (the others' general path has an arena of its own)
            with pytest.raises(ValueError, match="arena"):
                red.reduce([x], [out])
        assert nat.launches() == before
    finally:
        device.value -= 1
        ctx.device_index -= 1
    torch.cuda.synchronize()
    assert bool((out == 5.0).all())
    red.reduce([x], [out])
    assert not bool((out == 5.0).any())


@pytest.mark.parametrize("n", [4097, 5000, 200003, 3000001])
@pytest.mark.parametrize("step", [1, 3, 16, 0])
@pytest.mark.parametrize("dense", [False, True])
def test_topk_any_number_of_ties_goes_to_the_first(n, step, dense):
    """Values rounded to halves, sixths or thirty-seconds, and one value everywhere: from some hundred entries at the threshold to all of
    them, on the candidate lists and beyond their room."""
    from gradient_compression_b200.ops.topk import TopKSelector

    gen = torch.Generator().manual_seed(n + step)
    a = torch.round(torch.randn(n, generator=gen) * 2 * step) / (2 * step) if step else torch.full((n,), -0.375)
    k = n // 30
    want = torch.sort(a.abs(), descending=True, stable=True)[1][:k].sort()[0]
    sel, x = TopKSelector([(0, n, k)], "cuda"), a.cuda()
    for _ in range(2):
        if dense:
            red, out = make_reducer("GlobalTopKReducer", "cuda", None, {"K": k}), torch.empty_like(x)
            red.reduce([x], [out])
            got, expected = out.cpu(), torch.zeros(n)
            expected[want] = a[want]
            assert torch.equal(got, expected) and torch.equal(red.state_dict()["memory"].cpu(), a - expected)
        else:
            assert torch.equal(sel.select(x, None)[0].cpu().long().sort()[0], want)
