"""Small things a captured step leaves out: a vector of metrics that exists already is not stacked again, VGG's pooling of one pixel is not run unless
it does something."""
import torch

from gradient_compression_b200 import models
from gradient_compression_b200.parallel import graph
from gradient_compression_b200.parallel.graph import _side_by_side


def test_side_by_side():
    base = torch.tensor([1.0, 2.0, 3.0])
    assert _side_by_side([base[0], base[1], base[2]]) is base
    for scalars in ([base[0], base[2], base[1]], [base[0], base[1]], [base[0].clone(), base[1], base[2]], list(torch.ones(3, dtype=torch.float64)), [torch.ones(1)] * 3):
        got = _side_by_side(scalars)
        assert got is not base and got.dtype == torch.float32 and got.tolist() == [float(v) for v in scalars]


def test_pooling_of_one_pixel():
    torch.manual_seed(0)
    net, x = models.VGG11().eval(), torch.randn(2, 3, 32, 32)
    want = net.features(x)
    assert torch.equal(net._features(x), want)
    seen = []
    handle = net.features[-1].register_forward_hook(lambda *_: seen.append(1))
    net._features(x)
    handle.remove()
    net.features[-1].divisor_override = 2
    assert seen == [1] and torch.equal(net._features(x), want / 2)


def test_status_buffer_outlives_its_mirror_until_the_copy_has_landed():
    class Event:
        done = False

        def query(self):
            return self.done

    mirror, event, before = graph._StatusMirror(torch.device("cpu")), Event(), len(graph._in_flight)
    mirror.host, mirror.event = torch.zeros(1, 2), event
    del mirror
    graph._release_landed()
    assert [e.event for e in graph._in_flight[before:]] == [event]
    event.done = True
    graph._release_landed()
    assert len(graph._in_flight) == before


def test_a_later_step_gives_back_the_status_buffer_of_one_that_is_gone():
    class Event:
        def query(self):
            return True

    mirror, other, before = graph._StatusMirror(torch.device("cpu")), graph._StatusMirror(torch.device("cpu")), len(graph._in_flight)
    mirror.host, mirror.event = torch.zeros(1, 2), Event()
    del mirror
    assert len(graph._in_flight) == before + 1
    other.check()                                   # its arenas stay as they are
    assert len(graph._in_flight) == before
