"""Kernels start while the one before them in the stream drains (programmatic stream serialization).  A chain of calls
that read, overwrite and reuse one another's buffers has to give the bits it gives when the device is waited for after
every call: on one stream, on two at a time, and captured in a graph."""
import pytest
import torch

import kermac_b200 as kermac
from kermac_b200 import _native

pytestmark = pytest.mark.gpu


def _chain(x, rows, wait):
    """Every step's input is the last one's result; `d` is overwritten while the kernel before still reads it."""
    seen = []

    def after(t):
        if wait:
            torch.cuda.synchronize()
        return t

    a, b = x, x.clone()
    d = torch.empty(1, rows, rows, device="cuda").transpose(1, 2)
    for p in (2.0, 1.0, 1.3):
        after(kermac.cdist(a, b, out=d, p=p))                              # overwritten in every round
        k = after(kermac.run_kernel(kermac.kernel_descriptor_laplace_l2, d[0], d[0], bandwidth=50.0))[0]
        c = after(k[:20] * 0.01)                                           # a torch kernel between two of ours
        y = after(kermac.kernel_matvec(kermac.kernel_descriptor_laplace_l1, d[0], d[0], c, bandwidth=500.0))
        y = y.reshape(rows, 20).t().contiguous()
        t = d[0].t().contiguous()
        g = after(kermac.cdist_grad(k, t, y, t, p=p))
        a = after(x + 1e-3 * torch.tanh(g.reshape(20, rows, rows)[0][:, :x.shape[1]]))
        seen += [t.clone() for t in (d, k, y, g)]
    return seen


def _inputs(seed, rows=400):
    gen = torch.Generator().manual_seed(seed)
    return torch.randn(rows, 40, generator=gen).cuda(), rows


@pytest.mark.parametrize("rows", [130, 400])
def test_one_stream(rows):
    x, rows = _inputs(1, rows)
    want = _chain(x, rows, True)
    for _ in range(5):
        got = _chain(x, rows, False)
        assert all(torch.equal(w, g) for w, g in zip(want, got))
    assert _native.device_error_flag() == 0


def test_two_streams():
    inputs = [_inputs(2), _inputs(3)]
    want = [_chain(*i, True) for i in inputs]
    streams = [torch.cuda.Stream() for _ in inputs]
    torch.cuda.synchronize()
    for _ in range(3):
        got = []
        for s, i in zip(streams, inputs):
            with torch.cuda.stream(s):
                got.append(_chain(*i, False))
        torch.cuda.synchronize()
        for w, g in zip(want, got):
            assert all(torch.equal(x, y) for x, y in zip(w, g))
    assert _native.device_error_flag() == 0


def test_captured():
    x, rows = _inputs(4)
    want = _chain(x, rows, True)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        _chain(x, rows, False)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = _chain(x, rows, False)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(w, g) for w, g in zip(want, got))
