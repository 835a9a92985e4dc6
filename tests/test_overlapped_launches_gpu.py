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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("size", [256, 1024, 2304])
def test_behind_a_matrix_product(size, dtype):
    """Library products may let the next kernel's blocks in while their own still run, and use tensor memory themselves:
    every kernel that takes some behind one, on what the product has just written."""
    gen = torch.Generator().manual_seed(size)
    x, w = (torch.randn(size, size, generator=gen).div(size ** 0.5).cuda().to(dtype) for _ in range(2))
    product = torch.empty(size, size, device="cuda", dtype=dtype)
    f32 = torch.empty(size, size, device="cuda")
    small, c = torch.randn(40, 130, generator=gen).cuda(), torch.randn(24, size, generator=gen).cuda()
    b = torch.randn(130, size, generator=gen).cuda()
    desc = kermac.kernel_descriptor_laplace_l2
    calls = {
        "signs": lambda: kermac.cdist_grad(f32, b, c, f32[:130], p=1.0, contraction="tensor"),
        "weights": lambda: kermac.cdist_grad(f32, b, c, f32[:130], p=1.5, contraction="tensor"),
        "matvec": lambda: kermac.kernel_matvec(desc, f32[:, :40], small.t(), c, bandwidth=8.0, contraction="tensor"),
        "cdist": lambda: kermac.cdist(f32[:, :40], small.t(), p=1.3),
    }

    def passes(wait):
        seen = []
        for name, call in calls.items():
            # with float32 the product's own result is the operand, else its copy
            for i in range(3):
                torch.matmul(x, w + 0.01 * i, out=product if dtype != torch.float32 else f32)
                if dtype != torch.float32:
                    f32.copy_(product)
                    torch.matmul(x, w, out=product)
                if wait:
                    torch.cuda.synchronize()
                seen.append(call())
                if wait:
                    torch.cuda.synchronize()
        return seen

    want = passes(True)
    for _ in range(3):
        assert all(torch.equal(w, g) for w, g in zip(want, passes(False)))
    assert _native.device_error_flag() == 0


def test_captured_with_joined_streams():
    """A fork and a join inside a capture: the kernels behind the join wait for both branches."""
    x, rows = _inputs(5)
    y = x.flip(0).contiguous()
    want = [_chain(x, rows, True), _chain(y, rows, True)]
    last = lambda branches: kermac.cdist(branches[0][0][0], branches[1][0][0], p=1.0)       # noqa: E731
    want.append([last(want)])
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(main):
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=main):
            side.wait_stream(main)
            with torch.cuda.stream(side):
                second = _chain(y, rows, False)
            got = [_chain(x, rows, False), second]
            main.wait_stream(side)
            got.append([last(got)])
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for w, g in zip(want, got):
        assert all(torch.equal(a, b) for a, b in zip(w, g))
    assert _native.device_error_flag() == 0
