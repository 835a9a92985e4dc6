"""The automatic k split of cdist_grad at sizes where one block per tile would leave the machine idle: against a
single pass over k (the same terms, regrouped) and against the float64 oracle.

Bound of the regrouping: each of the K additions of the single pass rounds by at most 2^-24 of a partial sum, which
stays about below the largest entry; independent, they add up to 2^-24 sqrt(K / 3) of it (one sigma).  Held to
2 * 2^-24 sqrt(K), 3.5 sigma of that."""
import contextlib
import ctypes
import math

import pytest
import torch

import kermac_b200 as kermac
from kermac_b200 import _native
from oracle import kermac_oracle as ko

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def full_device():
    """torch's allocator has no more than 1 MB to give."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / torch.cuda.get_device_properties(0).total_memory)
    held, size = [], 1 << 30                                     # what is free inside the segments in use
    try:
        while size >= 1 << 20:
            try:
                held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                size //= 2
        yield
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


def _single_pass(a, b, c, d, p):
    O, N, M = c.shape[-2], b.shape[-2], a.shape[-1]
    out = torch.full((O, N, M), float("nan"), device="cuda")
    g = _native.KmGradArgs()
    g.m, g.n, g.o, g.k, g.l = M, N, O, a.shape[-2], 1
    g.a, g.lda, g.b, g.ldb = a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0)
    g.c, g.ldc, g.d, g.ldd = c.data_ptr(), c.stride(0), d.data_ptr(), d.stride(0)
    g.out, g.out_stride_n, g.out_stride_o = out.data_ptr(), M, N * M
    g.norm_type = _native.NORM_L1 if p == 1.0 else _native.NORM_L2 if p == 2.0 else _native.NORM_P
    g.p, g.split_k = _native.hyper(p), 0
    wanted = _native.lib().kermac_b200_cdist_grad_scratch_bytes(ctypes.byref(g))
    g.split_k = 1
    _native.launch_grad(g, torch.cuda.current_stream().cuda_stream)
    return out, wanted // (4 * O * N * M)


@pytest.mark.parametrize("p", [1.0, 1.5, 1.7, 2.0])
@pytest.mark.parametrize("shape", [(225, 65, 17, 1), (130, 64, 16, 2), (257, 63, 15, 4), (1000, 200, 50, 8), (3000, 70, 33, 16),
                                   (500, 100, 30, 32), (2999, 33, 9, 33)])
def test_split_sums_match_a_single_pass(shape, p):
    K, M, N, O = shape
    gen = torch.Generator().manual_seed(K)
    a, b = torch.rand(K, M, generator=gen).cuda(), torch.randn(N, K, generator=gen).cuda()
    c, d = torch.randn(O, K, generator=gen).cuda(), torch.randn(N, M, generator=gen).cuda()
    want, splits = _single_pass(a, b, c, d, p)
    assert splits > 1, "the case must be one that splits"
    got = kermac.cdist_grad(a, b, c, d, p=p)
    assert float((got - want).abs().max()) <= 2.0 ** -23 * math.sqrt(K) * float(want.abs().max())
    assert ko.rel_err_signed(got, ko.cdist_grad_ref(a.cpu(), b.cpu(), c.cpu(), d.cpu(), p=p)[0]) < 5e-5
    assert _native.device_error_flag() == 0


def test_a_full_device_takes_a_single_pass():
    K, M, N, O = 3000, 4096, 320, 4                              # one partial result is 21 MB
    gen = torch.Generator().manual_seed(1)
    a, b = torch.rand(K, M, generator=gen).cuda(), torch.randn(N, K, generator=gen).cuda()
    c, d = torch.randn(O, K, generator=gen).cuda(), torch.randn(N, M, generator=gen).cuda()
    want, splits = _single_pass(a, b, c, d, 1.0)
    assert splits > 1, "the case must be one that splits"
    for debug in (False, True):                                  # the native call path and the ctypes one
        out = torch.full((O, N, M), float("nan"), device="cuda")
        with full_device():
            kermac.cdist_grad(a, b, c, d, out=out, p=1.0, debug=debug)
        assert torch.equal(out, want)
        assert not torch.equal(kermac.cdist_grad(a, b, c, d, out=out, p=1.0, debug=debug), want)      # split again


@pytest.mark.parametrize("O", [5, 16])
def test_one_automatic_split_whoever_holds_the_scratch(O):
    # The sign kernel takes fewer splits than callers are asked scratch for.  With room for its own ones, and in the
    # library's built-in array, it sums in the same groups as in the ordinary call.
    K, M, N = 30000, 64, 128
    gen = torch.Generator().manual_seed(7)
    a, b = torch.rand(K, M, generator=gen).cuda(), torch.randn(N, K, generator=gen).cuda()
    c, d = torch.randn(O, K, generator=gen).cuda(), torch.randn(N, M, generator=gen).cuda()
    want = kermac.cdist_grad(a, b, c, d, p=1.0)[0]
    g = _native.KmGradArgs()
    g.m, g.n, g.o, g.k, g.l = M, N, O, K, 1
    g.a, g.lda, g.b, g.ldb = a.data_ptr(), M, b.data_ptr(), K
    g.c, g.ldc, g.d, g.ldd = c.data_ptr(), K, d.data_ptr(), M
    g.out_stride_n, g.out_stride_o, g.norm_type, g.p = M, N * M, _native.NORM_L1, _native.hyper(1.0)
    g.out = want.data_ptr()
    plan = dict(word.split("=") for word in _native.describe_grad(g).split()[1:])
    need = int(plan["splits"]) * O * N * M * 4
    assert plan["kernel"] == "sign" and int(plan["splits"]) > 1 and need < _native.lib().kermac_b200_cdist_grad_scratch_bytes(ctypes.byref(g))
    stream = torch.cuda.current_stream().cuda_stream
    scratch = torch.empty(need // 4, device="cuda")
    for launch in (_native.launch_grad, _native.launch_grad_static):
        out = torch.full((O, N, M), float("nan"), device="cuda")
        g.out, g.scratch, g.scratch_bytes = out.data_ptr(), scratch.data_ptr(), need
        launch(g, stream)
        assert torch.equal(out, want)
    assert _native.device_error_flag() == 0
