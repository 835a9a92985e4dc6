"""Operands rewritten k-major before a large build: the scratch entry point against the plain one, which reads
them where they lie.  Square, |.| and product results are the same bits."""
import ctypes

import pytest
import torch

import kermac_b200 as kermac
from kermac_b200 import _native
from kermac_b200.build_a_kernel import _current_stream_for, _marshal_build
from kermac_b200.cdist import descriptor_for

pytestmark = pytest.mark.gpu


def _points(gen, lead, count, K, layout):
    if layout == "rows":
        return torch.randn(*lead, count, K, generator=gen).cuda()
    if layout == "off":                                        # rows that start one float off
        return torch.randn(*lead, count, K + 3, generator=gen).cuda()[..., 1:K + 1]
    pitch = (count + 3) // 4 * 4 + (1 if layout == "odd_pitch" else 0)
    return torch.randn(*lead, K, pitch, generator=gen).cuda()[..., :count].transpose(-1, -2)


def _call(a, b, out, p, scratch_bytes=None):
    descriptor, powers = descriptor_for(p, False)
    args, _, keep = _marshal_build(descriptor, a, b, out, powers.get("p"), powers.get("inner_p"), None, None, None, None, 0, 0)
    lib, stream = _native.lib(), ctypes.c_void_p(_current_stream_for(a.device))
    need = lib.kermac_b200_build_scratch_bytes(ctypes.byref(args))
    have = need if scratch_bytes is None else scratch_bytes
    scratch = torch.full((max(have // 4, 1),), float("nan"), device="cuda")
    _native.check(lib.kermac_b200_build_kernel_scratch(ctypes.byref(args), scratch.data_ptr() if have else None, have, stream), "build")
    del keep
    return need


@pytest.mark.parametrize("layouts", [("rows", "rows"), ("rows", "cols"), ("cols", "off"), ("off", "odd_pitch")])
@pytest.mark.parametrize("shape", [((), 4001, 4099, 130), ((), 8200, 3001, 96), ((2,), 3000, 2111, 260)])
def test_packed_operands_give_the_same_bits(layouts, shape):
    lead, M, N, K = shape
    gen = torch.Generator().manual_seed(M)
    a = _points(gen, lead, M, K, layouts[0])
    for b in (_points(gen, lead, N, K, layouts[1]), _points(gen, (), N, K, layouts[1])):       # the second broadcasts
        for out in (torch.empty(*lead, M, N, device="cuda"), torch.empty(*lead, N, M, device="cuda").transpose(-1, -2)):
            for p in (2.0, 1.0):
                _call(a, b, out.fill_(-1.0), p, scratch_bytes=0)
                want = out.clone()
                need = _call(a, b, out.fill_(-1.0), p)
                assert torch.equal(out, want)
                if p == 2.0:
                    assert need > 0, "the case must be one that packs"
                    _call(a, b, out.fill_(-1.0), p, scratch_bytes=need - 4)      # one element short: not used
                    assert torch.equal(out, want)
                    assert torch.equal(kermac.cdist(a, b, out=out.fill_(-1.0), p=p), want)
    assert _native.device_error_flag() == 0


@pytest.mark.parametrize("shape", [(3000, 3000, 301), (4001, 4003, 200), (6001, 5003, 130)])
def test_fractional_powers_do_not_depend_on_the_scratch(shape):
    M, N, K = shape                                             # below and above the line between the kernels
    gen = torch.Generator().manual_seed(K)
    a, b = _points(gen, (), M, K, "off"), _points(gen, (), N, K, "off")
    out, other = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
    assert _call(a, b, out, 1.3) > 0, "the case must be one that packs"
    _call(a, b, other, 1.3, scratch_bytes=0)
    assert torch.equal(out, other)


def test_one_matrix_is_packed_once_and_stays_symmetric():
    x = torch.randn(8001, 96, generator=torch.Generator().manual_seed(1)).cuda()
    out = torch.empty(8001, 8001, device="cuda")
    need = _call(x, x, out, 2.0)
    assert need == 96 * 8032 * 4
    assert torch.equal(out, out.t())
    other = torch.empty_like(out)
    _call(x, x, other, 2.0, scratch_bytes=0)
    assert torch.equal(out, other)


@pytest.mark.parametrize("desc", ["l1", "l2"])
@pytest.mark.parametrize("layouts", [("rows", "rows"), ("cols", "off"), ("off", "cols")])
@pytest.mark.parametrize("shape", [((), 10007, 1009, 27, 5), ((), 5000, 6001, 40, 17), ((3,), 4100, 2000, 65, 2)])
def test_matvec_on_packed_operands(shape, layouts, desc):
    # the operands as given against the same points already contiguous along the points: the same kernel
    # arithmetic and the same split over m, so the same bits
    lead, M, N, K, O = shape
    descriptor = kermac.kernel_descriptor_laplace_l1 if desc == "l1" else kermac.kernel_descriptor_laplace_l2
    gen = torch.Generator().manual_seed(K)
    a, c = _points(gen, lead, M, K, layouts[0]), torch.randn(*lead, O, M, generator=gen).cuda()
    for b in (_points(gen, lead, N, K, layouts[1]), _points(gen, (), N, K, layouts[1])):
        def aligned(x):
            buf = torch.zeros(*x.shape[:-2], K, (x.shape[-2] + 3) // 4 * 4, device="cuda")
            buf[..., :x.shape[-2]] = x.transpose(-1, -2)
            return buf[..., :x.shape[-2]].transpose(-1, -2)
        got = kermac.kernel_matvec(descriptor, a, b, c, bandwidth=8.0)
        assert torch.equal(got, kermac.kernel_matvec(descriptor, aligned(a), aligned(b), c, bandwidth=8.0))
        x = aligned(a)                                         # one matrix on both sides: one copy serves both
        assert torch.equal(kermac.kernel_matvec(descriptor, a, a, c, bandwidth=8.0),
                           kermac.kernel_matvec(descriptor, x, x, c, bandwidth=8.0))
        split = kermac.kernel_matvec(descriptor, a, b, c, bandwidth=8.0, split_m=3)
        assert torch.allclose(got, split, rtol=0.0, atol=float(got.abs().max()) * 2e-6)    # sums of M terms, regrouped
    assert _native.device_error_flag() == 0
