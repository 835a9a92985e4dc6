"""The 64 x 64 build kernel against the 128 x 128 one (KERMAC_B200_VARIANT=cpasync forces the latter, any
layout): the same terms summed in the same k order, so |.|, square and product results are the same bits;
the fractional power takes one of two exp2 routes by position and agrees to their rounding (2.9e-7 per term
and a few more units from the outer power: 2e-6)."""
import pytest
import torch

import kermac_b200 as kermac
from kermac_b200 import _native

pytestmark = pytest.mark.gpu

PRODUCT = kermac.KernelDescriptor(kermac.InnerOperator.DOT, kermac.PowerType.NOOP, kermac.PowerType.NOOP,
                                  kermac.KernelType.NONE)


def _points(gen, lead, count, K, layout):
    if layout == "rows":                                   # k contiguous
        return torch.randn(*lead, count, K, generator=gen).cuda()
    if layout == "cols":                                   # tile dimension contiguous
        return torch.randn(*lead, K, count, generator=gen).cuda().transpose(-1, -2)
    if layout == "cols_pitch4":                            # the same with an aligned pitch
        pitch = (count + 3) // 4 * 4
        return torch.randn(*lead, K, pitch, generator=gen).cuda()[..., :count].transpose(-1, -2)
    return torch.randn(*lead, count, K + 5, generator=gen).cuda()[..., 1:K + 1]      # rows off by one float


def _both(call, monkeypatch):
    got = call()
    monkeypatch.setenv("KERMAC_B200_VARIANT", "cpasync")
    want = call()
    monkeypatch.delenv("KERMAC_B200_VARIANT")
    return got, want


def _same(got, want, exact):
    if exact:
        assert torch.equal(got, want)
    else:
        assert torch.allclose(got, want, rtol=2e-6, atol=0.0)


@pytest.mark.parametrize("layouts", [("rows", "rows"), ("cols_pitch4", "cols_pitch4"), ("cols", "rows"),
                                     ("rows", "off"), ("off", "cols_pitch4")])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 65, 15), (64, 64, 16), (63, 129, 17), (65, 63, 4), (130, 190, 48),
                                   (193, 70, 66)])
def test_same_bits_as_the_large_tiles(layouts, shape, monkeypatch):
    M, N, K = shape
    gen = torch.Generator().manual_seed(M * 1000 + N)
    for lead in ((), (3,)):
        a, b = _points(gen, lead, M, K, layouts[0]), _points(gen, lead, N, K, layouts[1])
        outs = (torch.empty(*lead, M, N, device="cuda"), torch.empty(*lead, N, M, device="cuda").transpose(-1, -2))
        for out in outs:
            for p in (1.0, 2.0, 1.3):
                _same(*_both(lambda: kermac.cdist(a, b, out=out.fill_(-7.0), p=p).clone(), monkeypatch), p != 1.3)
            _same(*_both(lambda: kermac.run_kernel(PRODUCT, a, b, out=out.fill_(-7.0)).clone(), monkeypatch), True)
    assert _native.device_error_flag() == 0


@pytest.mark.parametrize("layout", ["rows", "cols_pitch4"])
@pytest.mark.parametrize("M", [127, 129, 200, 321])
def test_symmetric_diagonal_and_chains(layout, M, monkeypatch):
    gen = torch.Generator().manual_seed(M)
    x, K = _points(gen, (), M, 40, layout), kermac
    for desc in (K.kernel_descriptor_laplace_l1, K.kernel_descriptor_laplace_l2,
                 K.KernelDescriptor(K.InnerOperator.DIFF, K.PowerType.SQUARE, K.PowerType.SQUARE, K.KernelType.GAUSSIAN)):
        got, want = _both(lambda: kermac.run_kernel(desc, x, x, bandwidth=9.0, regularization=0.5), monkeypatch)
        _same(got, want, True)
        assert torch.equal(got, got.transpose(-1, -2))
        for ox, oy in ((0, 70), (70, 0)):                  # shifted diagonal, no symmetry
            _same(*_both(lambda: kermac.run_kernel(desc, x, x, bandwidth=9.0, regularization=0.5,
                                                   regularization_offset_x=ox, regularization_offset_y=oy), monkeypatch), True)


def test_values_that_are_not_finite_and_batched_powers(monkeypatch):
    gen = torch.Generator().manual_seed(5)
    a, b = torch.randn(2, 70, 33, generator=gen).cuda(), torch.randn(2, 66, 33, generator=gen).cuda()
    a[0, 3, 5], a[1, 69, 32], b[0, 65, 0] = float("inf"), float("nan"), -float("inf")
    a[0, 10] = b[0, 11]                                    # a zero distance
    for p in (1.0, 2.0, 1.3):
        got, want = _both(lambda: kermac.cdist(a, b, p=p), monkeypatch)
        assert torch.allclose(got, want, rtol=2e-6, atol=0.0, equal_nan=True)
    p = torch.tensor([1.2, 2.5], device="cuda")
    got, want = _both(lambda: kermac.run_kernel(kermac.kernel_descriptor_p_norm, a, b, p=p), monkeypatch)
    assert torch.allclose(got, want, rtol=2e-6, atol=0.0, equal_nan=True)
