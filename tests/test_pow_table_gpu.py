"""|b - a|^p through the table of powers of two and a polynomial (a scalar p in [1.01, 4] that is not whole) against
float64 and against the lg2 / ex2 route, which a p given as a tensor takes.

Bounds.  On MUFU a term is 2^x, x = p lg2|d|: lg2.approx is within 2^-22 of lg2|d| between 1/2 and 2 and within 2^-22 of
its size elsewhere, the product rounds by 2^-24 of x, ex2.approx by 2^-22 of the result, so a term is within
2^-22 (ln 2 (1.25 |x| + p) + 1) of the power.  The table and its polynomial are within 3.5e-7 up to p = 2, 5e-7 up to 3 and 9e-7 up to 4
(_polynomial_error), about as much as that leaves for |d| = 1 and less elsewhere.  Adding K positive
terms rounds by at most K units of 2^-25 in the mean.  Raw sums are compared, so no outer power adds to it."""
import numpy as np
import pytest
import torch

import kermac_b200 as kermac
from kermac_b200 import _native

RAW = kermac.KernelDescriptor(kermac.InnerOperator.DIFF, kermac.PowerType.POW, kermac.PowerType.NOOP,
                              kermac.KernelType.NONE)
gpu = pytest.mark.gpu


def _exact(a, b, p):
    a, b = a.double(), b.double()
    rows = [((b[None] - x[:, None]).abs() ** p).sum(-1) for x in a.split(64)]
    return torch.cat(rows)


def _bound(a, b, p):
    d = (b.double()[None] - a.double()[:, None]).abs()
    x = p * d[d > 0].log2().abs().max().item() if (d > 0).any() else 0.0
    return 2.0 ** -22 * (0.87 * x + 0.7 * p + 1.0) + a.shape[1] * 2.0 ** -25


def _both_routes(a, b, p):
    table = kermac.cdist(a, b, p=p, skip_epilogue=True).reshape(a.shape[0], b.shape[0])
    mufu = kermac.run_kernel(RAW, a, b, inner_p=torch.tensor([p], device="cuda")).reshape(a.shape[0], b.shape[0])
    return table, mufu


def _build_args(p, n=8000, k=300):
    args = _native.KmBuildArgs()
    args.a = args.b = args.out = 0x1000
    args.m = args.n = n
    args.k, args.l = k, 1
    args.a_stride_m, args.a_stride_k = 1, n
    args.b_stride_n, args.b_stride_k = 1, n
    args.out_stride_m, args.out_stride_n = 1, n
    args.inner_operator, args.inner_power = _native.INNER_DIFF, _native.POW_POW
    args.outer_power, args.kernel_type = _native.POW_NOOP, _native.KERNEL_NONE
    args.p_inner = _native.hyper(p)
    return args


@pytest.mark.parametrize("p, table", [(1.0, False), (1.005, False), (1.01, True), (1.3, True), (2.0, False), (2.5, True),
                                      (3.0, False), (4.0, False), (3.999, True), (4.001, False), (0.5, False), (-1.0, False),
                                      (0.0, False), (float("nan"), False), (float("inf"), False)])
def test_which_exponents_take_the_table(p, table):
    assert ("pow=table" in _native.describe_build(_build_args(p))) is table


@pytest.mark.parametrize("n", [40, 1000, 8000])
@pytest.mark.parametrize("rows", [False, True])
def test_few_features_keep_the_mufu_route(rows, n):
    """The line lies at 6 features, for a matrix with itself at 11 to 15 and from 21 on, and follows neither the tile range nor
    whether the mirror image is computed."""
    for k in range(1, 40):
        for same in (False, True):
            args = _build_args(1.3, n, k)
            if rows:
                args.a_stride_m, args.a_stride_k, args.b_stride_n, args.b_stride_k = k, 1, k, 1
            if not same:
                args.b = 0x2000
            table = "pow=table" in _native.describe_build(args)
            assert table is (k in range(11, 16) or k > 20 if same else k >= 6)
            args.symmetry = 1
            assert ("pow=table" in _native.describe_build(args)) is table
            args.symmetry, args.tile_count = 0, 1
            assert ("pow=table" in _native.describe_build(args)) is table


def test_a_tensor_exponent_and_the_tma_variant_keep_the_mufu_route():
    args = _build_args(1.3)
    args.variant = _native.VARIANT_TMA
    assert "variant=tma" in _native.describe_build(args) and "pow=table" not in _native.describe_build(args)
    args = _build_args(1.3)
    args.p_inner.ptr = 0x1000
    assert "pow=table" not in _native.describe_build(args)


@gpu
@pytest.mark.parametrize("variant", ["auto", "cpasync"])
@pytest.mark.parametrize("p", [1.01, 1.3, 1.5, 2.5, 3.7, 3.999])
@pytest.mark.parametrize("shape", [(1, 1, 1), (64, 64, 16), (65, 130, 17), (129, 67, 70)])
def test_against_float64(shape, p, variant, monkeypatch):
    if variant != "auto":                                    # the 128 x 128 kernel
        monkeypatch.setenv("KERMAC_B200_VARIANT", variant)
    M, N, K = shape
    gen = torch.Generator().manual_seed(K)
    for scale in (1.0, 3e-6, 4e5):
        a, b = (torch.randn(c, K, generator=gen).cuda() * scale for c in (M, N))
        want, rtol = _exact(a, b, p), _bound(a, b, p)
        for got in _both_routes(a, b, p):
            assert torch.allclose(got.double(), want, rtol=rtol, atol=1e-36)
        cols = kermac.cdist(a.t().contiguous().t(), b.t().contiguous().t(), p=p, skip_epilogue=True)
        assert torch.allclose(cols.reshape(M, N).double(), want, rtol=rtol, atol=1e-36)


@gpu
@pytest.mark.parametrize("variant", ["auto", "cpasync"])
@pytest.mark.parametrize("p", [1.01, 1.3, 2.3, 3.7])
@pytest.mark.parametrize("features", [3, 8])
def test_values_at_the_ends_of_the_range(features, p, variant, monkeypatch):
    # one value against zeros in every place of a register block, so that every pair's route sees it
    if variant != "auto":
        monkeypatch.setenv("KERMAC_B200_VARIANT", variant)
    inf, nan = float("inf"), float("nan")
    values = torch.tensor([0.0, -0.0, 1e-45, 1e-39, 1.2e-38, 2e-30, 1.0, 1.9999999, 1e9, 1e19, 8e37, 1.6e38, 1.8e38, 3.4e38,
                           inf, nan])
    values = torch.cat([values, -values])
    a = torch.zeros(40 * len(values), features, device="cuda")
    a[:, 0] = values.repeat_interleave(40)
    b = torch.zeros(130, features, device="cuda")
    want = values.repeat_interleave(40)[:, None].expand(-1, 130).cuda().double().abs() ** p
    for got in _both_routes(a, b, p):
        assert torch.equal(got.isnan(), want.isnan())
        big = want > 3.5e38
        assert torch.equal(got.isinf(), big)
        rest = ~(want.isnan() | big)
        # |lg2| is at most 128 here; what lg2.approx.ftz and ex2.approx.ftz flush is below 2^-126
        rtol = 2.0 ** -22 * (0.87 * 128 * p + 0.7 * p + 1.0)
        assert torch.allclose(got[rest].double(), want[rest], rtol=rtol, atol=2.0 ** -125)


@gpu
@pytest.mark.parametrize("features", [2, 24])
def test_infinite_and_undefined_differences(features):
    inf = float("inf")
    a = torch.zeros(4, features, device="cuda")
    a[:, :2] = torch.tensor([[inf, 1.0], [-inf, 1.0], [3e38, 0.0], [0.0, 0.0]])
    got, mufu = _both_routes(a, a, 1.3)
    want = _exact(a, a, 1.3)                                 # inf - inf is NaN, 6e38 overflows
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), mufu.isinf())
    assert torch.equal(got.isnan(), mufu.isnan())


def _polynomial_error(p, m):
    """Largest relative error of the degree-6 polynomial through m^p at the Chebyshev nodes of [1, 2), its coefficients and
    each step rounded to float32 (a product of two floats is exact in float64)."""
    nodes = 1.5 + 0.5 * np.cos(np.pi * (np.arange(7) + 0.5) / 7)
    c = np.polyfit(nodes - 1.5, nodes ** p, 6).astype(np.float32).astype(np.float64)
    f = m - 1.5
    q = np.full_like(f, c[0])
    for coefficient in c[1:]:
        q = (q * f + coefficient).astype(np.float32).astype(np.float64)
    return np.abs(q / m ** p - 1.0).max()


@pytest.mark.parametrize("low, high, bound", [(1.01, 2.0, 3.5e-7), (2.0, 3.0, 5e-7), (3.0, 4.0, 9e-7)])
def test_the_polynomial_stays_within_the_stated_error(low, high, bound):
    m = np.concatenate([np.arange(1.0, 2.0, 2.0 ** -12), 1.0 + np.arange(512) * 2.0 ** -23])
    worst = max(_polynomial_error(float(np.float32(p)), m) for p in np.arange(low, high, 0.003))
    assert 0.5 * bound < worst <= bound


@gpu
@pytest.mark.parametrize("p", [1.01, 1.3, 1.72, 1.99, 2.88, 3.46, 3.7, 3.999])
@pytest.mark.parametrize("variant", ["auto", "cpasync"])
def test_pairs_that_take_the_table(p, variant, monkeypatch):
    """One feature that is not zero, the b side zero, a contiguous along the points: column n of the result is the power of a
    alone, by lg2 and ex2 for even n and by the table for odd n, where 2^0 m^p is the polynomial as it is."""
    if variant != "auto":
        monkeypatch.setenv("KERMAC_B200_VARIANT", variant)
    m = torch.cat([torch.arange(0, 4096) * 2.0 ** -12, torch.arange(0, 512) * 2.0 ** -23]) + 1.0
    for octave in (0, -7, 5):
        x = torch.ldexp(m, torch.tensor(octave)).cuda()
        a, b = torch.zeros(6, len(x), device="cuda"), torch.zeros(6, 70, device="cuda")
        a[2] = x
        out = torch.empty(1, 70, len(x), device="cuda").transpose(1, 2)
        kermac.cdist(a.t(), b.t(), out=out, p=p, skip_epilogue=True)
        even, odd = out[0][:, ::2], out[0][:, 1::2]
        assert torch.equal(even, even[:, :1].expand_as(even)) and torch.equal(odd, odd[:, :1].expand_as(odd))
        assert not torch.equal(even, odd)
        exact = x.double() ** float(torch.tensor(p, dtype=torch.float32))
        # elsewhere the table entry, within a unit of its last place, and the product's rounding come to it
        bound = (3.5e-7 if p < 2 else 9e-7) + (0.0 if octave == 0 else 2.0 ** -23 + 2.0 ** -24)
        assert ((odd[:, 0].double() - exact) / exact).abs().max() <= bound
