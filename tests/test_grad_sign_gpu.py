"""GPU parity of the p = 1 tensor-core form of cdist_grad (signs as a matrix operand) against the float64 CPU
oracle.  Reached with contraction="tensor" from 96 rows n on.  Tolerance: max |x - ref| / max |ref| <= 5e-5 as for
the other gradient kernels; where the test is about accuracy it is tighter and says why."""
import pytest
import torch

import kermac_b200 as kermac
from kermac_b200 import _native
from oracle import kermac_oracle as ko

pytestmark = pytest.mark.gpu
TOL = 5e-5


def gen(shape, seed, dist="randn"):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn if dist == "randn" else torch.rand)(*shape, generator=g, dtype=torch.float32)


def inputs(K, M, N, O, seed=3):
    return gen((K, M), seed, "rand"), gen((N, K), seed + 1), gen((O, K), seed + 2), gen((N, M), seed + 3)


def check(a, b, c, d, tol=TOL):
    got = kermac.cdist_grad(a.cuda(), b.cuda(), c.cuda(), d.cuda(), p=1.0, contraction="tensor")
    assert ko.rel_err_signed(got, ko.cdist_grad_ref(a, b, c, d, p=1.0)) < tol
    assert _native.device_error_flag() == 0
    return got


@pytest.mark.parametrize("O", [1, 4, 5, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N", [96, 128, 129])
def test_channel_tiles_and_rows(N, O):
    check(*inputs(70, 13, N, O))


@pytest.mark.parametrize("M", [1, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("O", [3, 20])
def test_columns_around_the_tiles(M, O):
    check(*inputs(100, M, 98, O))


@pytest.mark.parametrize("K", [1, 15, 16, 17, 31, 32, 33, 127, 128, 129, 511, 512, 513, 1600])
@pytest.mark.parametrize("O", [4, 8, 16, 32])
def test_k_extents_around_slabs_and_chains(K, O):
    # 32 k per slab, 512 per accumulation chain, cut at staggered slabs for the columns m of a block
    check(*inputs(K, 9, 100, O))


@pytest.mark.parametrize("K", [36, 260, 3000])
def test_staging_by_tma_and_by_copies_gives_the_same_bits(K):
    a, b, c, d = (t.cuda() for t in inputs(K, 24, 130, 20))
    b_view = torch.zeros(130, K + 1, device="cuda")[:, :K]
    c_view = torch.zeros(20, K + 3, device="cuda")[:, 1:K + 1]
    b_view.copy_(b)
    c_view.copy_(c)
    want = kermac.cdist_grad(a, b, c, d, p=1.0, contraction="tensor")
    for _ in range(3):
        assert torch.equal(want, kermac.cdist_grad(a, b_view, c_view, d, p=1.0, contraction="tensor"))
        assert torch.equal(want, kermac.cdist_grad(a, b, c, d, p=1.0, contraction="tensor"))
    assert _native.device_error_flag() == 0


@pytest.mark.parametrize("O", [4, 24])
def test_same_sign_sums_stay_at_fp32_accuracy(O):
    # 20000 terms of one sign.  A chain adds 32 MMA results, each addition truncating at most 2^-23 of the partial
    # sum, 2e-6 of the chain at the very most; the chains are added in fp32.
    K, M, N = 20000, 12, 100
    a, c = gen((K, M), 24, "rand"), gen((O, K), 25, "rand")
    b, d = gen((N, K), 26, "rand"), gen((N, M), 27, "rand") + 2.0
    check(a, b, c, d, 2e-6)


def test_batches_broadcasting_and_unaligned_output():
    L, K, M, N, O = 2, 90, 18, 100, 6
    a, b, c, d = gen((L, K, M), 20, "rand"), gen((N, K), 21), gen((1, O, K), 22), gen((L, N, M), 23)
    check(a, b, c, d)
    a, b, c, d = inputs(90, 18, 100, 6)
    big = torch.full((6, 100, 20), -3.0, device="cuda")
    got = kermac.cdist_grad(a.cuda(), b.cuda(), c.cuda(), d.cuda(), out=big[:, :, 1:19], p=1.0, contraction="tensor")
    assert ko.rel_err_signed(got, ko.cdist_grad_ref(a, b, c, d, p=1.0)[0]) < TOL
    assert float(big[:, :, 0].max()) == -3.0 and float(big[:, :, -1].max()) == -3.0


def test_ties_infinities_and_nan_as_in_the_fp32_kernel():
    a, b, c, d = inputs(70, 9, 100, 5)
    d = b[:, :1].expand(100, 9).contiguous()          # exact ties count as +1
    check(a, b, c, d)
    a[7, 2], c[1, 40], b[5, 9], d[6, 1] = float("inf"), float("inf"), float("nan"), float("-inf")
    a[8, 3] = float("nan")
    args = [t.cuda() for t in (a, b, c, d)]
    got = kermac.cdist_grad(*args, p=1.0, contraction="tensor")
    want = kermac.cdist_grad(*args, p=1.0, contraction="fp32")
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.isinf(got), torch.isinf(want))
    assert torch.equal(got[torch.isinf(got)], want[torch.isinf(want)])
    finite = torch.isfinite(want)
    assert float((got - want)[finite].abs().max()) < TOL * float(want[finite].abs().max())


@pytest.mark.parametrize("shape", [(300, 33, 64, 9), (257, 500, 130, 24), (400, 64, 70, 40), (256, 31, 200, 4)])
def test_the_automatic_choice_agrees_with_the_fp32_kernel(shape):
    a, b, c, d = (t.cuda() for t in inputs(*shape))
    got, want = (kermac.cdist_grad(a, b, c, d, p=1.0, contraction=k) for k in ("auto", "fp32"))
    # K terms rounded in another order
    assert float((got - want).abs().max()) <= 2.0 ** -23 * shape[0] ** 0.5 * float(want.abs().max())
    assert _native.device_error_flag() == 0


@pytest.mark.parametrize("O", [4, 8, 16, 32])
@pytest.mark.parametrize("shift", [0, 60, 110, 118])
def test_small_products_keep_their_bits(O, shift):
    # kernel values of distant points as weights: the products c * a are normal numbers down to 2^-120 here.  bf16 ends
    # at 2^-133, so pieces that were not scaled up would be 2^-15 of such a product off.  Terms of random sign: a
    # rounded product each and 32 truncating additions per chain stay below 2^-22 of the largest entry.
    K, M, N = 600, 24, 128
    a, b, c, d = inputs(K, M, N, O)
    a, c = (a + 0.5), torch.copysign(c.abs().clamp(0.5, 2.0), c)
    got = kermac.cdist_grad((a * 2.0 ** -shift).cuda(), b.cuda(), c.cuda(), d.cuda(), p=1.0, contraction="tensor")
    ref = ko.cdist_grad_ref(a, b, c, d, p=1.0)
    assert float((got.cpu().double() * 2.0 ** shift - ref).abs().max()) < 2.0 ** -22 * float(ref.abs().max())
    assert _native.device_error_flag() == 0
