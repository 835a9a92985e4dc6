"""GPU parity of the p = 1 tensor-core form of cdist_grad (signs as a matrix operand) against the float64 CPU
oracle.  Reached with contraction="tensor" from 96 rows n on (unless the other kernel is much faster; every call here
checks which kernel it gets).  Tolerance: max |x - ref| / max |ref| <= 5e-5 as for the other gradient kernels; where the
test is about accuracy it is tighter and says why."""
import ctypes

import pytest
import torch

import kermac_b200 as kermac
from kermac_b200 import _native
from kermac_b200.cdist_grad import _marshal_grad
from oracle import kermac_oracle as ko

pytestmark = pytest.mark.gpu
TOL = 5e-5


def gen(shape, seed, dist="randn"):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn if dist == "randn" else torch.rand)(*shape, generator=g, dtype=torch.float32)


def inputs(K, M, N, O, seed=3):
    return gen((K, M), seed, "rand"), gen((N, K), seed + 1), gen((O, K), seed + 2), gen((N, M), seed + 3)


def arguments(a, b, c, d, out, contraction="tensor", split_k=0):
    """The C-ABI arguments of a call on 2-D or batched operands."""
    g, _ = _marshal_grad(a, b, c, d, out, 1.0, contraction)
    g.split_k = split_k
    return g


def takes_sign(g):
    return "kernel=sign" in _native.describe_grad(g)


def check(a, b, c, d, tol=TOL):
    got = kermac.cdist_grad(a.cuda(), b.cuda(), c.cuda(), d.cuda(), p=1.0, contraction="tensor")
    assert takes_sign(arguments(a.cuda(), b.cuda(), c.cuda(), d.cuda(), got))
    assert ko.rel_err_signed(got, ko.cdist_grad_ref(a, b, c, d, p=1.0)) < tol
    assert _native.device_error_flag() == 0
    return got


def with_split(a, b, c, d, split_k):
    """The sums in `split_k` pieces of k (operands on the device)."""
    out = torch.full((c.shape[0], b.shape[0], a.shape[1]), float("nan"), device="cuda")
    g = arguments(a, b, c, d, out, split_k=split_k)
    assert takes_sign(g)
    need = _native.lib().kermac_b200_cdist_grad_scratch_bytes(ctypes.byref(g))
    scratch = torch.full((max(1, need // 4),), float("nan"), device="cuda")
    g.scratch, g.scratch_bytes = scratch.data_ptr(), need
    _native.launch_grad(g, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return out


def unaligned(t):
    """The same numbers in rows that are not 16-byte aligned."""
    view = torch.zeros(t.shape[0], t.shape[1] + (3 - t.shape[1]) % 4, device="cuda")[:, :t.shape[1]]
    view.copy_(t)
    return view


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
def test_k_extents_around_slabs(K, O):
    # 32 k per slab; the automatic split leaves a block one slab to a few
    check(*inputs(K, 9, 100, O))


@pytest.mark.parametrize("K", [511, 512, 513, 544, 1024, 1600, 5001])
@pytest.mark.parametrize("O", [4, 8, 16, 32])
def test_k_extents_around_chains_and_rings(K, O):
    # a single pass: 512 k per accumulation chain, cut at staggered slabs for the columns m of a block, and every ring of
    # barriers (4 slabs at most) goes round many times; then three pieces with a short last one
    a, b, c, d = inputs(K, 9, 100, O)
    ref = ko.cdist_grad_ref(a, b, c, d, p=1.0)[0]
    a, b, c, d = a.cuda(), b.cuda(), c.cuda(), d.cuda()
    views = unaligned(b), unaligned(c)
    for split_k in (1, 3):
        got = with_split(a, b, c, d, split_k)
        assert ko.rel_err_signed(got, ref) < TOL
        assert torch.equal(got, with_split(a, *views, d, split_k))      # staged by copies of 4 bytes
    assert _native.device_error_flag() == 0


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
    # in one pass 40 chains: their sum rounds by 2^-25 of a partial sum, half of the result on average, each time
    got = with_split(a.cuda(), b.cuda(), c.cuda(), d.cuda(), 1)
    assert ko.rel_err_signed(got, ko.cdist_grad_ref(a, b, c, d, p=1.0)[0]) < 2e-6 + 40 * 2.0 ** -26


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


@pytest.mark.parametrize("O", [4, 8, 16, 32])
def test_values_that_are_not_finite_stay_in_their_sums(O):
    # over several chains of 512 k: infinities of one and of both signs, products that overflow, and a NaN whose payload
    # is lost when it is cut to bf16
    a, b, c, d = inputs(1600, 9, 100, O)
    a[7, 2] = float("inf")
    a[40, 3], a[900, 3] = float("inf"), float("-inf")
    a[1100, 5], c[1, 1100] = 1e30, 1e30
    a.view(torch.int32)[1300, 6] = 0x7F800001
    c[O - 1, 60] = float("nan")
    a, b, c, d = (t.cuda() for t in (a, b, c, d))
    got = with_split(a, b, c, d, 1)
    want = kermac.cdist_grad(a, b, c, d, p=1.0, contraction="fp32")[0]
    finite = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), finite) and torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
    assert 0 < int(finite.sum()) and float((got - want)[finite].abs().max()) < TOL * float(want[finite].abs().max())
    assert _native.device_error_flag() == 0


@pytest.mark.parametrize("shape, sign", [
    ((300, 33, 64, 9), False), ((257, 500, 130, 24), False), ((400, 64, 70, 40), False), ((256, 31, 200, 4), True),
    ((1000, 1000, 128, 3), True), ((1024, 130, 100, 16), True), ((4096, 250, 128, 24), True), ((2048, 250, 128, 32), True),
    ((1024, 130, 256, 64), True)])
def test_the_automatic_choice_agrees_with_the_fp32_kernel(shape, sign):
    a, b, c, d = (t.cuda() for t in inputs(*shape))
    got, want = (kermac.cdist_grad(a, b, c, d, p=1.0, contraction=k) for k in ("auto", "fp32"))
    assert takes_sign(arguments(a, b, c, d, got, "auto")) == sign
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
