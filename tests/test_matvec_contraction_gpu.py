"""Which contraction kernel_matvec takes by itself: |b - a| with few channels goes to the FP32 FMAs, on both sides of each
line of that rule.  The two kernels sum in different orders, so their bits tell which one ran; both are within 5e-5 of
the largest entry of the float64 product."""
import pytest
import torch

import kermac_b200 as kermac

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["rows", "cols"])
@pytest.mark.parametrize("kernel, K, O, expect", [
    ("l1", 7, 1, "fp32"), ("l1", 7, 2, "fp32"), ("l1", 15, 3, "tensor"), ("l1", 16, 3, "fp32"), ("l1", 40, 4, "fp32"),
    ("l1", 40, 5, "tensor"), ("l2", 7, 1, "tensor"), ("l2", 40, 4, "tensor")])
def test_automatic_contraction(kernel, K, O, expect, layout):
    gen = torch.Generator().manual_seed(K * 10 + O)
    points = [torch.randn(*((n, K) if layout == "rows" else (K, n)), generator=gen).cuda() for n in (1500, 260)]
    a, b = points if layout == "rows" else [x.t() for x in points]
    c = torch.randn(O, 1500, generator=gen).cuda()
    desc = kermac.kernel_descriptor_laplace_l1 if kernel == "l1" else kermac.kernel_descriptor_laplace_l2
    got = {name: kermac.kernel_matvec(desc, a, b, c, bandwidth=float(K), contraction=name) for name in ("auto", "fp32", "tensor")}
    assert not torch.equal(got["fp32"], got["tensor"])
    assert torch.equal(got["auto"], got[expect])
    diff = b.double()[:, None] - a.double()[None]
    dist = diff.abs().sum(-1) if kernel == "l1" else diff.square().sum(-1).sqrt()
    want = torch.exp(-dist / K) @ c.double().t()
    assert (got["auto"].reshape(want.shape).double() - want).abs().max() <= 5e-5 * want.abs().max()


@pytest.mark.parametrize("K, O", [(3, 1), (16, 2), (16, 4)])
def test_a_long_sum_in_one_block_is_not_one_chain_of_roundings(K, O):
    """131072 positive terms in one block, taken to the FP32 kernel by the rule above.  Summed tile by tile a running sum is
    rounded 1024 times; as random walks those come to sqrt(1024 / 3) * 0.4 * 2^-24 = 4e-7 of it, and 4e-6 is ten times
    that.  One chain over all terms is rounded 131072 times: 5e-6 in the mean and 1.5e-5 in the worst of these entries."""
    M, N = 131072, 300
    gen = torch.Generator().manual_seed(K + O)
    a, b = torch.randn(M, K, generator=gen).cuda(), torch.randn(N, K, generator=gen).cuda()
    c = (torch.rand(O, M, generator=gen) + 0.5).cuda()
    want = torch.zeros(N, O, dtype=torch.float64, device="cuda")
    for i in range(0, M, 8192):
        dist = (b.double()[:, None] - a[i:i + 8192].double()[None]).abs().sum(-1)
        want += torch.exp(-dist / (1.13 * K)) @ c[:, i:i + 8192].double().t()
    got = {name: kermac.kernel_matvec(kermac.kernel_descriptor_laplace_l1, a, b, c, bandwidth=1.13 * K, split_m=1, contraction=name)
           for name in ("auto", "fp32")}
    assert torch.equal(got["auto"], got["fp32"])
    assert (got["auto"].reshape(want.shape).double() - want).abs().max() <= 4e-6 * want.abs().max()
