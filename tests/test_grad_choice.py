"""Which kernel cdist_grad takes, without a GPU (the planner then assumes 148 SMs).

p = 1 has three: the FP32 kernel, the tensor-core kernel with the weights as the matrix operand, and the one with the
signs."""
import math
import random

import pytest
import torch

from kermac_b200 import _native

pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason="plans for the 148 SMs assumed without a device")
CONTRACTIONS = {"auto": 0, "fp32": 1, "tensor": 2}


def grad_args(K, M, N, O, contraction="auto", split_k=0, pitch=0):
    """Arguments of a p = 1 gradient; `pitch`: extra elements per row of b and c (rows of K + pitch a multiple of 4 can
    be copied 16 bytes at a time)."""
    g = _native.KmGradArgs()
    g.m, g.n, g.o, g.k, g.l = M, N, O, K, 1
    g.a = g.b = g.c = g.d = g.out = 0x1000
    g.lda = g.ldd = g.out_stride_n = M
    g.ldb = g.ldc = K + pitch
    g.out_stride_o = N * M
    g.norm_type, g.p = _native.NORM_L1, _native.hyper(1.0)
    g.split_k, g.contraction = split_k, CONTRACTIONS[contraction]
    return g


def described(g):
    """{'kernel': 'sign', 'channels': '32', ...}"""
    return dict(word.split("=") for word in _native.describe_grad(g).split()[1:])


@pytest.mark.parametrize("contraction", ["auto", "tensor"])
def test_a_launch_has_at_most_65535_channel_chunks(contraction):
    # a chunk of the sign kernel is half of one of the weights kernel: between the two limits only the latter can run
    for O in (32 * 65535, 32 * 65535 + 1, 64 * 65535):
        plan = described(grad_args(2560, 8, 128, O, contraction))
        assert plan["kernel"] == "weights" or O == 32 * 65535, (O, plan)
        assert int(plan["chunks"]) <= 65535, (O, plan)
    with pytest.raises(ValueError, match="too many output channels"):
        _native.describe_grad(grad_args(2560, 8, 128, 64 * 65535 + 1, contraction))


# us on B200, sign kernel / the other one (FP32 up to 16 channels, weights from 17 on).  The rule's line was drawn with an
# earlier sign kernel and moved by less than its times fell since: rows marked * keep the other kernel although the
# sign kernel is the faster one there.
@pytest.mark.parametrize("contraction, pitch, shape, sign", [
    ("auto", 0, (256, 4096, 1000, 4), False),         # 328 / 221: a block's start and end weigh more than its 8 slabs
    ("auto", 0, (320, 4096, 1000, 3), False),         # 358 / 273
    ("auto", 0, (256, 4096, 128, 4), False),          # 47 / 35
    ("auto", 0, (256, 4096, 1000, 64), False),        # * 1559 / 1647: the result does not fit L2
    ("auto", 0, (1024, 1000, 64, 32), False),         # * 55 / 60: half of the block's 128 rows are empty
    ("auto", 0, (8192, 1000, 64, 4), False),          # 172 / 124
    ("auto", 0, (512, 250, 500, 64), False),          # * 100 / 105: rows of 250 results are not stored 16 bytes at a time
    ("auto", 0, (256, 250, 1000, 64), False),         # 139 / 115
    ("auto", 0, (30000, 4096, 256, 2), False),        # * 4311 / 4443
    ("auto", 1, (8192, 1000, 1000, 4), False),        # * 1496 / 1723: b in rows that are copied word by word
    ("auto", 1, (1024, 1000, 64, 16), False),         # * 55 / 62
    ("auto", 0, (3000, 4096, 320, 4), False),         # * 736 / 832
    ("auto", 0, (255, 1000, 1000, 32), False),        # below 256 k: never
    ("auto", 0, (30000, 4096, 63, 32), False),        # below 64 rows: never
    ("auto", 0, (1024, 1000, 1000, 4), True),         # 181 / 250
    ("auto", 0, (8192, 1000, 1000, 4), True),         # 1201 / 1723
    ("auto", 0, (30000, 4096, 256, 3), True),         # 4313 / 6221
    ("auto", 0, (30000, 4096, 256, 4), True),         # 4314 / 6225
    ("auto", 0, (256, 1000, 1000, 16), True),         # 133 / 182
    ("auto", 0, (256, 1000, 1000, 32), True),         # 180 / 273
    ("auto", 0, (8192, 64, 128, 16), True),           # 26 / 53
    ("auto", 0, (30000, 4096, 256, 32), True),        # 8993 / 22054
    ("auto", 0, (8192, 1000, 320, 64), True),         # 1954 / 2629
    ("auto", 1, (8192, 1000, 1000, 16), True),        # 2780 / 5491
    ("auto", 1, (1024, 1000, 128, 32), True),         # 80 / 123
    ("fp32", 0, (30000, 4096, 256, 32), False),
    ("tensor", 0, (30000, 4096, 95, 32), False),      # a named tensor-core contraction: from 96 rows on ...
    ("tensor", 0, (30000, 4096, 96, 32), True),
    ("tensor", 1, (3000, 24, 130, 20), True),         # 17 / 20
    ("tensor", 1, (2048, 250, 160, 64), False),       # ... unless it costs much: 155 / 150
    ("tensor", 0, (30000, 4096, 129, 40), False),     # 17694 / 15911
    ("tensor", 0, (64, 4096, 1000, 32), False),       # 579 / 519
])
def test_the_sign_kernel_is_taken_where_it_measured_faster(contraction, pitch, shape, sign):
    assert (described(grad_args(*shape, contraction, pitch=pitch))["kernel"] == "sign") == sign


def test_splits_stay_within_the_scratch_that_callers_are_asked_for():
    rng, seen = random.Random(3), set()
    size = lambda low, high: int(math.exp(rng.uniform(math.log(low), math.log(high + 1))))       # noqa: E731
    for _ in range(400):
        K, M, N, O = size(1, 100000), size(1, 5000), size(1, 1000), size(1, 70)
        g = grad_args(K, M, N, O, rng.choice(("auto", "tensor")), pitch=rng.choice((0, 1)))
        plan = described(g)
        told = max(1, _native.lib().kermac_b200_cdist_grad_scratch_bytes(g) // (4 * M * N * O))
        assert 1 <= int(plan["splits"]) <= told and (plan["kernel"] == "sign" or int(plan["splits"]) == told)
        seen.add(plan["kernel"])
        for split_k in (1, 3):                                       # the kernel does not follow the split that is asked for
            g.split_k = split_k
            assert described(g) == dict(plan, splits=str(split_k))
        g.split_k, g.out, g.out_stride_n, g.out_stride_o = 0, 0x1004, M + 1, N * (M + 1)     # nor where the result goes
        assert described(g) == plan
    assert seen == {"fp32", "weights", "sign"}
