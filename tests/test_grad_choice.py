"""Which kernel cdist_grad takes, without a GPU (the planner then assumes 148 SMs).

p = 1 has three: the FP32 kernel, the tensor-core kernel with the weights as the matrix operand, and the one with the
signs."""
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
