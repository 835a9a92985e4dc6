"""The automatic splits of cdist_grad (over k) and kernel_matvec (over m), as their scratch sizes show them: the
planner looks at a few candidates only, and has to find what trying every split finds.  No GPU: the planner then
assumes 148 SMs."""
import ctypes
import math
import random
import time

import numpy as np
import pytest
import torch

from kermac_b200 import _native

SMS = 148


def _choose(cost, last):
    s = np.arange(1, last + 1, dtype=np.float64)
    c = cost(s)
    return int(s[np.argmax(c <= 1.005 * c.min())])


def _ceil(a, b):
    return -(-a // b)


def _grad_args(K, M, N, O, p):
    g = _native.KmGradArgs()
    g.m, g.n, g.o, g.k, g.l = M, N, O, K, 1
    g.a = g.b = g.c = g.d = g.out = 0x1000
    g.lda = g.ldd = g.out_stride_n = M
    g.ldb = g.ldc = K
    g.out_stride_o = N * M
    g.norm_type = {1.0: _native.NORM_L1, 2.0: _native.NORM_L2}.get(p, _native.NORM_P)
    g.p = _native.hyper(p)
    return g


def _grad_splits(g):
    return max(1, _native.lib().kermac_b200_cdist_grad_scratch_bytes(ctypes.byref(g)) // (4 * g.m * g.n * g.o))


def _grad_rule(K, M, N, O, p):
    tensor = O >= 17 and K >= 256
    ot = (64 if O > 32 else 32) if tensor else next(x for x in (1, 2, 4, 8, 16) if x >= min(O, 16))
    nt = 4 if ot <= 4 else 2 if ot == 8 else 1
    tm, tn = (32, 8 if ot == 64 else 16) if tensor else (64, 16 * nt)
    blocks, slabs, size = _ceil(M, tm) * _ceil(N, tn) * _ceil(O, ot), _ceil(K, 32), 4.0 * O * N * M
    slab_us = 2.0 if tensor else 0.6 + 0.16 * nt * (1 + ot) + (0.0 if p in (1.0, 2.0) else (0.5 if p == 1.5 else 1.4) * nt)

    def cost(s):
        per = _ceil(slabs, s)
        share = _ceil(blocks * _ceil(slabs, per), SMS)
        units = share if tensor else 0.9 * share + np.where(share % 2 == 1, 0.1, 0.0)
        return units * per * slab_us + 2.5 * share + np.where(s > 1, 3.0 + (2.0 * s + 1.0) * size / 5e6, 0.0)

    last = max(1, min(slabs, 16 * SMS // blocks, int(512e6 / size)))
    return _choose(cost, last)


def _matvec_args(M, N, K, O):
    g = _native.KmMatvecArgs()
    g.m, g.n, g.k, g.o, g.l = M, N, K, O, 1
    g.a = g.b = g.c = g.y = 0x1000
    g.a_stride_m, g.a_stride_k, g.b_stride_n, g.b_stride_k = 1, _ceil(M, 4) * 4, 1, _ceil(N, 4) * 4
    g.ldc, g.y_stride_n, g.y_stride_o = M, O, 1
    g.inner_power, g.outer_power, g.kernel_type = _native.POW_SQUARE, _native.POW_SQRT, _native.KERNEL_LAPLACE
    g.bandwidth = _native.hyper(1.0)
    return g


def _matvec_splits(g):
    return max(1, _native.lib().kermac_b200_kernel_matvec_scratch_bytes(ctypes.byref(g)) // (4 * g.n * g.o))


def _matvec_rule(M, N, K, O):
    blocks, chunks = _ceil(N, 128) * _ceil(O, 16), _ceil(M, 128)

    def cost(s):
        per = _ceil(chunks, s)
        share = _ceil(blocks * _ceil(chunks, per), SMS)
        return ((0.9 * share + np.where(share % 2 == 1, 0.12, 0.0)) * per * (4.5 + 0.155 * K) + 1.5 * share +
                np.where(s > 1, 3.0 + 0.05 * s, 0.0))

    last = max(1, min(chunks, 32 * SMS // blocks, (512 << 20) // (N * O * 4)))
    return _choose(cost, last)


pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason="plans for the 148 SMs assumed without a device")


def test_splits_are_those_of_the_whole_search():
    rng = random.Random(11)
    size = lambda low, high: int(math.exp(rng.uniform(math.log(low), math.log(high + 1))))       # noqa: E731
    several = 0
    for _ in range(400):
        shape = (size(1, 300000), size(1, 5000), size(1, 1000), size(1, 70), rng.choice((1.0, 1.5, 2.0, 1.7)))
        got = _grad_splits(_grad_args(*shape))
        assert got == _grad_rule(*shape), shape
        several += got > 1
        shape = (size(1, 1000000), size(1, 20000), size(1, 700), size(1, 40))
        got = _matvec_splits(_matvec_args(*shape))
        assert got == _matvec_rule(*shape), shape
        several += got > 1
    assert several > 200


def test_planning_stays_cheap_for_long_sums():
    grad, matvec = _grad_args(1000000, 64, 16, 4, 1.0), _matvec_args(1000000, 100, 64, 1)
    for plan in (lambda: _grad_splits(grad), lambda: _matvec_splits(matvec)):
        best = math.inf
        for _ in range(200):
            began = time.perf_counter()
            plan()
            best = min(best, time.perf_counter() - began)
        assert best < 20e-6        # (every split tried: 33 and 58 us where this takes 8 and 5)
