"""What the planners choose, without a GPU (they then assume 148 SMs).

Splits: the automatic ones of cdist_grad (over k) and kernel_matvec (over m), as their scratch sizes show them: the
planner looks at a few candidates only, and has to find what trying every split finds.

Tiles: the 64 x 64 build kernel is taken where it measured faster than the 128 x 128 one and not elsewhere."""
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


# us on B200, 128 x 128 / 64 x 64 kernel, for the square step
@pytest.mark.parametrize("layout, shape, tile", [
    ("unaligned", (1, 8000, 55, 701), 64),         # 144 / 110
    ("unaligned", (1, 1279, 1279, 127), 64),       # 39 / 33
    ("unaligned", (2, 7954, 55, 33), 64),          # 18.7 / 16.6
    ("unaligned", (2, 7954, 55, 371), 128),        # 82 / 107
    ("unaligned", (1, 2001, 2001, 371), 128),      # 148 / 176
    ("unaligned", (1, 2801, 2801, 129), 128),      # 117 / 127
    ("aligned", (1, 1536, 1536, 256), 64),         # 47.3 / 45.3
    ("aligned", (1, 1536, 1536, 700), 128),        # 111 / 115
    ("aligned", (1, 2112, 2112, 1024), 128),       # 302 / 313
    ("aligned", (1, 2000, 2000, 700), 64),         # 209 / 195
    ("aligned", (1, 2800, 2800, 700), 64),         # 408 / 371
    ("aligned with itself", (1, 1536, 1536, 700), 64),     # 113 / 90
    ("unaligned with itself", (1, 2001, 2001, 701), 64),   # 298 / 201
    ("unaligned with itself", (1, 3601, 3601, 259), 128),  # 190 / 209
    ("rows", (1, 1536, 1536, 1024), 64),           # rows that both kernels read: always the 64 x 64 one
])
def test_build_tile_sizes(layout, shape, tile):
    L, M, N, K = shape
    a = _native.KmBuildArgs()
    a.m, a.n, a.k, a.l = M, N, K, L
    a.a, a.b, a.out = 0x100000, 0x200000, 0x300000
    if layout == "rows":
        a.a_stride_m, a.a_stride_k, a.b_stride_n, a.b_stride_k = K, 1, K, 1
    else:
        pitch = 4 if layout.startswith("aligned") else 5
        a.b = a.a if "itself" in layout else a.b
        a.a_stride_m, a.a_stride_k, a.b_stride_n, a.b_stride_k = 1, _ceil(M, 8) * 8 + pitch, 1, _ceil(N, 8) * 8 + pitch
    a.a_stride_l, a.b_stride_l = (M + 16) * (K + 16) // 4 * 4 * 8, (N + 16) * (K + 16) // 4 * 4 * 8
    a.out_stride_m, a.out_stride_n, a.out_stride_l = 1, M, M * N
    a.inner_power, a.outer_power = _native.POW_SQUARE, _native.POW_SQRT
    assert _native.describe_build(a).split(";")[0].endswith(f"kernel_tile={tile}")
