// kermac_b200_cdist_grad: the p-norm gradient contraction
//   out[l, o, n, m] = sum_k c[l, o, k] * a[l, k, m] * g(d[l, n, m] - b[l, n, k])
// restating what the reference's kernel_cute_p_norm_kernel_gradient computes
// (include/p_norm_gradient.cuh:22-405) with a different work decomposition:
//   - a thread block owns a 64 (m) x TN (n) tile for up to OT output channels, with
//     OT chosen from {1, 2, 4, 8, 16} to fit O (the reference always spends 32);
//   - the weight w = a * g(diff) is formed once per (m, n, k) and reused for every
//     channel; for p = 1 the sign is applied with one bit operation on a;
//   - differences, weights and channel FMAs run on packed pairs along m;
//   - the contracted k range can be split over several thread blocks, whose partial
//     tiles go to caller-provided scratch and are summed in a fixed order by a
//     second kernel, so results do not depend on scheduling.  The split is the one with
//     the least estimated time (preferred_split);
//   - blocks that share a tile of the weight matrix a (the n-tiles of one m-column and
//     k range) are neighbours in launch order, so a is read from DRAM once;
//   - p = 1.5 takes |x|^(p-1) as one sqrt.approx instead of the lg2 / ex2 pair.
#include <algorithm>
#include <mutex>

#include "km_common.cuh"
#include "km_host.h"

namespace km {
namespace {

constexpr int G_THREADS = 256;
constexpr int G_TM      = 64;
constexpr int G_BK      = 32;   // k rows per staged slab (a multiple of 8)
constexpr int G_STAGES  = 3;
constexpr int G_UNROLL  = 32;   // k rows of a slab unrolled together
// Kernel-side norm kinds: the three of the C-ABI plus the square-root form of KM_NORM_P
// for p - 1 == 0.5, chosen by the launcher when p is a host scalar.
constexpr int G_NORM_SQRT = 3;
static_assert(G_NORM_SQRT == GT_NORM_SQRT && G_BK == GT_BK, "the two gradient kernels share the planner");
// Channels from which KM_CONTRACT_AUTO takes the tensor-core kernel.
constexpr int KM_GRAD_TENSOR_MIN_O = 17;

struct GradParams {
    int M, N, O, K, L;
    const float* A; long long lda, a_sl;
    const float* B; long long ldb, b_sl;
    const float* C; long long ldc, c_sl;
    const float* D; long long ldd, d_sl;
    float*       E; long long e_sn, e_so, e_sl;   // destination (out, or scratch when split)
    KmHyper p;
    int tiles_m, tiles_n, o_chunks, splits;
    int k_per_split;                                // multiple of G_BK
    long long split_stride;                         // elements between partial results of consecutive splits
    int a_vec, e_vec;
};

__device__ __forceinline__ u64 flip_sign2(u64 a, u64 diff) {
    // a with the sign bit of diff xor-ed in, lane-wise: copysign(1, diff) * a
    return a ^ (diff & 0x8000000080000000ull);
}

// Thread blocks resident per SM that every tile shape is compiled for.
constexpr int grad_min_blocks(int, int) { return 2; }

template <int NORM, int OT, int NT>
__global__ void __launch_bounds__(G_THREADS, grad_min_blocks(OT, NT)) grad_kernel(const __grid_constant__ GradParams p) {
    constexpr int TN      = 16 * NT;
    constexpr int PITCH_A = G_TM + 4;
    constexpr int PITCH_B = TN + 4;
    constexpr int PITCH_C = (OT < 4 ? 4 : OT);
    constexpr int STAGE_FLOATS = G_BK * (PITCH_A + PITCH_B + PITCH_C);
    extern __shared__ __align__(16) float smem[];      // G_STAGES * STAGE_FLOATS floats (grad_smem_bytes)

    const int tid = threadIdx.x;
    const int tmi = tid & 15, tni = tid >> 4;
    after_previous_grid();

    // n-tiles fastest: the blocks that read the same (k range, m-column) tile of a run together
    int bx          = blockIdx.x;
    const int tn    = bx % p.tiles_n; bx /= p.tiles_n;
    const int split = bx % p.splits;  bx /= p.splits;
    const int tm    = bx;
    const int oc    = blockIdx.y;
    const int l     = blockIdx.z;
    const int m0 = tm * G_TM, n0 = tn * TN, o0 = oc * OT;

    const int k_begin = split * p.k_per_split;
    const int k_end   = min(p.K, k_begin + p.k_per_split);
    const int ktiles  = (k_end > k_begin) ? (k_end - k_begin + G_BK - 1) / G_BK : 0;

    const float* A = p.A + (long long)l * p.a_sl + m0;
    const float* B = p.B + (long long)l * p.b_sl + (long long)n0 * p.ldb;
    const float* C = p.C + (long long)l * p.c_sl + (long long)o0 * p.ldc;
    const float* D = p.D + (long long)l * p.d_sl;

    float pm1 = 0.0f;
    if (NORM == KM_NORM_P) pm1 = read_hyper(p.p, l) - 1.0f;

    // d values of this thread: rows n0 + tni * NT + j, columns m0 + tmi * 4 + {0..3}
    u64 dv[NT][2];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        const int n = n0 + tni * NT + j;
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int m = m0 + tmi * 4 + e;
            v[e]        = (n < p.N && m < p.M) ? D[(long long)n * p.ldd + m] : 0.0f;
        }
        dv[j][0] = pack2(v[0], v[1]);
        dv[j][1] = pack2(v[2], v[3]);
    }

    u64 acc[NT][OT][2];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int o = 0; o < OT; ++o) acc[j][o][0] = acc[j][o][1] = 0ull;

    auto stage = [&](int s, int kt) {
        float* sa = smem + s * STAGE_FLOATS;
        float* sb = sa + G_BK * PITCH_A;
        float* sc = sb + G_BK * PITCH_B;
        const int k0 = k_begin + kt * G_BK;
        if (p.a_vec) {
            // G_BK k rows x 16 chunks of 4 m
#pragma unroll
            for (int i = 0; i < (G_BK * G_TM / 4) / G_THREADS; ++i) {
                const int idx = tid + i * G_THREADS;
                const int kk = idx >> 4, t = (idx & 15) << 2, gk = k0 + kk;
                int valid = min(4, p.M - m0 - t);
                valid     = (gk < k_end && valid > 0) ? valid : 0;
                cp_async_16(smem_u32(sa + kk * PITCH_A + t), valid ? A + (long long)gk * p.lda + t : p.A, valid * 4);
            }
        } else {
#pragma unroll
            for (int i = 0; i < (G_BK * G_TM) / G_THREADS; ++i) {
                const int idx = tid + i * G_THREADS;
                const int t = idx & (G_TM - 1), kk = idx >> 6, gk = k0 + kk;
                const bool ok = gk < k_end && (m0 + t) < p.M;
                cp_async_4(smem_u32(sa + kk * PITCH_A + t), ok ? A + (long long)gk * p.lda + t : p.A, ok ? 4 : 0);
            }
        }
        // b and c are k-contiguous in global memory and staged k-major.  A warp copies 8
        // consecutive k of 4 rows: 32-byte runs on the global side, and on the shared side
        // banks 4 kk + t (pitches are 4 mod 32 or 20), all different, so the 4-byte writes
        // do not collide.
        constexpr int K8 = G_BK / 8;
#pragma unroll
        for (int i = 0; i < (G_BK * TN + G_THREADS - 1) / G_THREADS; ++i) {
            const int idx = tid + i * G_THREADS;
            if (idx < G_BK * TN) {
                const int kk = (idx & 7) + ((idx >> 5) % K8) * 8;
                const int t  = ((idx >> 3) & 3) + (idx / (32 * K8)) * 4;
                const int gk = k0 + kk;
                const bool ok = gk < k_end && (n0 + t) < p.N;
                cp_async_4(smem_u32(sb + kk * PITCH_B + t), ok ? B + (long long)t * p.ldb + gk : p.B, ok ? 4 : 0);
            }
        }
        constexpr int C_ROWS = (OT < 4 ? 4 : OT);
#pragma unroll
        for (int i = 0; i < (G_BK * C_ROWS + G_THREADS - 1) / G_THREADS; ++i) {
            const int idx = tid + i * G_THREADS;
            if (idx < G_BK * C_ROWS) {
                const int kk = (idx & 7) + ((idx >> 5) % K8) * 8;
                const int t  = ((idx >> 3) & 3) + (idx / (32 * K8)) * 4;
                const int gk = k0 + kk;
                const bool ok = gk < k_end && (o0 + t) < p.O;
                if (t < OT) cp_async_4(smem_u32(sc + kk * PITCH_C + t), ok ? C + (long long)t * p.ldc + gk : p.C, ok ? 4 : 0);
            }
        }
    };

    auto step = [&](const float* sa, const float* sb, const float* sc, int kk) {
        const ulonglong2 a4 = *reinterpret_cast<const ulonglong2*>(sa + kk * PITCH_A + tmi * 4);
        const u64 av[2]     = {a4.x, a4.y};
        // b and c rows of this k: 128-bit shared loads where the tile shape allows
        float bv[NT];
        if constexpr (NT == 4) {
            const float4 b4 = *reinterpret_cast<const float4*>(sb + kk * PITCH_B + tni * 4);
            bv[0] = b4.x; bv[1] = b4.y; bv[2] = b4.z; bv[3] = b4.w;
        } else if constexpr (NT == 2) {
            const float2 b2 = *reinterpret_cast<const float2*>(sb + kk * PITCH_B + tni * 2);
            bv[0] = b2.x; bv[1] = b2.y;
        } else {
            bv[0] = sb[kk * PITCH_B + tni];
        }
        float cv[OT];
        if constexpr (OT >= 4) {
#pragma unroll
            for (int o = 0; o < OT; o += 4) {
                const float4 c4 = *reinterpret_cast<const float4*>(sc + kk * PITCH_C + o);
                cv[o] = c4.x; cv[o + 1] = c4.y; cv[o + 2] = c4.z; cv[o + 3] = c4.w;
            }
        } else {
#pragma unroll
            for (int o = 0; o < OT; ++o) cv[o] = sc[kk * PITCH_C + o];
        }
        u64 cd[OT];
#pragma unroll
        for (int o = 0; o < OT; ++o) cd[o] = pack2(cv[o], cv[o]);
        // Order of the 8 (n, m-pair) x OT channel FMAs of a k row.  They all cost the same in theory;
        // in practice the order decides which source operands repeat from one instruction to the next
        // and how the compiler lays the registers out, and a few per cent hang on it.  Measured at
        // K = 30000, M = 4096, N = 256, O = 4 (ms, orders: 0 = weight by weight as it is computed, then
        // with all weights of the row first, 1 = channel / n / pair, 3 = pair / channel / n):
        //   p = 1:   0: 6.45   1: 6.24   3: 6.39        p = 2:   0: 6.37   1: 6.25   3: 6.21
        //   p = 1.5: 0: 8.72   1: 8.82   3: 8.66        p = 1.7: 0: 14.84  1: 15.78  3: 15.06
        // With the two multiplicands exchanged (weight first, coefficient second) order 1 falls back to 6.9 ms:
        // what pays is the FIRST source repeating over a long run of instructions (the coefficient pair over
        // all 8 weights of the row).  With 8 and 16 channels a coefficient pair still meets 4 and 2 weights (orders 0 / 1 / 3,
        // us, K = 4000, M = 2000, N = 256): 16 channels, p = 2 1442 / 1349 / 1444, p = 1.5 1442 / 1437 / 1442; K = 64,
        // 1000^2, p = 2 56.2 / 52.1 / 56.8, p = 1.7 60.1 / 58.8 / 60.6; 8 channels, p = 1.5 896 / 880 / 890, p = 2 719 / 723 /
        // 745.  1 and 2 channels measured no difference and keep order 0.
        constexpr int ORDER = OT >= 8 ? (OT == 8 && NORM == KM_NORM_L2 ? 0 : 1) : (OT != 4) ? 0 : (NORM == KM_NORM_L1 ? 1 : ((NORM == KM_NORM_L2 || NORM == G_NORM_SQRT) ? 3 : 0));
        if constexpr (ORDER == 0) {
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const u64 bd = pack2(bv[j], bv[j]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const u64 diff = sub2(dv[j][h], bd);
                u64 w;
                if constexpr (NORM == KM_NORM_L1) {
                    w = flip_sign2(av[h], diff);
                } else if constexpr (NORM == KM_NORM_L2) {
                    w = mul2(av[h], diff);
                } else if constexpr (NORM == G_NORM_SQRT) {
                    // |x|^(1/2) sign(x): one MUFU operation per element instead of two
                    float d0, d1;
                    unpack2(diff, d0, d1);
                    w = flip_sign2(mul2(av[h], pack2(sqrt_approx(fabsf(d0)), sqrt_approx(fabsf(d1)))), diff);
                } else {
                    float d0, d1;
                    unpack2(diff, d0, d1);
                    if (h == 0 && (j & 1) == 0 && NT > 1) {
                        // one pair in four takes only lg2 on MUFU and the exponential on the
                        // FP32 pipe (ex2_poly2); more than that and instruction issue, not MUFU,
                        // becomes the limit
                        const u64 x = mul2(pack2(lg2_approx(fabsf(d0)), lg2_approx(fabsf(d1))), pack2(pm1, pm1));
                        float x0, x1;
                        unpack2(x, x0, x1);
                        u64 r, scale;
                        ex2_poly2(x0, x1, r, scale);
                        w = mul2(av[h], flip_sign2(mul2(r, scale), diff));
                    } else {
                        const float g0 = copysignf(pow_approx(fabsf(d0), pm1), d0);
                        const float g1 = copysignf(pow_approx(fabsf(d1), pm1), d1);
                        w              = mul2(av[h], pack2(g0, g1));
                    }
                }
#pragma unroll
                // A packed FMA whose three sources are three different register pairs (coefficient,
                // weight, accumulator) holds the FP32 pipe for about three cycles instead of two, which
                // is what bounds this loop (32 of them and 8 packed subtracts per k row: ~112 cycles for
                // 80 cycles of arithmetic).  Scalar FMAs (two per pair) and a half packed / half scalar
                // mix both measured slower: 7.5 and 7.0 ms against 6.6.
                for (int o = 0; o < OT; ++o) acc[j][o][h] = fma2(cd[o], w, acc[j][o][h]);
            }
        }
        } else {
            u64 wv[NT][2];
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const u64 bd = pack2(bv[j], bv[j]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                const u64 diff = sub2(dv[j][h], bd);
                u64 w;
                if constexpr (NORM == KM_NORM_L1) {
                    w = flip_sign2(av[h], diff);
                } else if constexpr (NORM == KM_NORM_L2) {
                    w = mul2(av[h], diff);
                } else if constexpr (NORM == G_NORM_SQRT) {
                    // |x|^(1/2) sign(x): one MUFU operation per element instead of two
                    float d0, d1;
                    unpack2(diff, d0, d1);
                    w = flip_sign2(mul2(av[h], pack2(sqrt_approx(fabsf(d0)), sqrt_approx(fabsf(d1)))), diff);
                } else {
                    float d0, d1;
                    unpack2(diff, d0, d1);
                    if (h == 0 && (j & 1) == 0 && NT > 1) {
                        // one pair in four takes only lg2 on MUFU and the exponential on the
                        // FP32 pipe (ex2_poly2); more than that and instruction issue, not MUFU,
                        // becomes the limit
                        const u64 x = mul2(pack2(lg2_approx(fabsf(d0)), lg2_approx(fabsf(d1))), pack2(pm1, pm1));
                        float x0, x1;
                        unpack2(x, x0, x1);
                        u64 r, scale;
                        ex2_poly2(x0, x1, r, scale);
                        w = mul2(av[h], flip_sign2(mul2(r, scale), diff));
                    } else {
                        const float g0 = copysignf(pow_approx(fabsf(d0), pm1), d0);
                        const float g1 = copysignf(pow_approx(fabsf(d1), pm1), d1);
                        w              = mul2(av[h], pack2(g0, g1));
                    }
                }
                    wv[j][h] = w;
                }
            }
            if constexpr (ORDER == 1) {
#pragma unroll
                for (int o = 0; o < OT; ++o)
#pragma unroll
                    for (int j = 0; j < NT; ++j)
#pragma unroll
                        for (int h = 0; h < 2; ++h) acc[j][o][h] = fma2(cd[o], wv[j][h], acc[j][o][h]);
            } else {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int o = 0; o < OT; ++o)
#pragma unroll
                        for (int j = 0; j < NT; ++j) acc[j][o][h] = fma2(cd[o], wv[j][h], acc[j][o][h]);
            }
        }
    };

#pragma unroll
    for (int s = 0; s < G_STAGES - 1; ++s) {
        if (s < ktiles) stage(s, s);
        cp_async_commit();
    }
    for (int kt = 0; kt < ktiles; ++kt) {
        cp_async_wait<G_STAGES - 2>();
        __syncthreads();
        const int nk = kt + G_STAGES - 1;
        if (nk < ktiles) stage(nk % G_STAGES, nk);
        cp_async_commit();
        const float* sa = smem + (kt % G_STAGES) * STAGE_FLOATS;
        const float* sb = sa + G_BK * PITCH_A;
        const float* sc = sb + G_BK * PITCH_B;
        const int kvalid = k_end - (k_begin + kt * G_BK);
        if (kvalid >= G_BK) {
            // The whole 32-row slab unrolled measured fastest (6.45 ms against 6.58 with 16-row slabs
            // and 6.65 with an unroll of 8 at K = 30000, M = 4096, N = 256, O = 4); the handful of
            // registers that spill are reloaded about four times per slab, not per k row.
#pragma unroll G_UNROLL
            for (int kk = 0; kk < G_BK; ++kk) step(sa, sb, sc, kk);
        } else {
#pragma unroll 1
            for (int kk = 0; kk < kvalid; ++kk) step(sa, sb, sc, kk);
        }
    }
    cp_async_wait<0>();

    float* E = p.E + (long long)split * p.split_stride + (long long)l * p.e_sl;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        const int n = n0 + tni * NT + j;
        if (n >= p.N) continue;
#pragma unroll
        for (int o = 0; o < OT; ++o) {
            if (o0 + o >= p.O) continue;
            float* row = E + (long long)(o0 + o) * p.e_so + (long long)n * p.e_sn;
            const int m = m0 + tmi * 4;
            float v[4];
            unpack2(acc[j][o][0], v[0], v[1]);
            unpack2(acc[j][o][1], v[2], v[3]);
            if (p.e_vec && m + 3 < p.M) {
                *reinterpret_cast<float4*>(row + m) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (m + e < p.M) row[m + e] = v[e];
            }
        }
    }
}

// out[l][o][n][m] = sum over splits of partial[split][l][o][n][m] (dense partials), in split order.  Bound by
// reading the partials: indices are 32-bit wherever they fit, because the 64-bit divisions take longer than the
// loads, and four splits are loaded ahead of the adds.
template <typename Index>
__global__ void __launch_bounds__(256) grad_reduce_kernel(const float* partial, float* out,
                                                          int M, int N, int O, int L, int splits, long long split_stride,
                                                          long long o_sn, long long o_so, long long o_sl) {
    after_previous_grid();
    const Index total = (Index)L * O * N * M;
    const Index step  = (Index)gridDim.x * blockDim.x;
    for (Index i = blockIdx.x * (Index)blockDim.x + threadIdx.x; i < total; i += step) {
        float s = 0.0f;
#pragma unroll 4
        for (int sp = 0; sp < splits; ++sp) s += partial[sp * split_stride + i];
        Index r = i;
        const Index m = r % M; r /= M;
        const Index n = r % N; r /= N;
        const Index o = r % O; r /= O;
        out[(long long)r * o_sl + (long long)o * o_so + (long long)n * o_sn + m] = s;
    }
}

typedef void (*GradFn)(const GradParams);

struct GradChoice {
    GradFn fn;
    int    smem_bytes;
};

constexpr int grad_smem_bytes(int ot, int nt) {
    return G_STAGES * G_BK * ((G_TM + 4) + (16 * nt + 4) + (ot < 4 ? 4 : ot)) * 4;
}

template <int NORM>
GradChoice grad_fn_for(int ot) {
    switch (ot) {
        case 1: return {grad_kernel<NORM, 1, 4>, grad_smem_bytes(1, 4)};
        case 2: return {grad_kernel<NORM, 2, 4>, grad_smem_bytes(2, 4)};
        case 4: return {grad_kernel<NORM, 4, 4>, grad_smem_bytes(4, 4)};
        case 8: return {grad_kernel<NORM, 8, 2>, grad_smem_bytes(8, 2)};
        default: return {grad_kernel<NORM, 16, 1>, grad_smem_bytes(16, 1)};
    }
}
int nt_for(int ot) { return ot <= 4 ? 4 : (ot == 8 ? 2 : 1); }

struct GradPlan {
    GradParams p;
    int ot, nt;
    bool tensor;               // channel contraction on the tensor cores (km_grad_tensor.cu)
    bool sign;                 // p = 1 with the signs as a matrix operand (km_grad_sign.cu)
    int splits_told;           // what callers are asked scratch for: the automatic split of the kernel without signs
    int splits;                // the automatic split of the kernel that runs, at most that
    long long partial_elems;   // elements of one dense partial result
};

// Preferred k split: the smallest within 0.5 % of the least estimated time.  An SM works through its share of
// the blocks, ceil(blocks / SMs), two at a time, or one by one 10 % slower per slab (the tensor-core kernel: one
// at a time); a slab of 32 k takes about the time below, a block 2.5 us besides, and the partial results of a
// split are written and read back at about 5 TB/s.  Measured on B200, us, against the rule before (whole waves,
// at least 8 slabs a block, at most 64 splits), for K, M, N, O, p:
//   1000, 200, 50, 4, 1.5:  101 (2 splits) -> 17 (32)     2000, 64, 64, 8, 1:     54 (5) -> 17 (63)
//   500, 64, 16, 4, 1:      68 (1) -> 13 (16)             30000, 64, 16, 16, 1.7: 74 (59) -> 46 (134)
//   500, 100, 30, 32, 1:    35 (1) -> 15 (16)             8000, 500, 20, 4, 1.7:  175 (31) -> 156 (36)
//   30000, 4096, 256, 4, 1: 6244 (8) -> 6237 (4)          64, 1000, 1000, 16, 1.5: 57 (1) either way
int preferred_split(const GradPlan& plan, int norm_type, bool square_root) {
    const GradParams& p    = plan.p;
    const long long blocks = (long long)p.tiles_m * p.tiles_n * p.o_chunks * p.L;
    const long long slabs  = ceil_div_ll(p.K, G_BK);
    const long long sms    = sm_count();
    const double bytes     = 4.0 * p.L * p.O * p.N * p.M;
    if (blocks <= 0 || slabs <= 1) return 1;
    double slab_us = 2.0;
    if (!plan.tensor) {
        slab_us = 0.6 + 0.16 * plan.nt * (1 + plan.ot);
        if (norm_type == KM_NORM_P) slab_us += (square_root ? 0.5 : 1.4) * plan.nt;
    }
    auto cost = [&](long long s, long long per_split) {
        const long long share = ceil_div_ll(blocks * s, sms);
        const double units    = plan.tensor ? (double)share : 0.9 * share + ((share & 1) ? 0.1 : 0.0);
        return units * per_split * slab_us + 2.5 * share + (s > 1 ? 3.0 + (2.0 * s + 1.0) * bytes / 5e6 : 0.0);
    };
    // more than 16 blocks per SM gain nothing, and partial results stay within 512 MB
    const double cap = 512e6 / (bytes > 0.0 ? bytes : 1.0);
    long long last   = std::min(slabs, 16 * sms / blocks);
    if ((double)last > cap) last = (long long)cap;
    return cheapest_split(slabs, last, cost);
}

// What the kernels of the p = 1 gradient take, us: a slab of 32 k and the rest of a block (its set-up, first slabs, last
// sums and stores); what rows of the result that cannot be stored 16 bytes at a time add to the latter, and rows of b or
// c that cannot be copied 16 bytes at a time to the former (warps of the sign kernel then copy 128 rows of b word by
// word).  The numbers of the FP32 and the weights kernel were fitted on B200 to 10558 calls (K 256 to 30000, M 9 to 4096, N 64
// to 1000, O 1 to 64), of which 95 % are within 8 to 20 % of estimated_us().  The sign kernel's were fitted so too and then
// lowered when it became faster, but by less than its times fell: for 4 / 8 / 16 / 32 channels a slab takes 0.66 / 0.73 / 0.55
// / 0.69 us and words 0.16 to 0.45.  Its times are therefore overestimated, and calls near the line keep the other kernel
// although the sign kernel is up to 1.2 times as fast there (the lines marked * at consider_sign()).  Of 6000 calls of
// the same ranges 475 had changed their kernel with the lowered numbers, and none of them became slower by it.
struct P1Cost {
    double slab, block, ragged, words;
};
P1Cost p1_cost(const GradPlan& plan) {
    if (plan.sign) {
        switch (plan.ot) {
            case 4: return {0.77, 5.3, 0.5, 0.25};
            case 8: return {0.74, 6.7, 1.6, 0.20};
            case 16: return {0.56, 5.1, 1.8, 0.56};
            default: return {0.84, 7.8, 3.6, 0.50};
        }
    }
    if (plan.tensor) return plan.ot == 16 ? P1Cost{1.50, 3.1, 0.3, 0.0} : plan.ot == 32 ? P1Cost{1.67, 5.9, 0.3, 0.0} : P1Cost{1.17, 5.9, 0.3, 0.0};
    const double slab = plan.ot == 1 ? 2.49 : plan.ot == 2 ? 3.05 : plan.ot == 4 ? 4.22 : plan.ot == 8 ? 3.64 : 3.51;
    return {slab, 1.0, 2.0, 0.0};
}

// Estimated time of a p = 1 plan whose k range is cut into `s` pieces of at most `per` slabs, us.  An SM has one block of
// a tensor-core kernel at a time, two of the FP32 kernel 10 % faster per slab than one; the sign kernel's last wave
// overlaps a little with the others.
double estimated_us(const GradPlan& plan, const KmGradArgs* a, long long sms, long long s, long long per) {
    const GradParams& p    = plan.p;
    const P1Cost cost      = p1_cost(plan);
    const long long blocks = (long long)p.tiles_m * p.tiles_n * p.o_chunks * p.L * s;
    const long long share  = ceil_div_ll(blocks, sms);
    double waves = (double)share, work = (double)share, slab = cost.slab;
    if (plan.sign) {
        waves = work   = 0.85 * share + 0.15 * std::max(1.0, (double)blocks / sms);
        const bool vec = aligned16(a->b) && aligned16(a->c) && a->ldb % 4 == 0 && a->ldc % 4 == 0 && a->b_stride_l % 4 == 0 &&
                         a->c_stride_l % 4 == 0;
        if (!vec) slab += cost.words * p.N / ((double)GS_TN * p.tiles_n);
    } else if (!plan.tensor) {
        work = 0.9 * share + ((share & 1) ? 0.1 : 0.0);
    }
    // (dense rows assumed: which memory the result goes to has no say in how it is computed)
    const bool stores_vec = p.M % 4 == 0;
    const double mbytes = 4e-6 * p.L * p.O * p.N * p.M;
    // the sign kernel writes rows 16 bytes at a time, which costs more where the result does not fit L2
    const double stores = plan.sign ? 0.2 * std::max(0.0, mbytes - 128.0) : 0.0;
    return 3.0 + stores + work * per * slab + waves * (cost.block + (stores_vec ? 0.0 : cost.ragged)) +
           (s > 1 ? 3.0 + 0.06 * s + 0.2 * (2 * s + 1) * mbytes : 0.0);
}

// Turns a plan for p = 1 into one for the kernel with the signs as a matrix operand (km_grad_sign.cu) where that is
// estimated to be the faster one.  A block of it costs the same for 1 to 128 rows n, takes a multiple of its channel tile
// and is alone on its SM, so short sums lose what many k win.  Measured on B200, us, sign kernel against the other one
// (FP32 up to 16 channels, weights from 17 on):
//   K      M     N     O    sign   other         K      M     N     O    sign   other
//   256    4096  1000  4    328    221           256    1000  1000  16   133    182
//   320    4096  1000  3    358    273           1024   1000  1000  4    181    251
//   256    4096  128   4    47     35            8192   1000  1000  16   1976   5456
// * 512    250   500   64   100    105           8192   1000  1000  4    1201   1723
// * 30000  4096  256   2    4311   4443          30000  4096  256   4    4314   6225
//   30000  4096  256   32   8993   22054         30000  4096  256   64   18030  29480
// b and c in rows that are not 16-byte aligned:
// * 8192   1000  1000  4    1497   1723          30000  4096  256   16   9760   19950
// * 30000  4096  256   4    5397   6226          30000  4096  256   32   15410  22840
// * 30000  4096  256   64   30760  36350       * 1001   1000  300   4    92     97
// Its split of k stays within the one that callers were told of (see kermac_b200_cdist_grad_scratch_bytes).
void consider_sign(const KmGradArgs* a, GradPlan* plan) {
    if (a->norm_type != KM_NORM_L1 || a->contraction == KM_CONTRACT_FP32 || plan->partial_elems == 0) return;
    const bool named = a->contraction == KM_CONTRACT_TENSOR;
    // below 256 k the automatic choice has always been the FP32 kernel
    if (a->k < (named ? 1 : 8 * G_BK) || a->n < (named ? 96 : 64)) return;
    GradPlan sign = *plan;
    GradParams& p = sign.p;
    sign.sign = sign.tensor = true;
    sign.ot                 = gs_ot_for(a->o);
    // (its tiles and channel chunks are smaller than those of the plan: calls that would need too many keep theirs)
    const long long tiles_m = ceil_div_ll(p.M, gs_mt_for(sign.ot)), tiles_n = ceil_div_ll(p.N, GS_TN);
    const long long chunks = ceil_div_ll(p.O, sign.ot), slabs = ceil_div_ll(p.K, G_BK), sms = sm_count();
    if (tiles_m * tiles_n > (1LL << 26) || chunks > 65535) return;
    p.tiles_m = (int)tiles_m; p.tiles_n = (int)tiles_n; p.o_chunks = (int)chunks;
    // for 16 blocks per SM and more a further split gains nothing
    const long long last = std::min<long long>(plan->splits_told, 16 * sms / (tiles_m * tiles_n * chunks * p.L));
    sign.splits = cheapest_split(slabs, last, [&](long long s, long long per) { return estimated_us(sign, a, sms, s, per); });
    // compared with the automatic splits, also where the caller asks for others: a call that has no room for partial sums
    // then takes the kernel of the same call with split_k = 1
    auto us = [&](const GradPlan& q) {
        const long long per = ceil_div_ll(slabs, q.splits);
        return estimated_us(q, a, sms, ceil_div_ll(slabs, per), per);
    };
    // Callers who name the tensor cores get this kernel from 96 rows on unless the other one is estimated to be a tenth
    // and 5 us faster, so that near ties do not follow the operands' alignment.  The automatic choice wants 3 % for the
    // estimate's error.
    const double with = us(sign), without = us(*plan);
    if (named ? with <= std::max(1.1 * without, without + 5.0) : 1.03 * with < without) *plan = sign;
}

// (splits_told does not depend on the sign kernel: without `any_kernel` the plan is done before that is looked at)
int make_grad_plan(const KmGradArgs* a, GradPlan* plan, bool any_kernel = true) {
    if (!a) return fail(KM_ERR_NULL_POINTER, "args is NULL");
    if (a->m < 0 || a->n < 0 || a->o < 0 || a->k < 0 || a->l < 1)
        return fail(KM_ERR_BAD_SHAPE, "bad extents m=%d n=%d o=%d k=%d l=%d", a->m, a->n, a->o, a->k, a->l);
    if (a->l > 65535) return fail(KM_ERR_TOO_LARGE, "at most 65535 batch entries per call");
    const bool empty = (a->m == 0 || a->n == 0 || a->o == 0);
    if (!empty && (!a->out || !a->d || (a->k > 0 && (!a->a || !a->b || !a->c))))
        return fail(KM_ERR_NULL_POINTER, "a, b, c, d and out must be device pointers");
    if (a->norm_type < KM_NORM_L1 || a->norm_type > KM_NORM_P)
        return fail(KM_ERR_BAD_ENUM, "norm_type %d is not a KmNormType", a->norm_type);
    if ((a->k > 1 && a->lda < a->m) || (a->n > 1 && a->ldb < a->k) || (a->o > 1 && a->ldc < a->k) ||
        (a->n > 1 && a->ldd < a->m) || (a->n > 1 && a->out_stride_n < a->m))
        return fail(KM_ERR_BAD_STRIDE, "a row pitch is smaller than the row it spans");
    if (a->a_stride_l < 0 || a->b_stride_l < 0 || a->c_stride_l < 0 || a->d_stride_l < 0 || a->out_stride_l < 0 ||
        a->out_stride_o < 0)
        return fail(KM_ERR_BAD_STRIDE, "strides must be non-negative");
    if (a->l > 1 && a->out_stride_l == 0) return fail(KM_ERR_BAD_STRIDE, "out cannot be broadcast over the batch");
    if (!hyper_ok(a->p)) return fail(KM_ERR_BAD_HYPERPARAM, "p needs a non-negative batch stride");
    if (a->split_k < 0) return fail(KM_ERR_BAD_SHAPE, "split_k must be >= 0");
    if (a->contraction < KM_CONTRACT_AUTO || a->contraction > KM_CONTRACT_TENSOR)
        return fail(KM_ERR_BAD_ENUM, "contraction must be KM_CONTRACT_AUTO, _FP32 or _TENSOR");

    GradParams& p = plan->p;
    p.M = a->m; p.N = a->n; p.O = a->o; p.K = a->k; p.L = a->l;
    p.A = a->a; p.lda = a->lda; p.a_sl = a->a_stride_l;
    p.B = a->b; p.ldb = a->ldb; p.b_sl = a->b_stride_l;
    p.C = a->c; p.ldc = a->ldc; p.c_sl = a->c_stride_l;
    p.D = a->d; p.ldd = a->ldd; p.d_sl = a->d_stride_l;
    p.p = a->p;
    int ot = 1;
    while (ot < a->o && ot < 16) ot *= 2;
    // The tensor-core kernel forms each weight once for up to 64 channels and leaves the channel
    // products to the MMA.  Up to 16 channels the FP32 kernel is level or faster (K = 30000, M = 4096,
    // N = 256: 20.4 against 19.1 ms at 16, 20.3 when the operands cannot be staged by TMA); from 17 on
    // it needs a second pass and the tensor cores win (40.4 against 22.0 ms at 32, 80.7 against 29.6 at
    // 64).  The tensor kernel needs at least one slab of k.  For p = 1 consider_sign() may put a third kernel in
    // place of the one chosen here.
    plan->tensor = a->k > 0 && (a->contraction == KM_CONTRACT_TENSOR ||
                                (a->contraction == KM_CONTRACT_AUTO && a->o >= KM_GRAD_TENSOR_MIN_O && a->k >= 8 * G_BK));
    plan->sign = false;
    if (plan->tensor) ot = gt_ot_for(a->o);
    plan->ot = ot;
    plan->nt = nt_for(ot);
    p.tiles_m  = (int)ceil_div_ll(p.M, plan->tensor ? GT_TM : G_TM);
    p.tiles_n  = (int)ceil_div_ll(p.N, plan->tensor ? gt_tn_for(ot) : 16 * plan->nt);
    p.o_chunks = (int)ceil_div_ll(p.O > 0 ? p.O : 1, ot);
    p.a_vec    = aligned16(p.A) && p.lda % 4 == 0 && p.a_sl % 4 == 0;
    if ((long long)p.tiles_m * p.tiles_n > (1LL << 26)) return fail(KM_ERR_TOO_LARGE, "too many output tiles");
    if (p.o_chunks > 65535) return fail(KM_ERR_TOO_LARGE, "too many output channels");

    plan->splits = plan->splits_told = preferred_split(*plan, a->norm_type, !a->p.ptr && a->p.value == 1.5f);
    plan->partial_elems = (long long)p.L * p.O * p.N * p.M;
    if (any_kernel) consider_sign(a, plan);
    return 0;
}

}  // namespace
}  // namespace km

extern "C" int64_t kermac_b200_cdist_grad_scratch_bytes(const KmGradArgs* args) {
    using namespace km;
    GradPlan plan;
    if (make_grad_plan(args, &plan, false)) return 0;
    int splits = args->split_k > 0 ? args->split_k : plan.splits_told;
    if (splits <= 1) return 0;
    return (int64_t)splits * plan.partial_elems * 4;
}

extern "C" int kermac_b200_describe_grad(const KmGradArgs* args, char* buf, int32_t buf_len) {
    using namespace km;
    if (!buf || buf_len <= 0) return fail(KM_ERR_NULL_POINTER, "buf is NULL or empty");
    GradPlan plan;
    if (int rc = make_grad_plan(args, &plan)) return rc;
    snprintf(buf, (size_t)buf_len, "cdist_grad kernel=%s channels=%d tiles=%dx%d chunks=%d batches=%d splits=%d",
             plan.sign ? "sign" : plan.tensor ? "weights" : "fp32", plan.ot, plan.p.tiles_m, plan.p.tiles_n, plan.p.o_chunks,
             plan.p.L, args->split_k > 0 ? args->split_k : plan.splits);
    return 0;
}

// Launches the plan with this split; scratch holds the partial results of more than one.
namespace km {
namespace {

int run_plan(const KmGradArgs* args, GradPlan& plan, int splits, void* scratch, cudaStream_t st) {
    GradParams& p   = plan.p;
    int slabs       = (int)ceil_div_ll(p.K > 0 ? p.K : 1, G_BK);
    p.k_per_split   = (int)ceil_div_ll(slabs, splits) * G_BK;
    splits          = (int)ceil_div_ll(p.K > 0 ? p.K : 1, p.k_per_split);
    p.splits        = splits;
    if (splits > 1) {
        p.E = static_cast<float*>(scratch);
        p.e_sn = p.M; p.e_so = (long long)p.N * p.M; p.e_sl = (long long)p.O * p.N * p.M;
        p.split_stride = plan.partial_elems;
        p.e_vec = aligned16(p.E) && p.M % 4 == 0;
    } else {
        p.E = args->out;
        p.e_sn = args->out_stride_n; p.e_so = args->out_stride_o; p.e_sl = args->out_stride_l;
        p.split_stride = 0;
        p.e_vec = aligned16(p.E) && p.e_sn % 4 == 0 && p.e_so % 4 == 0 && p.e_sl % 4 == 0;
    }
    // a host scalar p = 1.5 means |x|^(1/2): the square-root kernels; a device vector of p is only
    // known to the kernel, which then takes the general lg2 / ex2 route
    const bool sqrt_route = (args->norm_type == KM_NORM_P && !args->p.ptr && args->p.value == 1.5f);
    if (plan.tensor) {
        GradTensorParams t;
        t.M = p.M; t.N = p.N; t.O = p.O; t.K = p.K; t.L = p.L;
        t.A = p.A; t.lda = p.lda; t.a_sl = p.a_sl;
        t.B = p.B; t.ldb = p.ldb; t.b_sl = p.b_sl;
        t.C = p.C; t.ldc = p.ldc; t.c_sl = p.c_sl;
        t.D = p.D; t.ldd = p.ldd; t.d_sl = p.d_sl;
        t.E = p.E; t.e_sn = p.e_sn; t.e_so = p.e_so; t.e_sl = p.e_sl;
        t.p = p.p;
        t.ot = plan.ot;
        t.rg = gt_rg_for(plan.ot);
        t.tiles_m = p.tiles_m; t.tiles_n = p.tiles_n; t.o_chunks = p.o_chunks; t.splits = p.splits;
        t.k_per_split = p.k_per_split; t.split_stride = p.split_stride;
        t.c_vec = aligned16(p.C) && p.ldc % 4 == 0 && p.c_sl % 4 == 0;
        t.e_vec = p.e_vec;
        if (int rc = plan.sign ? grad_sign_launch(t, st) : grad_tensor_launch(t, sqrt_route ? GT_NORM_SQRT : args->norm_type, st))
            return rc;
    } else {
    GradChoice choice = {nullptr, 0};
    switch (args->norm_type) {
        case KM_NORM_L1: choice = grad_fn_for<KM_NORM_L1>(plan.ot); break;
        case KM_NORM_L2: choice = grad_fn_for<KM_NORM_L2>(plan.ot); break;
        default: choice = sqrt_route ? grad_fn_for<G_NORM_SQRT>(plan.ot) : grad_fn_for<KM_NORM_P>(plan.ot); break;
    }
    GradFn fn = choice.fn;
    if (int rc = cuda_status(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, choice.smem_bytes),
                             "cudaFuncSetAttribute(grad_kernel)"))
        return rc;
    dim3 grid((unsigned)((long long)p.tiles_m * p.tiles_n * splits), (unsigned)p.o_chunks, (unsigned)p.L);
    if (int rc = cuda_status(launch_overlapped(fn, grid, G_THREADS, choice.smem_bytes, st, p), "launch of grad_kernel")) return rc;
    }
    if (splits > 1) {
        const long long total = plan.partial_elems;
        int blocks = (int)(ceil_div_ll(total, 256) < 8LL * sm_count() ? ceil_div_ll(total, 256) : 8LL * sm_count());
        // (below 2^31 the grid stride cannot overflow 32 unsigned bits)
        auto reduce = total < (1LL << 31) ? grad_reduce_kernel<unsigned int> : grad_reduce_kernel<long long>;
        if (int rc = cuda_status(launch_overlapped(reduce, dim3((unsigned)blocks), 256, 0, st, p.E, args->out, p.M, p.N, p.O, p.L,
                                                   splits, plan.partial_elems, args->out_stride_n, args->out_stride_o,
                                                   args->out_stride_l),
                                 "launch of grad_reduce_kernel"))
            return rc;
    }
    return 0;
}

}  // namespace
}  // namespace km

extern "C" int kermac_b200_cdist_grad(const KmGradArgs* args, void* stream) {
    using namespace km;
    GradPlan plan;
    if (int rc = make_grad_plan(args, &plan)) return rc;
    if (plan.partial_elems == 0) return 0;
    if (int rc = require_sm100()) return rc;
    int splits = args->split_k > 0 ? args->split_k : plan.splits;
    if (splits > 1) {
        const int64_t need = (int64_t)splits * plan.partial_elems * 4;
        if (!args->scratch || args->scratch_bytes < need) {
            if (args->split_k > 1)
                return fail(KM_ERR_BAD_SHAPE, "split_k=%d needs %lld bytes of scratch, got %lld", splits, (long long)need,
                            (long long)(args->scratch ? args->scratch_bytes : 0));
            splits = 1;   // automatic mode falls back to a single pass
        }
    }
    return run_plan(args, plan, splits, args->scratch, static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------
// kermac_b200_cdist_grad_static: the split-k gradient for callers that have no way
// to hand over scratch memory.
//
// Some hosts of this library may not allocate device memory at the point where they
// call it: a plugin running inside another runtime's memory pool with a fixed budget,
// a real-time loop whose latency budget excludes allocator calls, or a binding whose
// foreign-function layer only passes through the pointers it was given.  For them the
// partial sums of the k split live in the array below, which is part of the library
// image: every GPU that loads the library carries it (KM_GRAD_STATIC_SCRATCH_BYTES)
// from load until the process exits.
//
// Rules that follow from sharing one array:
//   * it keeps whatever the previous call left in it.  Nothing in it has to start at
//     zero, because every partial tile a call reads back is first written in full by
//     that same call;
//   * two calls whose kernels overlap on the GPU (different streams, different host
//     threads) would write the same partials and corrupt each other: callers must
//     order them;
//   * the first call on each device looks up the array's device address.  That lookup
//     is a runtime API call, so make the first call per device outside any stream
//     capture.  The library calls no allocator, but the CUDA runtime places the array
//     when it loads this module on a device (at the latest during that first call), so
//     that warm-up call also belongs outside any region that must not see device memory
//     being reserved;
//   * the looked-up address is kept per device ordinal for the life of the process: it
//     does not survive cudaDeviceReset() or the teardown of the device's primary context.
namespace km {
namespace {

constexpr long long KM_GRAD_STATIC_FLOATS = KM_GRAD_STATIC_SCRATCH_BYTES / 4;
static __device__ __align__(256) float g_grad_static_scratch[KM_GRAD_STATIC_FLOATS];

// Device address of g_grad_static_scratch per device ordinal.  In host code the
// array's name only stands for the symbol; the address a kernel can use has to be
// asked for with the owning device current.
float*     g_grad_static_ptr[64] = {nullptr};
std::mutex g_grad_static_mutex;

int grad_static_scratch(float** out) {
    int dev = -1;
    if (int rc = cuda_status(cudaGetDevice(&dev), "cudaGetDevice")) return rc;
    if (dev < 0 || dev >= 64) return fail(KM_ERR_INTERNAL, "device ordinal %d is out of range", dev);
    std::lock_guard<std::mutex> lock(g_grad_static_mutex);
    if (!g_grad_static_ptr[dev]) {
        void* p = nullptr;
        if (int rc = cuda_status(cudaGetSymbolAddress(&p, g_grad_static_scratch),
                                 "cudaGetSymbolAddress(g_grad_static_scratch)"))
            return rc;
        if (!p) return fail(KM_ERR_INTERNAL, "the static scratch array has no device address");
        g_grad_static_ptr[dev] = static_cast<float*>(p);
    }
    *out = g_grad_static_ptr[dev];
    return 0;
}

}  // namespace
}  // namespace km

extern "C" int kermac_b200_cdist_grad_static(const KmGradArgs* args, void* stream) {
    using namespace km;
    if (!args) return fail(KM_ERR_NULL_POINTER, "args is NULL");
    GradPlan plan;
    if (int rc = make_grad_plan(args, &plan)) return rc;
    int splits = args->split_k;
    const int64_t cap      = KM_GRAD_STATIC_FLOATS * 4;
    const int64_t per_split = plan.partial_elems * 4;
    if (splits > 1) {
        // an explicit split either fits the built-in array or is refused
        const int64_t need = (int64_t)splits * per_split;
        if (need > cap)
            return fail(KM_ERR_TOO_LARGE,
                        "split_k = %d needs %lld bytes of scratch but the built-in array holds %lld; pass a smaller "
                        "split_k (1 always fits), or call kermac_b200_cdist_grad with your own scratch",
                        splits, (long long)need, (long long)cap);
    } else if (splits == 0) {
        // automatic: the preferred split, reduced to the largest one whose partial sums fit (down to a
        // single pass)
        const long long fit = per_split > 0 ? cap / per_split : plan.splits;
        splits              = (int)std::max(1LL, std::min<long long>(plan.splits, fit));
    }
    float* scratch = nullptr;
    if (splits > 1)
        if (int rc = grad_static_scratch(&scratch)) return rc;
    if (plan.partial_elems == 0) return 0;
    if (int rc = require_sm100()) return rc;
    return run_plan(args, plan, splits, scratch, static_cast<cudaStream_t>(stream));
}
