// Kernel-matrix build in 64 x 64 output tiles.
//
// What bounds a small or middle-sized problem is not the arithmetic but how evenly the tiles fall on
// the 148 SMs and the latency in front of and behind each block's k loop.  A block here is 128 threads
// with 8 (n) x 4 (m) values each, four to six of them resident per SM, so a tile is a quarter of the
// 128 x 128 kernels' work and blocks hide one another's staging and stores.  The price is 3 shared
// loads and 8 duplicate moves for 16 packed pairs instead of 4 and 8 for 32, which the square and |.|
// steps pay once the k loop is long; the fractional power is bound by its own dependency chain and is
// faster here for few tiles and level for many.  small_preferred() in km_build_launch.cu has the measured line.
//
// Operands are staged k-major ([k][64]) whatever their layout, in slabs of 16 k rows:
//   TMA = true    both operands contiguous along the tile dimension and 16-byte aligned: tiled TMA
//                 copies into a ring, each stage refilled by the arrival that completes its empty phase
//   TMA = false   per operand, chosen by its strides (SmallStage):
//                   tile dimension contiguous, 16-byte aligned:  16-byte cp.async
//                   k contiguous, 16-byte aligned (torch rows):  16-byte loads of four k of a row, held
//                     in registers while the slab before is consumed and then stored transposed.  A warp
//                     covers two quads of k by 16 rows: whole 32-byte sectors on the global side, and on
//                     the shared side banks 16 q + t (4 rows of 68 floats are 16 mod 32), all different
//                   anything else:  4-byte cp.async
// The sum over k runs in the same order over the same terms as in the 128 x 128 kernels, so |.|, square
// and product results are the same bits.
#include <cuda.h>

#include <cstring>

#include "km_build_params.cuh"
#include "km_build_small.h"
#include "km_build_tma.cuh"
#include "km_host.h"
#include "km_mbar.cuh"

namespace km {
namespace {

constexpr int SB_TILE    = 64;
constexpr int SB_THREADS = 128;
constexpr int SB_WARPS   = SB_THREADS / 32;
constexpr int SB_BK      = 16;
constexpr int SB_RING    = 3;               // TMA stages
constexpr int SB_PITCH   = SB_TILE + 4;     // floats per staged k row without TMA

// Resident blocks per SM the inner steps are compiled for.  Measured with 4 / 5 / 6 / 7 blocks (128 / 102 /
// 85 / 73 registers): |.| 4000 x 4000 x 512 569 / 572 / 623 / 626 us and |.|^1.3 2048 x 2048 x 64 107 / 109 /
// 115 / 116 us want the registers; the square is level (16384 x 16384 x 512 8247 / 8246 / 8178 / 8227 us).
// The power by MUFU and table takes more registers still, for a slab loop unrolled by 4 (blocks x unroll x sixteenths of the
// pairs on MUFU, us, p = 1.3):         4 x 4 x 7   4 x 1 x 8   4 x 2 x 8   3 x 2 x 8   3 x 4 x 8   5 x 4 x 7   4 x 8 x 7
//   500 x 600 x 300, two of them         115.3       113.9                   112.6       109.4
//   3000 x 1000 x 800 rows               828         823                     813         806
//   8000^2 x 96 rows                     1730        1723        1735        1732        1709        1867        2059
//   6000^2 x 200, with itself            1048        1064        1039        1041        1061        1134        1223
constexpr int small_min_blocks(int inner) {
    return inner == IN_DIFF_POW_TABLE ? 3 : (inner == IN_DIFF_ABS || inner == IN_DIFF_POW) ? 4 : 6;
}

__device__ int g_small_wait_expired = 0;

enum SmallStage { SB_TILE_VEC = 0, SB_K_VEC, SB_SCALAR };

struct SmallParams {
    BuildParams b;
    int stage_a, stage_b;      // SmallStage
};

// One operand's slab of SB_BK k rows, without TMA.  `start` issues it (cp.async, or loads into
// registers), `finish` stores what was held in registers.
struct SlabLoader {
    const float* base;         // first element of the tile
    long long s_t, s_k;
    int rem_t, K, mode, tid;
    float4 held[2];

    __device__ __forceinline__ void start(float* dst, int kt) {
        const int k0 = kt * SB_BK;
        if (mode == SB_K_VEC) {
            const int t = (tid >> 5) * 16 + ((tid & 31) >> 1);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int k      = k0 + 4 * ((tid & 1) + 2 * i);
                const float* src = base + static_cast<long long>(t) * s_t + k;
                held[i]          = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (t < rem_t) {
                    if (k + 4 <= K) {
                        held[i] = *reinterpret_cast<const float4*>(src);
                    } else {
                        if (k < K) held[i].x = src[0];
                        if (k + 1 < K) held[i].y = src[1];
                        if (k + 2 < K) held[i].z = src[2];
                    }
                }
            }
        } else if (mode == SB_TILE_VEC) {
#pragma unroll
            for (int i = 0; i < (SB_BK * SB_TILE / 4) / SB_THREADS; ++i) {
                const int idx = tid + i * SB_THREADS;
                const int kk  = idx >> 4;
                const int t   = (idx & 15) << 2;
                int valid     = min(4, rem_t - t);
                valid         = (k0 + kk < K && valid > 0) ? valid : 0;
                const float* src = valid ? base + static_cast<long long>(k0 + kk) * s_k + t : base;
                cp_async_16(smem_u32(dst + kk * SB_PITCH + t), src, valid * 4);
            }
        } else {
            const bool k_contig = (s_k == 1);
#pragma unroll 4
            for (int i = 0; i < (SB_BK * SB_TILE) / SB_THREADS; ++i) {
                const int idx = tid + i * SB_THREADS;
                int kk, t;
                if (k_contig) {         // 8 k of 4 rows per warp: 32-byte runs, banks 4 kk + t
                    kk = (idx & 7) + ((idx >> 5) & 1) * 8;
                    t  = ((idx >> 3) & 3) + (idx >> 6) * 4;
                } else {
                    t  = idx & (SB_TILE - 1);
                    kk = idx >> 6;
                }
                const bool ok    = (k0 + kk < K) && (t < rem_t);
                const float* src = ok ? base + static_cast<long long>(t) * s_t + static_cast<long long>(k0 + kk) * s_k : base;
                cp_async_4(smem_u32(dst + kk * SB_PITCH + t), src, ok ? 4 : 0);
            }
        }
    }
    __device__ __forceinline__ void finish(float* dst) const {
        if (mode != SB_K_VEC) return;
        const int t = (tid >> 5) * 16 + ((tid & 31) >> 1);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float* d = dst + 4 * ((tid & 1) + 2 * i) * SB_PITCH + t;
            d[0 * SB_PITCH] = held[i].x;
            d[1 * SB_PITCH] = held[i].y;
            d[2 * SB_PITCH] = held[i].z;
            d[3 * SB_PITCH] = held[i].w;
        }
    }
};

template <int OP, int KT>
__device__ __forceinline__ void small_chain(const Epilogue& e, u64 (&acc)[8][2]) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float v0, v1;
            unpack2(acc[j][i], v0, v1);
            acc[j][i] = pack2(epilogue_value<OP, KT>(e, v0), epilogue_value<OP, KT>(e, v1));
        }
}

// The outer chain on the thread's values and their stores; `mirror`: also transposed.
// acc[j][i] holds row n = n_base + (j / 4) * 16 + j % 4, columns m = m_base + 2 i + {0, 1}.
template <bool SYM>
__device__ __forceinline__ void small_finish(const BuildParams& p, int l, u64 (&acc)[8][2], int m_base, int n_base,
                                             bool mirror) {
    // The chains that have names get straight-line code, chosen once: a small call is over before the
    // instructions of a per-value switch have been fetched.
    const Epilogue e = make_epilogue(p.outer_power, p.kernel_type, p.p_outer, p.bandwidth, p.epsilon, l);
    const int op = p.outer_power, kt = p.kernel_type;
    if (kt == KM_KERNEL_NONE) {
        if (op == KM_POW_ABS) small_chain<KM_POW_ABS, KM_KERNEL_NONE>(e, acc);
        else if (op == KM_POW_SQUARE) small_chain<KM_POW_SQUARE, KM_KERNEL_NONE>(e, acc);
        else if (op == KM_POW_SQRT) small_chain<KM_POW_SQRT, KM_KERNEL_NONE>(e, acc);
        else if (op == KM_POW_POW) small_chain<KM_POW_POW, KM_KERNEL_NONE>(e, acc);
    } else if (op == KM_POW_SQRT && kt == KM_KERNEL_LAPLACE) {
        small_chain<KM_POW_SQRT, KM_KERNEL_LAPLACE>(e, acc);
    } else if (op == KM_POW_NOOP && kt == KM_KERNEL_LAPLACE) {
        small_chain<KM_POW_NOOP, KM_KERNEL_LAPLACE>(e, acc);
    } else if (op == KM_POW_NOOP && kt == KM_KERNEL_GAUSSIAN) {
        small_chain<KM_POW_NOOP, KM_KERNEL_GAUSSIAN>(e, acc);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float v0, v1;
                unpack2(acc[j][i], v0, v1);
                acc[j][i] = pack2(e(v0), e(v1));
            }
    }
    if (kt != KM_KERNEL_NONE) {
        const float reg       = read_hyper(p.regularization, l);
        const long long delta = (long long)p.reg_off_n - (long long)p.reg_off_m;     // diagonal: m == n + delta
        if (reg != 0.0f && m_base + 4 > n_base + delta && m_base < n_base + 20 + delta) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int n = n_base + (j >> 2) * 16 + (j & 3);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float v0, v1;
                    unpack2(acc[j][i], v0, v1);
                    if (m_base + 2 * i == n + delta) v0 = 1.0f + reg;
                    if (m_base + 2 * i + 1 == n + delta) v1 = 1.0f + reg;
                    acc[j][i] = pack2(v0, v1);
                }
            }
        }
    }
    float* C      = p.C + static_cast<long long>(l) * p.c_sl;
    const bool mc = p.c_multicast != 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int n = n_base + (j >> 2) * 16 + (j & 3);
        if (n >= p.N) continue;
        float* dst = C + static_cast<long long>(n) * p.c_ld + m_base;
        float v[4];
        unpack2(acc[j][0], v[0], v[1]);
        unpack2(acc[j][1], v[2], v[3]);
        if (p.c_vec4 && m_base + 3 < p.M) {
            store_result4(dst, v[0], v[1], v[2], v[3], mc);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (m_base + q < p.M) store_result1(dst + q, v[q], mc);
        }
    }
    if constexpr (!SYM) return;
    if (!mirror) return;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int m = m_base + q;
        if (m >= p.M) continue;
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const int n = n_base + g * 16;
            float* dst  = C + static_cast<long long>(m) * p.c_ld + n;
            float v[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                float lo, hi;
                unpack2(acc[g * 4 + r][q >> 1], lo, hi);
                v[r] = (q & 1) ? hi : lo;
            }
            if (p.c_vec4 && n + 3 < p.N) {
                store_result4(dst, v[0], v[1], v[2], v[3], mc);
            } else {
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (n + r < p.N) store_result1(dst + r, v[r], mc);
            }
        }
    }
}

template <int INNER, bool TMA, bool SYM>
__global__ void __launch_bounds__(SB_THREADS, small_min_blocks(INNER))
build_small_kernel(const __grid_constant__ SmallParams sp, const __grid_constant__ CUtensorMap map_a,
                   const __grid_constant__ CUtensorMap map_b) {
    constexpr int PITCH        = TMA ? SB_TILE : SB_PITCH;
    constexpr int STAGES       = TMA ? SB_RING : 2;
    constexpr int STAGE_FLOATS = 2 * SB_BK * PITCH;
    __shared__ __align__(128) float smem[STAGES * STAGE_FLOATS];
    __shared__ __align__(8) unsigned long long bars[2 * SB_RING];
    const BuildParams& p = sp.b;

    const int tid  = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int l    = blockIdx.y;

    int tm, tn;
    if constexpr (SYM) {
        // only the tiles on and above the diagonal are launched, column by column: tn (tn + 1) / 2 + tm
        const int t = blockIdx.x;
        tn = static_cast<int>((sqrtf(8.0f * static_cast<float>(t) + 1.0f) - 1.0f) * 0.5f);
        while ((tn + 1) * (tn + 2) / 2 <= t) ++tn;
        while (tn * (tn + 1) / 2 > t) --tn;
        tm = t - tn * (tn + 1) / 2;
    } else {
        // four blocks per 128 x 128 tile of the launcher's order, so that ranges of that order and its
        // reuse of operand tiles in L2 carry over
        tile_coords(p.tile_first + (blockIdx.x >> 2), p.tiles_m, p.tiles_n, p.panel, tm, tn);
        tm = tm * 2 + (blockIdx.x & 1);
        tn = tn * 2 + ((blockIdx.x >> 1) & 1);
    }
    const int m0 = tm * SB_TILE, n0 = tn * SB_TILE;
    if (m0 >= p.M || n0 >= p.N) {
        after_previous_grid();
        return;
    }
    const int K  = p.K;
    const int ktiles = (K + SB_BK - 1) / SB_BK;

    const int tm_off = (warp & 1) * 32 + (lane & 7) * 4;
    const int tn_off = (warp >> 1) * 32 + (lane >> 3) * 4;   // + {0, 16}

    u64 acc[8][2];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j][0] = acc[j][1] = 0ull;

    float p_inner = 0.0f;
    if constexpr (TMA) {
        const uint32_t smem_base = smem_u32(smem);
        const uint32_t bar_base  = smem_u32(bars);
        auto full_bar  = [&](int s) { return bar_base + 8u * s; };
        auto empty_bar = [&](int s) { return bar_base + 8u * (SB_RING + s); };
        const int la = (p.a_sl == 0) ? 0 : l;   // broadcast operands have a single batch slice in their map
        const int lb = (p.b_sl == 0) ? 0 : l;
        auto issue = [&](int slab) {
            const int s        = slab % SB_RING;
            const uint32_t dst = smem_base + s * STAGE_FLOATS * 4;
            mbar_expect_tx(full_bar(s), STAGE_FLOATS * 4);
            tma_load_3d(dst, &map_a, m0, slab * SB_BK, la, full_bar(s));
            tma_load_3d(dst + SB_BK * SB_TILE * 4, &map_b, n0, slab * SB_BK, lb, full_bar(s));
        };
        if (tid == 0) {
#pragma unroll
            for (int s = 0; s < SB_RING; ++s) {
                mbar_init(full_bar(s), 1);
                mbar_init(empty_bar(s), SB_WARPS);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncthreads();
        after_previous_grid();
        if (tid == 0) {
            for (int s = 0; s < SB_RING && s < ktiles; ++s) issue(s);
        }

        bool alive  = true;
        int fail_kt = -1;   // first slab whose wait ran out on this thread
        for (int kt = 0; kt < ktiles; ++kt) {
            const int s = kt % SB_RING;
            if (alive && !mbar_wait_bounded(full_bar(s), (kt / SB_RING) & 1)) alive = false;
            const float* sa = smem + s * STAGE_FLOATS + tm_off;
            const float* sb = smem + s * STAGE_FLOATS + SB_BK * PITCH + tn_off;
            consume_slab<INNER, SB_BK, PITCH>(acc, sa, sb, K - kt * SB_BK, p_inner, 1.0f);
            __syncwarp();
            if (lane == 0 && mbar_arrive_pending(empty_bar(s)) == 1 && kt + SB_RING < ktiles && alive) {
                mbar_try_wait(empty_bar(s), (kt / SB_RING) & 1);   // the acquire side of the hand-over
                issue(kt + SB_RING);
            }
            if (!alive && fail_kt < 0) fail_kt = kt;
        }
        if (!alive) {
            atomicExch(&g_small_wait_expired, 1);
            if (tid == 0) {
                // copies already handed to the TMA engine get a bounded chance to land before this
                // block's shared memory is released
                const int last = fail_kt + SB_RING < ktiles ? fail_kt + SB_RING : ktiles;
                for (int slab = fail_kt; slab < last; ++slab)
                    for (int i = 0; i < (1 << 16); ++i)
                        if (mbar_try_wait(full_bar(slab % SB_RING), (slab / SB_RING) & 1)) break;
            }
            return;
        }
    } else {
        SlabLoader la = {p.A + static_cast<long long>(l) * p.a_sl + static_cast<long long>(m0) * p.a_sm,
                         p.a_sm, p.a_sk, p.M - m0, K, sp.stage_a, tid, {}};
        SlabLoader lb = {p.B + static_cast<long long>(l) * p.b_sl + static_cast<long long>(n0) * p.b_sn,
                         p.b_sn, p.b_sk, p.N - n0, K, sp.stage_b, tid, {}};
        PowTable table;
        if constexpr (INNER == IN_DIFF_POW_TABLE) {
            // (the first barrier of the k loop publishes it)
            __shared__ float s_pow[POW_ENTRIES];
            p_inner = p.p_inner.value;
            fill_pow_table(s_pow, p.pow, p_inner, tid, SB_THREADS);
            table.base = smem_u32(s_pow);
#pragma unroll
            for (int i = 0; i <= POW_DEGREE; ++i) table.c[i] = pack2(p.pow.c[i], p.pow.c[i]);
        }
        after_previous_grid();
        if (INNER == IN_DIFF_POW) p_inner = read_hyper(p.p_inner, l);
        la.start(smem, 0);
        lb.start(smem + SB_BK * PITCH, 0);
        cp_async_commit();
        la.finish(smem);
        lb.finish(smem + SB_BK * PITCH);
        for (int kt = 0; kt < ktiles; ++kt) {
            float* cur  = smem + (kt & 1) * STAGE_FLOATS;
            float* next = smem + ((kt + 1) & 1) * STAGE_FLOATS;
            cp_async_wait<0>();
            __syncthreads();           // slab kt is in place, and nobody reads `next` any more
            const bool more = kt + 1 < ktiles;
            if (more) {
                la.start(next, kt + 1);
                lb.start(next + SB_BK * PITCH, kt + 1);
            }
            cp_async_commit();
            consume_slab<INNER, SB_BK, PITCH>(acc, cur + tm_off, cur + SB_BK * PITCH + tn_off, K - kt * SB_BK, p_inner, 1.0f, table);
            if (more) {
                la.finish(next);
                lb.finish(next + SB_BK * PITCH);
            }
        }
        cp_async_wait<0>();
    }
    small_finish<SYM>(p, l, acc, m0 + tm_off, n0 + tn_off, SYM && tm != tn);
}

// ------------------------------------------------------------------ host side
typedef void (*SmallKernelFn)(const SmallParams, const CUtensorMap, const CUtensorMap);

template <int INNER>
SmallKernelFn pick(bool tma, bool symmetric) {
    if constexpr (INNER == IN_DIFF_SQUARE || INNER == IN_DOT_NOOP) {
        if (tma) return symmetric ? build_small_kernel<INNER, true, true> : build_small_kernel<INNER, true, false>;
    }
    return symmetric ? build_small_kernel<INNER, false, true> : build_small_kernel<INNER, false, false>;
}

SmallKernelFn small_kernel(int inner, bool tma, bool symmetric) {
    switch (inner) {
        case IN_DIFF_ABS: return pick<IN_DIFF_ABS>(tma, symmetric);
        case IN_DIFF_SQUARE: return pick<IN_DIFF_SQUARE>(tma, symmetric);
        case IN_DIFF_POW: return pick<IN_DIFF_POW>(tma, symmetric);
        case IN_DIFF_POW_TABLE: return pick<IN_DIFF_POW_TABLE>(tma, symmetric);
        case IN_DOT_NOOP: return pick<IN_DOT_NOOP>(tma, symmetric);
    }
    return nullptr;
}

int stage_mode(const float* base, long long s_t, long long s_k, long long s_l, int K, int L) {
    const bool aligned = aligned16(base) && (L <= 1 || s_l % 4 == 0);
    if (s_t == 1 && aligned && (s_k % 4 == 0 || K <= 1)) return SB_TILE_VEC;
    if (s_k == 1 && aligned && s_t % 4 == 0) return SB_K_VEC;
    return SB_SCALAR;
}

}  // namespace

int small_take_wait_flag() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_small_wait_expired, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_small_wait_expired, &zero, sizeof(int));
    return v ? 1 : 0;
}

bool small_wide_loads(const float* base, long long s_t, long long s_k, long long s_l, int K, int L) {
    return stage_mode(base, s_t, s_k, s_l, K, L) != SB_SCALAR;
}

bool small_supported(const BuildParams& p) {
    // (the tile counts keep block indices within 31 bits)
    return p.K >= 1 && p.L <= 65535 && p.tile_count <= 0x1fffffff && (!p.symmetric || p.tiles_n <= 23000) &&
           small_kernel(p.inner_id, false, false) != nullptr;
}

int launch_build_small(const BuildParams& p, bool tma, cudaStream_t stream) {
    SmallKernelFn fn = small_kernel(kernel_inner(p), tma, p.symmetric != 0);
    if (!fn) return fail(KM_ERR_INTERNAL, "no 64 x 64 kernel for inner id %d", p.inner_id);
    SmallParams sp;
    sp.b       = p;
    sp.stage_a = stage_mode(p.A, p.a_sm, p.a_sk, p.a_sl, p.K, p.L);
    sp.stage_b = stage_mode(p.B, p.b_sn, p.b_sk, p.b_sl, p.K, p.L);
    CUtensorMap map_a, map_b;
    std::memset(&map_a, 0, sizeof(map_a));
    std::memset(&map_b, 0, sizeof(map_b));
    if (tma) {
        if (int rc = encode_tma_box(&map_a, p.A, p.M, p.K, p.L, p.a_sk, p.a_sl, SB_TILE, SB_BK)) return rc;
        if (int rc = encode_tma_box(&map_b, p.B, p.N, p.K, p.L, p.b_sk, p.b_sl, SB_TILE, SB_BK)) return rc;
    }
    const long long edge = ceil_div_ll(p.N, SB_TILE);
    const long long tiles = p.symmetric ? edge * (edge + 1) / 2 : 4LL * p.tile_count;
    return cuda_status(launch_overlapped(fn, dim3((unsigned)tiles, (unsigned)p.L, 1), SB_THREADS, 0, stream, sp, map_a, map_b),
                       "launch of build_small_kernel");
}

}  // namespace km
