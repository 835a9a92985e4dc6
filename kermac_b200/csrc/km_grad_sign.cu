// Tensor-core form of the p = 1 gradient contraction
//   out[l, o, n, m] = sum_k c[l, o, k] * a[l, k, m] * sign(d[l, n, m] - b[l, n, k])
// (what the reference's kernel_cute_p_norm_kernel_gradient computes for NormType.L1,
// include/p_norm_gradient.cuh:22-405; sign() is copysign(1, x)).
//
// For a fixed m the sum is a matrix product over k of S_m[n, k] = sign(d[n, m] - b[n, k]) and the
// products P_m[o, k] = c[o, k] * a[k, m].  The signs are exact in bf16, so only P has to be split to
// keep fp32 accuracy: each fp32 product becomes three bf16 pieces by truncation (8 + 8 + 8 significant
// bits; the second and third scaled by powers of two, so that no bit of a normal product is lost), and one tcgen05.mma kind::f16 of 128 rows (n) x 3 OT columns (piece, channel)
// x 16 k takes all three.  The general tensor-core kernel (km_grad_tensor.cu) has the weights
// a * g(d - b) in the A operand, split per (n, m, k); here the A operand costs a subtract, a byte
// permute and one logic operation per two k, and the split is done once per (o, k, m), shared by the
// 128 rows n of the block.
//
// Work decomposition: a thread block owns 128 rows n, MT columns m and up to OT channels.
//   8 to 16 generating warps (2 to 4 groups of 4): a thread owns one row n (a tensor-memory lane); a group takes
//      every second to fourth slab of 32 k, or 16 k of every second one, reads them once for all m and writes the signs
//      (8 columns of packed bf16 pairs per m and 16 k) with tcgen05.st into a ring of A buffers, one slab each;
//   2 to 8 product warps in two groups that take the slabs in turn: P_m for the slab, split and parked in shared memory as
//      the B operand (K-major rows of 64 bytes, 64-byte swizzle; row = piece * OT + channel);
//   2 warps (4 with few channels) issue the MMAs, one accumulator of 3 OT columns (rounded up to 16) per m;
//   4 draining warps: the tensor core truncates when it accumulates, so a chain is cut every 512 k (32
//      MMAs), read back and added, rounding to nearest, to running sums in shared memory; the cuts of the
//      MT accumulators are staggered, so the MMAs of the others keep the pipe busy meanwhile;
//   1 warp copies slabs of a (transposed) and c into shared memory;
//   1 warp brings the 128 x 32 slabs of b into shared memory (128-byte swizzle, so the
//      16-byte reads of 32 different rows do not collide) by TMA when the rows of b are 16-byte
//      aligned, 4 warps by 4-byte cp.async otherwise, same bits either way.
// The product warps have no global loads of their own: their fence to the asynchronous units waits for
// every memory operation of the thread, and behind loads in flight it made each slab as long as a load.
// What bounds it (B200, K = 30000, M = 4096, N = 256; ms, in brackets the kernel that took these calls before):
// 4 channels 4.31 (6.2), 8: 4.72 (10.6), 16: 7.13 (20.3), 32: 9.0 with the
// same inputs again, 9.3 to 9.4 with new ones (22.0), 64: 18.0 to 18.4.
// The MMAs alone would take 2.5 ms at 32 channels (an MMA of 128 rows x N columns holds the tensor pipe N / 2 cycles,
// also with the stores to tensor memory beside it), the ALU pipe (permutes and logic, half rate) about 3.5.  Instructions are
// what the rest goes to: at 4 channels the generating warps hardly rest, at 32 the product warps, each warp issuing once in five to
// nine cycles beside the others, and the hand-overs are a third of what is issued.  On the way
// here (ms at 4 / 32 channels): one thread issuing all MMAs 18.5 / -; every role handing over per 16 k by its own
// barrier, four issuing warps 6.7 / 14.5; global loads taken from the product warps 7.0 / 14.2; eight product warps
// and carried copy addresses 7.5 / 12.4; all MMAs of a slab in one elected block 6.2 / 11.9; 16 k of all eight m
// per group and slab instead of four 5.5 / 11.9; pieces scaled 5.5 / 12.1; infinite and NaN products left to the sums
// (bf16_joined) instead of being looked for in each product 5.25 / 11.3; the constants of sign_pair in registers 4.6 / 10.9;
// whole slabs for a group of generating warps 4.6 / 9.6; two groups of product warps 4.3 / 9.2; sleeping waits - / 8.9.
// Hand-over is by mbarriers, one round per slab; every wait is bounded, and a wait that runs out sets a
// flag (kermac_b200_device_error_flag) and lets the block run to its end without its results.
#include <cstring>

#include "km_build_tma.cuh"
#include "km_common.cuh"
#include "km_host.h"
#include "km_mbar.cuh"
#include "km_tcgen05.cuh"

namespace km {
namespace {

constexpr int GS_BK       = 32;     // k per slab (two MMAs)
constexpr int GS_KA       = 16;     // k per MMA
constexpr int GS_DRAIN    = 4;
constexpr int GS_B_BYTES  = GS_TN * GS_BK * 4;   // one staged slab of b
constexpr int GS_B_STAGES = 4;
constexpr int GS_P_SLOTS  = 3;      // slabs of split products
constexpr int GS_AC_SLOTS = 4;      // slabs of a (transposed) and c
constexpr int GS_C_PITCH  = GS_BK + 4;
constexpr int GS_DONE     = 4;      // ring of slab-done barriers
constexpr int GS_CHAIN    = 16;     // slabs per accumulation chain

template <int OT, int MT, bool TMA>
struct GsShape {
    static constexpr int COLS      = (3 * OT + 15) / 16 * 16;          // MMA width: pieces x channels
    static constexpr int P_BYTES   = COLS * GS_BK * 2;                 // split products of one m and slab
    static constexpr int A_OFF     = MT * COLS;                        // tensor-memory columns before the A buffers
    static constexpr int A_COLS    = MT * GS_BK / 2;                   // one A buffer: a slab's signs for all m
    static constexpr int NB        = (512 - A_OFF) / A_COLS >= GS_DONE ? GS_DONE : (512 - A_OFF) / A_COLS;
    // Groups of four generating warps, and how many of the two halves of a slab's k a group takes.  Whole slabs mean half
    // as many hand-overs, each some 65 instructions a warp against 96 (4 m) or 192 (8 m) for the signs of a half; they pay
    // where there are as many A buffers as groups, or with fewer groups.  Measured at K = 30000, M = 4096, N = 256, ms:
    //   groups x halves   4 x 1    2 x 2    3 x 2    4 x 2      (one group of product warps)
    //   4 channels        4.61     4.92     5.06     4.73
    //   8                 5.37     4.84     4.88     4.89
    //   16                8.10     8.14     8.22     7.64
    //   32               10.87     9.80     9.68    10.04       (with two groups 2 x 2 9.20, 3 x 2 9.35)
    static constexpr int GROUPS    = OT == 8 || OT == 32 ? 2 : 4;
    static constexpr int HALVES    = OT == 4 ? 1 : 2;
    // Product warps in groups that take every PGROUPS-th slab: a wait for a phase that is long complete costs such a warp
    // 180 cycles and the fence behind its stores about as much, so it is better off with more products between them.
    //   warps x groups   one group  2 x 2   4 x 2   8 x 2   3 x 3   6 x 3   12 x 3
    //   4 channels       4.61 (4)   4.31    4.51            4.38    4.36
    //   8                4.86 (4)   5.86    4.73    4.98    5.88    4.75
    //   16               7.62 (8)           7.13    7.15            7.85
    //   32               9.63 (8)                   9.20                    9.15 (sums of 8192 k and less: 8 x 2)
    static constexpr int PROD      = OT == 4 ? 2 : OT == 32 ? 8 : 4;
    static constexpr int PGROUPS   = 2;
    static constexpr int PWARPS    = PROD / PGROUPS;
    // warps that issue MMAs (two MMAs per accumulator and slab): with few channels there are more accumulators
    // (half as many: 4 / 8 / 16 channels 6.1 / 5.0 / 9.3 ms)
    static constexpr int ISSUERS   = OT >= 16 ? 2 : 4;
    static constexpr int GEN       = 4 * GROUPS;
    // warps that bring slabs of b: one with TMA, four that copy a quarter of the rows each without
    static constexpr int BWARPS    = TMA ? 1 : 4;
    static constexpr int WARPS     = GEN + PROD + GS_DRAIN + ISSUERS + 1 + BWARPS;
    static constexpr int THREADS   = 32 * WARPS;
    static constexpr int AC_FLOATS = MT * GS_BK + OT * GS_C_PITCH;
    static constexpr int OFF_B     = 0;                                // shared memory, from a 1024-byte boundary
    static constexpr int OFF_P     = OFF_B + GS_B_STAGES * GS_B_BYTES;
    static constexpr int OFF_RUN   = OFF_P + GS_P_SLOTS * MT * P_BYTES;
    static constexpr int OFF_AC    = OFF_RUN + MT * OT * GS_TN * 4;
    static constexpr int SMEM_USED = 1024 + OFF_AC + GS_AC_SLOTS * AC_FLOATS * 4;
    // more than half of an SM's shared memory: a second block would wait inside tcgen05.alloc
    static constexpr int SMEM      = SMEM_USED > 117 * 1024 ? SMEM_USED : 117 * 1024;
    static constexpr int OCTS      = OT >= 8 ? OT / 8 : 1;             // product warps per m: eight channels each
    static constexpr int MSUB      = OT >= 8 ? 1 : 8 / OT;             // m that a product warp takes at a time
    static constexpr int STAGGER   = GS_CHAIN / MT;                    // slabs between the chain cuts of two m
    static_assert(MT % 4 == 0 && GS_CHAIN % MT == 0 && NB >= 2 && GS_P_SLOTS <= GS_DONE &&
                  SMEM <= 227 * 1024, "shape");
};

__device__ int g_grad_sign_wait_expired = 0;

// Two k of the A operand: +-1 in bf16 with the signs of two differences, (halves & SIGN_BITS) | ONES.  One LOP3 takes at
// most one constant of its own: written with both as constants it became two, 512 of 2218 ALU instructions a block and
// slab at 4 channels, so both are kept in registers (signs_in_registers; 4 / 8 / 16 / 32 channels 5.23 / 5.79 / 8.56 /
// 11.31 -> 4.61 / 5.37 / 8.10 / 10.87 ms).
struct SignConstants {
    uint32_t sign_bits, ones;
};
__device__ __forceinline__ SignConstants signs_in_registers() {
    SignConstants k;
    asm volatile("mov.b32 %0, 0x80008000;" : "=r"(k.sign_bits));
    asm volatile("mov.b32 %0, 0x3F803F80;" : "=r"(k.ones));
    return k;
}
__device__ __forceinline__ uint32_t sign_pair(u64 diff, SignConstants k) {
    uint32_t w;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(w) : "r"(upper_halves(diff)), "r"(k.sign_bits), "r"(k.ones));
    return w;
}

template <int OT, int MT, bool TMA>
__global__ void __launch_bounds__(GsShape<OT, MT, TMA>::THREADS, 1)
grad_sign_kernel(const __grid_constant__ GradTensorParams p, const __grid_constant__ CUtensorMap map_b) {
    using S = GsShape<OT, MT, TMA>;
    extern __shared__ unsigned char smem_raw[];
    constexpr int BARS = 2 * GS_B_STAGES + 2 * GS_AC_SLOTS + GS_P_SLOTS + S::NB + GS_DONE + 2 * MT + 1;
    __shared__ __align__(8) unsigned long long s_bars[BARS];
    __shared__ uint32_t s_tmem;
    __shared__ int s_expired;

    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base     = (raw_addr + 1023u) & ~1023u;
    unsigned char* tiles    = smem_raw + (base - raw_addr);

    const int tid  = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;

    // n-tiles fastest: the blocks that read the same (k range, m-column) tile of a run together
    int bx          = blockIdx.x;
    const int tn    = bx % p.tiles_n; bx /= p.tiles_n;
    const int split = bx % p.splits;  bx /= p.splits;
    const int tm    = bx;
    const int oc    = blockIdx.y;
    const int l     = blockIdx.z;
    const int m0 = tm * MT, n0 = tn * GS_TN, o0 = oc * OT;

    const int k_begin = split * p.k_per_split;
    const int k_end   = min(p.K, k_begin + p.k_per_split);
    const int nslabs  = (k_end > k_begin) ? (k_end - k_begin + GS_BK - 1) / GS_BK : 0;

    const uint32_t bars = smem_u32(s_bars);
    auto bar_at  = [&](int i) { return bars + 8u * i; };
    auto bfull   = [&](int st) { return bar_at(st); };
    auto bempty  = [&](int st) { return bar_at(GS_B_STAGES + st); };
    auto acfull  = [&](int sl) { return bar_at(2 * GS_B_STAGES + sl); };
    auto acempty = [&](int sl) { return bar_at(2 * GS_B_STAGES + GS_AC_SLOTS + sl); };
    constexpr int BAR_P = 2 * GS_B_STAGES + 2 * GS_AC_SLOTS;
    auto pfull   = [&](int sl) { return bar_at(BAR_P + sl); };
    auto afull   = [&](int b) { return bar_at(BAR_P + GS_P_SLOTS + b); };
    auto done    = [&](int i) { return bar_at(BAR_P + GS_P_SLOTS + S::NB + i); };   // MMAs of a slab
    auto dfull   = [&](int m) { return bar_at(BAR_P + GS_P_SLOTS + S::NB + GS_DONE + m); };
    auto dfree   = [&](int m) { return bar_at(BAR_P + GS_P_SLOTS + S::NB + GS_DONE + MT + m); };
    const uint32_t last_bar = bar_at(BARS - 1);

    if (tid == 0) {
        for (int st = 0; st < GS_B_STAGES; ++st) {
            mbar_init(bfull(st), TMA ? 1 : 32 * S::BWARPS);
            mbar_init(bempty(st), 8 / S::HALVES);      // a slab is read by one or two groups of four warps
        }
        for (int sl = 0; sl < GS_AC_SLOTS; ++sl) {
            mbar_init(acfull(sl), 32);
            mbar_init(acempty(sl), S::PWARPS);
        }
        for (int sl = 0; sl < GS_P_SLOTS; ++sl) mbar_init(pfull(sl), S::PWARPS);
        for (int b = 0; b < S::NB; ++b) mbar_init(afull(b), 8 / S::HALVES);
        for (int i = 0; i < GS_DONE; ++i) mbar_init(done(i), S::ISSUERS);
        for (int m = 0; m < MT; ++m) {
            mbar_init(dfull(m), 1);
            mbar_init(dfree(m), GS_DRAIN);
        }
        mbar_init(last_bar, S::ISSUERS);
        s_expired = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tc::fence_smem_to_async();
    }
    constexpr int MMA_WARP = S::GEN + S::PROD + GS_DRAIN;
    after_previous_grid();
    if (warp == MMA_WARP) tc::tmem_alloc(smem_u32(&s_tmem), 512);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = s_tmem;
    bool expired = false;
    // (One lane waiting for its warp instead of all 32 was three times slower in all.)
    auto wait = [&](uint32_t bar, int parity) {
        // once a wait has run out this warp stops waiting: a stuck barrier costs one limit, not one per slab
        // (sleeping: 32 channels 9.19 -> 8.91 ms, where the generating warps rest three quarters of the time; 4 channels
        // 4.31 -> 4.48, 16 on unaligned rows 2.23 -> 2.26)
        if (!expired && !(OT == 32 ? mbar_sleep_bounded(bar, parity) : mbar_wait_bounded(bar, parity))) {
            expired = true;
            *reinterpret_cast<volatile int*>(&s_expired) = 1;
        }
    };

    if (warp < S::GEN) {
        // ------------------------------------------------------------------ signs
        const int q = warp & 3, group = warp >> 2;
        const int row = 32 * q + lane;
        const int n   = n0 + row;
        const float* D = p.D + (long long)l * p.d_sl;
        // a group takes all 32 k of every GROUPS-th slab, or two groups make up a slab and take 16 k each
        const int hf0 = S::HALVES == 2 ? 0 : group & 1;
        u64 dd[MT];
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const float v = (n < p.N && m0 + i < p.M) ? D[(long long)n * p.ldd + m0 + i] : 0.0f;
            dd[i] = pack2(v, v);
        }
        const uint32_t t_row = tmem + (static_cast<uint32_t>(32 * q) << 16) + S::A_OFF;
        const SignConstants signs = signs_in_registers();
        const unsigned char* brow = tiles + S::OFF_B + row * (GS_BK * 4);
        for (int s = group * S::HALVES / 2; s < nslabs; s += S::GROUPS * S::HALVES / 2) {
            const int st = s % GS_B_STAGES;
            wait(bfull(st), (s / GS_B_STAGES) & 1);
            const int buf = s % S::NB, before = s - S::NB;
            if (before >= 0) wait(done(before % GS_DONE), (before / GS_DONE) & 1);
            __syncwarp();
            tc::fence_after_sync();
#pragma unroll
            for (int h = 0; h < S::HALVES; ++h) {
                const int hf = hf0 + h;
                u64 b2[GS_KA / 2];
#pragma unroll
                for (int i = 0; i < GS_KA / 4; ++i) {
                    const int chunk = (hf * (GS_KA / 4) + i) ^ (row & 7);
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(brow + st * GS_B_BYTES + chunk * 16);
                    b2[2 * i]     = v.x;
                    b2[2 * i + 1] = v.y;
                }
#pragma unroll
                for (int i = 0; i < MT; i += 2) {
                    uint32_t w[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) w[j] = sign_pair(sub2(dd[i + (j >> 3)], b2[j & 7]), signs);
                    tc::st_32x32b_x16(t_row + buf * S::A_COLS + (hf * MT + i) * (GS_KA / 2), w);
                }
            }
            tc::wait_st();
            tc::fence_before_sync();
            __syncwarp();
            // only now: the stores have consumed what was read from the stage (an arrival right after the reads
            // were issued let the next copy overtake them)
            if (lane == 0) {
                mbar_arrive(bempty(st));
                mbar_arrive(afull(buf));
            }
        }
    } else if (warp < S::GEN + S::PROD) {
        // ------------------------------------------------------------------ split products
        const int pw  = (warp - S::GEN) % S::PWARPS;
        const int o   = OT >= 8 ? (pw % S::OCTS) * 8 + (lane >> 2) : ((lane >> 2) & (OT - 1));
        const int kc  = lane & 3;                                   // eight k of the slab
        const int mi0 = (pw / S::OCTS) * S::MSUB + (OT >= 8 ? 0 : (lane >> 2) / OT);
        constexpr int MSTEP = (S::PWARPS / S::OCTS) * S::MSUB;
        static_assert(MT % MSTEP == 0, "every product warp takes the same number of m");
        for (int s = (warp - S::GEN) / S::PWARPS; s < nslabs; s += S::PGROUPS) {
            const int ac = s % GS_AC_SLOTS;
            wait(acfull(ac), (s / GS_AC_SLOTS) & 1);
            const int slot = s % GS_P_SLOTS, before = s - GS_P_SLOTS;
            if (before >= 0) wait(done(before % GS_DONE), (before / GS_DONE) & 1);
            __syncwarp();
            const float* as = reinterpret_cast<const float*>(tiles + S::OFF_AC) + ac * S::AC_FLOATS + kc * 8;
            const float* cs = as + MT * GS_BK + o * GS_C_PITCH;
            const ulonglong2 c0 = *reinterpret_cast<const ulonglong2*>(cs);
            const ulonglong2 c1 = *reinterpret_cast<const ulonglong2*>(cs + 4);
            const u64 c2[4] = {c0.x, c0.y, c1.x, c1.y};
#pragma unroll
            for (int it = 0; it < MT / MSTEP; ++it) {
                const int mi = mi0 + it * MSTEP;
                const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(as + mi * GS_BK);
                const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(as + mi * GS_BK + 4);
                const u64 a2[4] = {a0.x, a0.y, a1.x, a1.y};
                uint32_t p1[4], p2[4], p3[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const u64 v  = mul2(c2[e], a2[e]);
                    const u64 r  = bf16_remainder2(v, BF16_STEP_2);
                    const u64 r2 = bf16_remainder2(r, BF16_STEP_3);
                    p1[e]        = upper_halves(v);
                    p2[e]        = upper_halves(r);
                    p3[e]        = upper_halves(r2);
                }
                unsigned char* dst = tiles + S::OFF_P + (slot * MT + mi) * S::P_BYTES;
#pragma unroll
                for (int piece = 0; piece < 3; ++piece) {
                    const int r   = piece * OT + o;
                    const int off = r * 64 + ((kc ^ ((r >> 1) & 3)) << 4);
                    const uint32_t* w = piece == 0 ? p1 : piece == 1 ? p2 : p3;
                    *reinterpret_cast<uint4*>(dst + off) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            tc::fence_smem_to_async();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(pfull(slot));
                mbar_arrive(acempty(ac));
            }
        }
    } else if (warp < MMA_WARP) {
        // ------------------------------------------------------------------ chain sums and results
        const int q = warp & 3;
        const int row = 32 * q + lane;
        const int n   = n0 + row;
        const uint32_t t_row = tmem + (static_cast<uint32_t>(32 * q) << 16);
        float* run = reinterpret_cast<float*>(tiles + S::OFF_RUN) + row;
        auto drain = [&](int m, int chain) {
            wait(dfull(m), chain & 1);
            __syncwarp();
            tc::fence_after_sync();
            float v[OT];
            if constexpr (OT == 4) {
                uint32_t r[16];
                tc::ld_32x32b_x16(t_row + m * S::COLS, r);
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = bf16_joined(__uint_as_float(r[i]), __uint_as_float(r[4 + i]), __uint_as_float(r[8 + i]));
            } else if constexpr (OT == 8) {
                uint32_t r1[16], r3[8];
                tc::ld_32x32b_x16(t_row + m * S::COLS, r1);
                tc::ld_32x32b_x8(t_row + m * S::COLS + 16, r3);
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = bf16_joined(__uint_as_float(r1[i]), __uint_as_float(r1[8 + i]), __uint_as_float(r3[i]));
            } else {
#pragma unroll
                for (int o = 0; o < OT; o += 16) {
                    uint32_t r1[16], r2[16], r3[16];
                    const uint32_t t = t_row + m * S::COLS + o;
                    tc::ld3_32x32b_x16(t, t + OT, t + 2 * OT, r1, r2, r3);
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[o + i] = bf16_joined(__uint_as_float(r1[i]), __uint_as_float(r2[i]), __uint_as_float(r3[i]));
                }
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(dfree(m));
            float* dst = run + m * OT * GS_TN;
#pragma unroll
            for (int i = 0; i < OT; ++i) dst[i * GS_TN] = chain ? dst[i * GS_TN] + v[i] : v[i];
        };
        // cut e comes after slab STAGGER * e - 1 and belongs to accumulator -e mod MT
        for (int e = 1; S::STAGGER * e < nslabs; ++e) {
            const int m = (MT - e % MT) % MT;
            drain(m, (S::STAGGER * (e + m) - 1) / GS_CHAIN);
        }
        if (nslabs > 0)
            for (int m = 0; m < MT; ++m) drain(m, (nslabs - 1 + S::STAGGER * m) / GS_CHAIN);
        asm volatile("bar.sync 2, %0;" ::"n"(32 * GS_DRAIN) : "memory");
        if (!*reinterpret_cast<volatile int*>(&s_expired) && n < p.N) {
            float* E = p.E + (long long)split * p.split_stride + (long long)l * p.e_sl + (long long)n * p.e_sn + m0;
            for (int o = 0; o < OT && o0 + o < p.O; ++o) {
                float* dst = E + (long long)(o0 + o) * p.e_so;
#pragma unroll
                for (int m = 0; m < MT; m += 4) {
                    float v[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[i] = nslabs > 0 ? run[((m + i) * OT + o) * GS_TN] : 0.0f;
                    if (p.e_vec && m0 + m + 3 < p.M) {
                        *reinterpret_cast<float4*>(dst + m) = make_float4(v[0], v[1], v[2], v[3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (m0 + m + i < p.M) dst[m + i] = v[i];
                    }
                }
            }
        }
    } else if (warp < MMA_WARP + S::ISSUERS) {
        // ------------------------------------------------------------------ MMA issue (one lane per warp)
        // Everything here is warp-uniform and shared out over several warps: beside the generating warps an MMA and
        // what prepares it take such a warp some 150 cycles, though the tensor pipe needs 3 OT / 2.
        constexpr uint32_t idesc = tc::instr_desc_bf16(GS_TN, S::COLS);
        constexpr int PER  = MT / S::ISSUERS;
        const int first    = __shfl_sync(0xFFFFFFFFu, warp - MMA_WARP, 0) * PER;
        const uint32_t tm0 = __shfl_sync(0xFFFFFFFFu, tmem, 0);
        int slot = 0, slot_parity = 0, buf = 0, buf_parity = 0;
        for (int s = 0; s < nslabs; ++s) {
            wait(pfull(slot), slot_parity);
            wait(afull(buf), buf_parity);
            int heads = 0, tails = 0;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int phase = s + S::STAGGER * (first + i);
                if (phase % GS_CHAIN == GS_CHAIN - 1 || s == nslabs - 1) tails |= 1 << i;
                if (phase % GS_CHAIN == 0 || s == 0) {
                    heads |= 1 << i;
                    if (s > 0) wait(dfree(first + i), (phase / GS_CHAIN - 1) & 1);   // the finished chain has been read
                }
            }
            __syncwarp();
            tc::fence_after_sync();
            const uint64_t b0 = tc::smem_desc_k_major_sw64(base + S::OFF_P + (slot * MT + first) * S::P_BYTES);
            const uint32_t a  = tm0 + S::A_OFF + buf * S::A_COLS + first * (GS_KA / 2);
            const uint32_t d  = tm0 + first * S::COLS;
            if (tc::elect_one()) {
#pragma unroll
                for (int i = 0; i < PER; ++i)
                    tc::mma_bf16_a_tmem(d + i * S::COLS, a + i * (GS_KA / 2), b0 + i * (S::P_BYTES >> 4), idesc, !(heads >> i & 1));
#pragma unroll
                for (int i = 0; i < PER; ++i)
                    tc::mma_bf16_a_tmem(d + i * S::COLS, a + (MT + i) * (GS_KA / 2), b0 + i * (S::P_BYTES >> 4) + 2, idesc, true);
                if (tails) {
#pragma unroll
                    for (int i = 0; i < PER; ++i)
                        if (tails >> i & 1) tc::commit(dfull(first + i));
                }
                tc::commit(done(s % GS_DONE));
            }
            __syncwarp();
            if (++slot == GS_P_SLOTS) { slot = 0; slot_parity ^= 1; }
            if (++buf == S::NB) { buf = 0; buf_parity ^= 1; }
        }
        // nothing of this block is in flight when its memory is given back
        if (tc::elect_one()) tc::commit(last_bar);
        __syncwarp();
        if (!mbar_wait_bounded(last_bar, 0)) expired = true;
    } else if (warp == MMA_WARP + S::ISSUERS) {
        // ------------------------------------------------------------------ slabs of a (transposed) and c
        // This warp's instructions per slab set its pace, so its addresses are carried from slab to slab.
        const int channels = min(OT, p.O - o0);
        const int mi = lane % MT, ka = lane / MT;        // a: one m, every (32 / MT)th k
        const int oc0 = lane >> 3, kc = (lane & 7) * 4;  // c: every fourth channel, four k (16 bytes at a time)
        const int a_bytes = m0 + mi < p.M ? 4 : 0;
        const float* a_src = a_bytes ? p.A + (long long)l * p.a_sl + (long long)(k_begin + ka) * p.lda + m0 + mi : p.A;
        const float* c_src = p.C + (long long)l * p.c_sl + (long long)o0 * p.ldc + k_begin;
        const long long a_step = a_bytes ? (long long)(32 / MT) * p.lda : 0;
        const uint32_t a_dst   = base + S::OFF_AC + (mi * GS_BK + ka) * 4;
        const uint32_t c_dst   = base + S::OFF_AC + MT * GS_BK * 4;
        for (int s = 0; s < nslabs; ++s) {
            const int ac = s % GS_AC_SLOTS;
            if (s >= GS_AC_SLOTS) wait(acempty(ac), (s / GS_AC_SLOTS - 1) & 1);
            __syncwarp();
            const uint32_t slot = ac * S::AC_FLOATS * 4;
            const int k0   = k_begin + s * GS_BK;
            const int krem = k_end - k0;
            if (krem >= GS_BK) {
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    cp_async_4(a_dst + slot + i * (32 / MT) * 4, a_src, a_bytes);
                    a_src += a_step;
                }
            } else {
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    const bool ok = ka + i * (32 / MT) < krem;
                    cp_async_4(a_dst + slot + i * (32 / MT) * 4, ok ? a_src : p.A, ok ? a_bytes : 0);
                    a_src += a_step;
                }
            }
            if (p.c_vec) {
                const float* src = c_src + (long long)oc0 * p.ldc + kc;
                const int valid  = max(0, min(4, krem - kc)) * 4;
#pragma unroll
                for (int i = 0; i < (OT + 3) / 4; ++i) {
                    const bool ok = 4 * i + oc0 < channels && valid > 0;
                    if (4 * i + oc0 < OT) cp_async_16(c_dst + slot + ((4 * i + oc0) * GS_C_PITCH + kc) * 4, ok ? src : p.C, ok ? valid : 0);
                    src += 4 * p.ldc;
                }
            } else {
                const float* src = c_src + lane;
                const bool k_ok  = lane < krem;
#pragma unroll 8
                for (int o = 0; o < OT; ++o) {
                    const bool ok = o < channels && k_ok;
                    cp_async_4(c_dst + slot + (o * GS_C_PITCH + lane) * 4, ok ? src : p.C, ok ? 4 : 0);
                    src += p.ldc;
                }
            }
            c_src += GS_BK;
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(acfull(ac)) : "memory");
        }
        cp_async_wait<0>();
    } else {
        // ------------------------------------------------------------------ slabs of b
        if constexpr (TMA) {
            if (lane == 0) {
                const int lb = (p.b_sl == 0) ? 0 : l;   // a broadcast operand has one batch slice
                int s = 0;
                for (; s < nslabs; ++s) {
                    const int st = s % GS_B_STAGES;
                    if (s >= GS_B_STAGES) wait(bempty(st), (s / GS_B_STAGES - 1) & 1);
                    if (expired) break;
                    mbar_expect_tx(bfull(st), GS_B_BYTES);
                    tma_load_3d(base + S::OFF_B + st * GS_B_BYTES, &map_b, k_begin + s * GS_BK, n0, lb, bfull(st));
                }
                // copies still in flight land before the block's shared memory is given back
                for (int i = s > GS_B_STAGES ? s - GS_B_STAGES : 0; i < s; ++i)
                    for (int j = 0; j < (1 << 16); ++j)
                        if (mbar_try_wait(bfull(i % GS_B_STAGES), (i / GS_B_STAGES) & 1)) break;
            }
            __syncwarp();
        } else {
            constexpr int ROWS = GS_TN / S::BWARPS;
            const int first    = (warp - (MMA_WARP + S::ISSUERS + 1)) * ROWS;
            const int rows     = max(0, min(ROWS, p.N - n0 - first));
            const float* b_src = p.B + (long long)l * p.b_sl + (long long)(n0 + first) * p.ldb + k_begin + lane;
            for (int s = 0; s < nslabs; ++s) {
                const int st = s % GS_B_STAGES;
                if (s >= GS_B_STAGES) wait(bempty(st), (s / GS_B_STAGES - 1) & 1);
                __syncwarp();
                const bool k_ok    = k_begin + s * GS_BK + lane < k_end;
                const uint32_t dst = base + S::OFF_B + st * GS_B_BYTES + first * 128 + (lane & 3) * 4;
                const float* src   = k_ok ? b_src : p.B;
                const int bytes    = k_ok ? 4 : 0;
                const long long step = k_ok ? p.ldb : 0;
                // rows past n keep what is there: their results are not stored
#pragma unroll 8
                for (int i = 0; i < rows; ++i) {
                    cp_async_4(dst + i * 128 + (((lane >> 2) ^ (i & 7)) << 4), src, bytes);
                    src += step;
                }
                b_src += GS_BK;
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bfull(st)) : "memory");
            }
            cp_async_wait<0>();
        }
    }

    if (expired) atomicExch(&g_grad_sign_wait_expired, 1);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == MMA_WARP) tc::tmem_dealloc(tmem, 512);
}

template <int OT, int MT, bool TMA>
int grad_sign_launch_as(const GradTensorParams& p, cudaStream_t st) {
    using S = GsShape<OT, MT, TMA>;
    CUtensorMap map_b;
    memset(&map_b, 0, sizeof(map_b));
    if (TMA) {
        if (int rc = encode_tma_box(&map_b, p.B, p.K, p.N, p.L, p.ldb, p.b_sl, GS_BK, GS_TN, true)) return rc;
    }
    auto fn = grad_sign_kernel<OT, MT, TMA>;
    if (int rc = cuda_status(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM),
                             "cudaFuncSetAttribute(grad_sign_kernel)"))
        return rc;
    dim3 grid((unsigned)((long long)p.tiles_m * p.tiles_n * p.splits), (unsigned)p.o_chunks, (unsigned)p.L);
    return cuda_status(launch_overlapped(fn, grid, S::THREADS, S::SMEM, st, p, map_b), "launch of grad_sign_kernel");
}

template <int OT>
int grad_sign_launch_ot(const GradTensorParams& p, cudaStream_t st) {
    constexpr int MT = gs_mt_for(OT);
    // tiled TMA copies need a 16-byte aligned base and a pitch that is a multiple of 16 bytes
    if (tma_operand_ok(p.B, 1, p.ldb, p.b_sl, p.N, p.L)) return grad_sign_launch_as<OT, MT, true>(p, st);
    return grad_sign_launch_as<OT, MT, false>(p, st);
}

}  // namespace

int grad_sign_launch(const GradTensorParams& p, cudaStream_t st) {
    switch (p.ot) {
        case 4: return grad_sign_launch_ot<4>(p, st);
        case 8: return grad_sign_launch_ot<8>(p, st);
        case 16: return grad_sign_launch_ot<16>(p, st);
        case 32: return grad_sign_launch_ot<32>(p, st);
    }
    return fail(KM_ERR_INTERNAL, "no sign gradient kernel for %d channels per block", p.ot);
}

int grad_sign_take_wait_flag() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_grad_sign_wait_expired, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_grad_sign_wait_expired, &zero, sizeof(int));
    return v ? 1 : 0;
}

}  // namespace km
