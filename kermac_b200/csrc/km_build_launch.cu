// kermac_b200_build_kernel: validation, operand exchange for n-contiguous outputs,
// variant choice and launch.  Host-side counterpart of the second half of the
// reference's run_kernel (src/kermac/build_a_kernel.py:237-392).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "km_build_cpasync_table.cuh"
#include "km_build_small.h"
#include "km_build_tma.cuh"
#include "km_host.h"
#include "km_pack.h"

namespace km {

namespace {

BuildKernelFn cpasync_kernel(int inner, bool avec, bool bvec, bool symmetric) {
    return inner < IN_DOT_NOOP ? cpasync_kernel_diff(inner, avec, bvec, symmetric)
                               : cpasync_kernel_dot(inner, avec, bvec, symmetric);
}

// One of the two layouts TensorStats accepts (src/kermac/common.py:96-102):
// the stride along `rows` or along `cols` is 1 and the other spans the unit one.
bool layout_ok(long long rows, long long cols, long long s_row, long long s_col) {
    if (rows <= 0 || cols <= 0) return true;
    if (s_col == 1 && s_row >= cols) return true;
    if (s_row == 1 && s_col >= rows) return true;
    return false;
}

// What takes the values of a function of f at the N Chebyshev nodes of [-0.5, 0.5] to the coefficients of the polynomial
// through them.
struct Interpolation {
    static constexpr int N = POW_DEGREE + 1;
    double node[N], coef[N][N];
    Interpolation() {
        std::memset(coef, 0, sizeof(coef));
        for (int j = 0; j < N; ++j) node[j] = 0.5 * std::cos(M_PI * (j + 0.5) / N);
        double t_prev[N] = {1.0}, t_now[N] = {0.0, 1.0};                         // T_0 and T_1 by powers of 2 f
        for (int k = 0; k < N; ++k) {
            const double* t = k ? t_now : t_prev;
            for (int i = 0; i < N; ++i)
                for (int j = 0; j < N; ++j)
                    coef[i][j] += std::ldexp(t[i], i) * (k ? 2.0 : 1.0) / N * std::cos(M_PI * k * (j + 0.5) / N);
            if (k == 0) continue;
            for (int i = N - 1; i >= 0; --i) {                                   // T_{k+1} = 2 x T_k - T_{k-1}
                const double next = (i ? 2.0 * t_now[i - 1] : 0.0) - t_prev[i];
                t_prev[i] = t_now[i];
                t_now[i]  = next;
            }
        }
    }
};

// The table route's coefficients for |x|^exponent: m^exponent on [1, 2) through the Chebyshev nodes.  Exponents outside
// the range, or whose polynomial has no sign where the topmost exponent bits need one, keep the MUFU route.
PowCoefs pow_coefs(float exponent) {
    static const Interpolation through;
    PowCoefs pc;
    std::memset(&pc, 0, sizeof(pc));
    if (!(exponent >= POW_MIN && exponent <= POW_MAX)) return pc;
    double value[Interpolation::N];
    for (int j = 0; j < Interpolation::N; ++j) value[j] = std::pow(1.5 + through.node[j], (double)exponent);
    for (int i = 0; i < Interpolation::N; ++i) {
        double sum = 0.0;
        for (int j = 0; j < Interpolation::N; ++j) sum += through.coef[i][j] * value[j];
        pc.c[i] = (float)sum;
    }
    float at_zero = pc.c[POW_DEGREE];                                            // f = -1.5, as the kernel computes it
    for (int i = POW_DEGREE - 1; i >= 0; --i) at_zero = std::fmaf(at_zero, -1.5f, pc.c[i]);
    pc.use  = at_zero != 0.0f && pc.c[POW_DEGREE] != 0.0f;
    pc.t254 = std::copysign(INFINITY, at_zero);
    pc.t255 = std::copysign(1.0f, pc.c[POW_DEGREE]);
    return pc;
}

struct BuildPlan {
    BuildParams p;
    bool avec, bvec;       // can be copied 16 bytes at a time along the points
    bool awide, bwide;     // ... or along k
    bool swapped;
    int  variant;
    bool small;      // 64 x 64 tiles
    bool automatic;  // the caller left the variant to this file
};

// When the 64 x 64 kernel is the faster one (K >= 1, an inner step it has).  Measured on B200, 128 x 128
// kernels against the 64 x 64 one, us:
//   torch rows, 16-byte aligned: always, because the 64 x 64 kernel loads those 16 bytes at a time too
//       square  2 x 1000^2 x 64: 22.9 / 18.8   8000^2 x 96: 580 / 431   16384^2 x 256: 5330 / 4695
//       |.|     2 x 1000^2 x 64: 28.9 / 17.6   8000^2 x 96: 637 / 429   16384^2 x 256: 5947 / 4671
//       |.|^1.3 2 x 1000^2 x 64: 57.1 / 49.5   8000^2 x 96: 1875 / 1708 16384^2 x 256: 20322 / 18460
// Otherwise the gain is in how evenly tiles fall on the 148 SMs: an SM's share is ceil(4 T / 148) quarter tiles, or
// ceil(T / 148) whole ones.  The 64 x 64 kernel is the faster one where quarters make the largest share smaller by
// more than its longer k step costs, and where the k loop is short in any case (T: 128 x 128 tiles).
//   an operand that both can only copy word by word (the longer step costs most here: the square above 512 tiles
//   and |.| with a long k loop are left to the 128 x 128 kernel):
//       square  share 2/4  8000 x 55 (T 63) x 371: 82 / 64   x 701: 144 / 114
//               share 3/4  1279^2 (T 100) x 127: 39.1 / 33.0   x 259: 63.7 / 63.8   x 371: 84 / 88
//                          2301^2 (T 324) x 127: 86.1 / 84.2   x 259: 159 / 164
//               share 7/8  2801^2 (T 484) x 33: 47.3 / 45.3   x 65: 71.9 / 74.0   x 701: 522 / 643
//               share 1    1401 x 1301 (T 121) x 33: 20.7 / 17.2   x 65: 27.5 / 26.8   x 97: 33.0 / 35.0   x 701: 146 / 203
//       |.|     share 3/4  1279^2 x 259: 72 / 57   x 701: 162 / 140   2301^2 x 701: 428 / 383
//               share 7/8  2801^2 x 259: 231 / 226   x 371: 314 / 317   x 701: 564 / 583
//               share 1    1401 x 1301 x 127: 45.2 / 38.1   x 259: 72.0 / 71.9   x 701: 162 / 179
//               4001 x 4003 (T 1024) x 65: 156 / 128   x 127: 225 / 217   x 259: 405 / 427   8001 x 8003 x 65: 540 / 490
//       with itself (quarters below the diagonal are left out as well, T counts what is launched)
//               square  2001^2 (T 136) x 701: 298 / 201   3601^2 (T 435) x 97: 96 / 88   x 259: 190 / 209
//               |.|     2801^2 (T 253) x 701: 326 / 307   3601^2 x 372: 283 / 278   x 701: 494 / 508
//   both operands contiguous along the points:
//       square  share 7/8  2000^2 (T 256) x 200: 67.8 / 59.7   x 700: 209 / 191   2800^2 (T 484) x 1024: 589 / 530
//               share 1    1536^2 (T 144) x 256: 46.4 / 45.4   x 512: 84.3 / 86.1   x 1024: 158 / 166
//                          2688^2 (T 441) x 256: 121 / 119   x 512: 230 / 233   x 1024: 451 / 459
//               4000^2 (T 1024) x 256: 273 / 268   x 512: 520 / 527   16384^2 x 128: 2145 / 2124   x 256: 4109 / 4153
//       |.|     share 7/8  2000^2 x 200: 74.0 / 67.3   x 700: 232 / 216   2800^2 x 1024: 647 / 601
//               share 1    1536^2 x 256: 51.6 / 50.2   x 512: 92.5 / 94.8   2112^2 (T 289) x 372: 129 / 133   x 1024: 332 / 352
//               with itself 1536^2 x 700: 131 / 103   4000^2 (T 528) x 372: 266 / 229
//               4000^2 x 256: 303 / 293   x 512: 580 / 576   16384^2 x 96: 1858 / 1825   x 128: 2374 / 2397
//   |.|^1.3, operands not held as aligned rows: a short k loop, or up to 2048 tiles (table of powers; in brackets the step
//   by lg2 and ex2 alone, which a p in device memory takes):
//       contiguous points 2048^2 x 512: 702 / 603 (919 / 804)   4000^2 x 1024: 4778 / 4490 (6279 / 6026)
//               4736 x 4096 x 600: 3207 / 3135 (4220 / 4197)   4400^2 x 600: 3596 / 3221 (4725 / 4319)
//               5760^2 x 600: 5579 / 5359 (7338 / 7178)   16384^2 x 64: 4866 / 4880 (6370 / 6302)
//               x 128: 9573 / 9445 (12559 / 12416)   x 256: 18899 / 18480 (24800 / 24638)
//       word by word 1000^2 x 27: 28.6 / 15.0 (34.6 / 18.6)   4001 x 4000 x 600: 3056 / 2932 (3911 / 3810)
//               5501 x 5500 x 600: 5627 / 5400 (7214 / 7028)   8001 x 8003 x 300: 5873 / 5849 (7524 / 7594)
//       with itself 4400^2 x 600: 2171 / 1720 (2760 / 2255)   5700^2 x 600: 3022 / 2816 (3860 / 3693)
//               8000^2 x 200: 2033 / 1839 (2586 / 2392)
//   (The line was drawn for the step without the table, when the two kernels were level beyond it; above 2048 tiles and 128
//   features the 128 x 128 kernel is now 2 to 5 % the slower one, 10 % with itself.)
// The line is drawn by the whole problem, not by the launch's tile range, so that ranges add up to the full
// launch's bits.  For |.|^p, whose two forms of the exponential the two kernels spread differently over a tile, it
// must not depend either on whether operands have been packed (the caller's scratch) or on symmetry (which a range
// switches off): it counts every tile, and is the same for contiguous points as for operands copied word by word
// (packed rows are rows that the 64 x 64 kernel reads as well, so they are never packed).
bool small_preferred(const BuildParams& p, bool avec, bool bvec, bool awide, bool bwide) {
    const bool rows = awide && bwide && !(avec && bvec);
    if (p.inner_id == IN_DIFF_POW) return rows || p.K <= 128 || (long long)p.tiles_m * p.tiles_n * p.L <= 2048;
    if (rows) return true;
    const long long tiles =
        (p.symmetric ? (long long)p.tiles_n * (p.tiles_n + 1) / 2 : (long long)p.tiles_m * p.tiles_n) * p.L;
    const bool absolute = p.inner_id == IN_DIFF_ABS;
    const long long sms = sm_count(), quarters = ceil_div_ll(4 * tiles, sms), whole = 4 * ceil_div_ll(tiles, sms);
    if (!awide || !bwide) {
        if (absolute && p.K <= 128) return true;
        if (p.symmetric) return tiles <= sms || (tiles <= 512 && p.K <= (absolute ? 512 : 192));
        if (tiles > 512) return false;
        if (absolute) return 4 * quarters <= 3 * whole || p.K <= 256;
        return 2 * quarters <= whole || p.K <= (4 * quarters <= 3 * whole ? 192 : 48);
    }
    if (p.K <= (absolute ? 96 : 128)) return true;
    // (many waves even out by themselves)
    if (p.K > 256 && quarters == whole && tiles <= 5 * sms && !p.symmetric) return false;
    return tiles <= 512 || (tiles <= 1024 && p.K <= 512);
}

// Where |.|^p with few features is faster through the table of powers, although every block fills the table first and the 64 x 64
// kernel then has three blocks on an SM instead of four.  Measured on B200, p = 1.3, time with the table over time
// without (contiguous points, rows and words alike), features:
//                      1      2      3      4      5      6      7      8      10     12     16     17     18     20     24
//   64^2               1.06   1.12   1.12   1.10   1.06   1.03   1.01   0.99   0.94   0.91   1.01
//   1000^2             1.21   1.13   1.02   0.98   0.94   0.91   0.89   0.87   0.86   0.84   0.87
//   4 x 1000^2         1.47   1.26   1.18   1.10   1.05   1.00   0.97   0.94   0.90   0.86   0.91
//   20000^2            1.47   1.33   1.18   1.08   1.01   0.98   0.95   0.93   0.87   0.84   0.90
// and of a matrix with itself, where blocks store their tile twice and lean more on one another; slabs are 16 features, and one
// that is whole runs other code than the one that is not, so that 17 features fetch both:
//   1000^2             1.15   1.11   1.08   1.06   1.04   1.02   1.01   1.00   0.97   0.95   0.98   0.98   0.97   0.95   0.93
//   4 x 1000^2         1.56   1.54   1.50   1.39   1.27   1.19   1.16   1.13   1.08   0.98   0.97   0.98   0.97   0.95   0.90
//   20000^2            1.40   1.37   1.31   1.23   1.15   1.09   1.05   1.04   0.99   0.95   1.03   1.09   1.07   1.01   0.91
// (Without a line at all 12000^2 x 1 took 291 us instead of 200.)  By what the operands are and not by p.symmetric, which tile
// ranges and KM_SYMMETRY_OFF switch off: the bits stay the same.
bool pow_table_preferred(const BuildParams& p) {
    const bool same = p.A == p.B && p.M == p.N && p.a_sm == p.b_sn && p.a_sk == p.b_sk && p.a_sl == p.b_sl;
    return same ? p.K > 20 || (p.K >= 11 && p.K <= 15) : p.K >= 6;
}

int make_plan(const KmBuildArgs* a, BuildPlan* plan) {
    if (!a) return fail(KM_ERR_NULL_POINTER, "args is NULL");
    if (a->m < 0 || a->n < 0 || a->k < 0 || a->l < 1)
        return fail(KM_ERR_BAD_SHAPE, "bad extents m=%d n=%d k=%d l=%d", a->m, a->n, a->k, a->l);
    const bool empty = (a->m == 0 || a->n == 0);
    if (!empty && (!a->out || ((!a->a || !a->b) && a->k > 0)))
        return fail(KM_ERR_NULL_POINTER, "a, b and out must be device pointers");
    if (a->inner_operator < 0 || a->inner_operator > KM_INNER_DOT)
        return fail(KM_ERR_BAD_ENUM, "inner_operator %d is not a KmInnerOperator", a->inner_operator);
    if (a->inner_power < 0 || a->inner_power > KM_POW_POW)
        return fail(KM_ERR_BAD_ENUM, "inner_power %d is not a KmPowerType", a->inner_power);
    if (a->outer_power < 0 || a->outer_power > KM_POW_POW)
        return fail(KM_ERR_BAD_ENUM, "outer_power %d is not a KmPowerType", a->outer_power);
    if (a->kernel_type < 0 || a->kernel_type > KM_KERNEL_GAUSSIAN)
        return fail(KM_ERR_BAD_ENUM, "kernel_type %d is not a KmKernelType", a->kernel_type);
    if (a->variant < KM_VARIANT_AUTO || a->variant > KM_VARIANT_TMA)
        return fail(KM_ERR_BAD_ENUM, "variant %d is not a KM_VARIANT_*", a->variant);
    if (!layout_ok(a->m, a->k, a->a_stride_m, a->a_stride_k))
        return fail(KM_ERR_BAD_STRIDE, "a has a non-standard memory layout: strides (%lld, %lld) for shape (%d, %d)",
                    (long long)a->a_stride_m, (long long)a->a_stride_k, a->m, a->k);
    if (!layout_ok(a->n, a->k, a->b_stride_n, a->b_stride_k))
        return fail(KM_ERR_BAD_STRIDE, "b has a non-standard memory layout: strides (%lld, %lld) for shape (%d, %d)",
                    (long long)a->b_stride_n, (long long)a->b_stride_k, a->n, a->k);
    if (!layout_ok(a->m, a->n, a->out_stride_m, a->out_stride_n))
        return fail(KM_ERR_BAD_STRIDE, "out has a non-standard memory layout: strides (%lld, %lld) for shape (%d, %d)",
                    (long long)a->out_stride_m, (long long)a->out_stride_n, a->m, a->n);
    if (a->a_stride_l < 0 || a->b_stride_l < 0 || a->out_stride_l < 0)
        return fail(KM_ERR_BAD_STRIDE, "batch strides must be non-negative");
    if (a->l > 1 && a->out_stride_l == 0)
        return fail(KM_ERR_BAD_STRIDE, "out cannot be broadcast over the batch");
    if (!hyper_ok(a->p_inner) || !hyper_ok(a->p_outer) || !hyper_ok(a->bandwidth) || !hyper_ok(a->regularization))
        return fail(KM_ERR_BAD_HYPERPARAM, "hyper-parameter vectors need a non-negative batch stride");

    BuildParams& p = plan->p;
    std::memset(&p, 0, sizeof(p));
    // An out whose n stride is 1 is written by the same kernel after exchanging the
    // roles of a and b (the kernel always writes its first tile dimension contiguously).
    const bool out_m_contig = (a->out_stride_m == 1 && (a->out_stride_n >= a->m || a->n <= 1));
    plan->swapped           = !out_m_contig;
    p.K = a->k;
    p.L = a->l;
    if (!plan->swapped) {
        p.M = a->m; p.N = a->n;
        p.A = a->a; p.a_sm = a->a_stride_m; p.a_sk = a->a_stride_k; p.a_sl = a->a_stride_l;
        p.B = a->b; p.b_sn = a->b_stride_n; p.b_sk = a->b_stride_k; p.b_sl = a->b_stride_l;
        p.c_ld = a->out_stride_n;
        p.reg_off_m = a->reg_off_x; p.reg_off_n = a->reg_off_y;
        p.sgn = 1.0f;
    } else {
        p.M = a->n; p.N = a->m;
        p.A = a->b; p.a_sm = a->b_stride_n; p.a_sk = a->b_stride_k; p.a_sl = a->b_stride_l;
        p.B = a->a; p.b_sn = a->a_stride_m; p.b_sk = a->a_stride_k; p.b_sl = a->a_stride_l;
        p.c_ld = a->out_stride_m;
        p.reg_off_m = a->reg_off_y; p.reg_off_n = a->reg_off_x;
        p.sgn = -1.0f;
    }
    p.C    = a->out;
    p.c_sl = a->out_stride_l;
    p.inner_id = inner_id(a->inner_operator, a->inner_power);
    if (p.inner_id < 0) return fail(KM_ERR_BAD_ENUM, "unsupported inner operator / power pair");
    p.outer_power    = a->outer_power;
    p.kernel_type    = a->kernel_type;
    p.p_inner        = a->p_inner;
    if (p.inner_id == IN_DIFF_POW && !p.p_inner.ptr && pow_table_preferred(p)) p.pow = pow_coefs(p.p_inner.value);
    p.p_outer        = a->p_outer;
    p.bandwidth      = a->bandwidth;
    p.regularization = a->regularization;
    p.epsilon        = a->epsilon;
    p.tiles_m        = (int)ceil_div_ll(p.M, BUILD_TILE);
    p.tiles_n        = (int)ceil_div_ll(p.N, BUILD_TILE);
    p.panel          = 16;
    if ((long long)p.tiles_m * p.tiles_n > 0x7fffffffLL) return fail(KM_ERR_TOO_LARGE, "too many output tiles");
    p.c_vec4 = aligned16(p.C) && (p.c_ld % 4 == 0) && (p.c_sl % 4 == 0);
    if (a->out_multicast != 0 && a->out_multicast != 1)
        return fail(KM_ERR_BAD_ENUM, "out_multicast must be 0 or 1");
    p.c_multicast = a->out_multicast;
    const int total_tiles = p.tiles_m * p.tiles_n;
    if (a->tile_first < 0 || a->tile_count < 0 || a->tile_first > total_tiles ||
        (long long)a->tile_first + a->tile_count > total_tiles)
        return fail(KM_ERR_BAD_SHAPE, "tile range [%d, %d + %d) is outside the %d tiles of this problem", a->tile_first,
                    a->tile_first, a->tile_count, total_tiles);
    p.tile_first = a->tile_first;
    p.tile_count = a->tile_count > 0 ? a->tile_count : total_tiles - a->tile_first;
    const bool all_tiles = (p.tile_first == 0 && p.tile_count == total_tiles);

    // a and b the same matrix, a chain that does not change when m and n trade places (the
    // diagonal rule included): compute the tiles on and above the diagonal and mirror them.
    // The mirrored values are the same bits the skipped tiles would have produced: the sum
    // over k runs in the same order over the same terms.
    if (a->symmetry < KM_SYMMETRY_AUTO || a->symmetry > KM_SYMMETRY_OFF)
        return fail(KM_ERR_BAD_ENUM, "symmetry must be KM_SYMMETRY_AUTO or KM_SYMMETRY_OFF");
    const bool even_chain = (p.inner_id == IN_DIFF_ABS || p.inner_id == IN_DIFF_SQUARE || p.inner_id == IN_DIFF_POW ||
                             p.inner_id >= IN_DOT_NOOP);
    p.symmetric = (a->symmetry == KM_SYMMETRY_AUTO) && even_chain && p.M == p.N && p.tiles_m > 1 && p.A == p.B &&
                  p.a_sm == p.b_sn && p.a_sk == p.b_sk && p.a_sl == p.b_sl && p.reg_off_m == p.reg_off_n &&
                  !p.c_multicast && all_tiles;

    plan->avec = (p.a_sm == 1) && aligned16(p.A) && (p.a_sk % 4 == 0 || p.K <= 1) && (p.a_sl % 4 == 0);
    plan->bvec = (p.b_sn == 1) && aligned16(p.B) && (p.b_sk % 4 == 0 || p.K <= 1) && (p.b_sl % 4 == 0);

    const bool tma_ok = plan->avec && plan->bvec && tma_supported(p);
    int variant       = a->variant;
    if (variant == KM_VARIANT_TMA && !tma_ok)
        return fail(KM_ERR_BAD_STRIDE, "the TMA variant needs m-contiguous, 16-byte aligned a and b with 16-byte pitches");
    if (variant == KM_VARIANT_AUTO) variant = (tma_ok && tma_preferred(p)) ? KM_VARIANT_TMA : KM_VARIANT_CPASYNC;
    plan->variant = variant;
    plan->awide   = small_wide_loads(p.A, p.a_sm, p.a_sk, p.a_sl, p.K, p.L);
    plan->bwide   = small_wide_loads(p.B, p.b_sn, p.b_sk, p.b_sl, p.K, p.L);
    plan->automatic = a->variant == KM_VARIANT_AUTO;
    plan->small     = plan->automatic && small_supported(p) &&
                      small_preferred(p, plan->avec, plan->bvec, plan->awide, plan->bwide);
    return 0;
}

// Which operands of a planned call are worth rewriting k-major first.
struct PackPlan {
    PackJob job[2];
    int     n;            // operands to pack; 0: none
    bool    a, b;         // (kernel-side A / B)
    bool    shared;       // B is the same matrix as A
    long long floats[2];
};

// Measured on B200, the 64 x 64 kernel on torch rows against the kernel that packed operands take, us:
//   square  4000^2 x 64: 82 / 70   8000^2 x 96: 431 / 382   4000^2 x 512: 568 / 509   16384^2 x 512: 9050 / 8030
//   |.|     8000^2 x 96: 429 / 427   4000^2 x 512: 568 / 569   16384^2 x 512: 9090 / 8800
//   |.|^1.3 8000^2 x 96: 1708 / 1722   4000^2 x 512: 2255 / 2260   16384^2 x 512: 36650 / 36660
// so a pair and feature costs 7.4e-15 s less for the square and product steps, and 2e-15 s for |.| where packed
// operands go to the 128 x 128 kernel.  An operand that could only be copied word by word costs 1e-14 s more
// (square 8001 x 8003 x 300: 1561 us, packed 1150; |.| 1727 / 1250; |.|^1.3 5873 / 5429).  Packing must save half as much again as it costs.
void plan_pack_operands(const BuildPlan& plan, PackPlan* pack) {
    std::memset(pack, 0, sizeof(*pack));
    const BuildParams& p = plan.p;
    if ((plan.avec && plan.bvec) || p.M == 0 || p.N == 0 || !plan.automatic || !small_supported(p)) return;
    double gain = 7.4e-15;
    if (p.inner_id == IN_DIFF_ABS) gain = small_preferred(p, true, true, true, true) ? 0.0 : 2e-15;
    if (p.inner_id == IN_DIFF_POW) gain = 0.0;
    gain += ((plan.awide ? 0 : 1) + (plan.bwide ? 0 : 1)) * 1e-14;
    if (gain == 0.0) return;
    const double tiles = p.symmetric ? 0.5 * p.tiles_n * (p.tiles_n + 1.0) : (double)p.tile_count;
    const double pairs = tiles * p.L * std::min((double)BUILD_TILE, (double)p.M) * std::min((double)BUILD_TILE, (double)p.N);
    pack->a      = !plan.avec;
    pack->b      = !plan.bvec;
    pack->shared = p.A == p.B && p.M == p.N && p.a_sm == p.b_sn && p.a_sk == p.b_sk && p.a_sl == p.b_sl;
    if (pack->a) {
        pack->floats[pack->n] = plan_pack(&pack->job[pack->n], p.A, p.M, p.K, p.L, p.a_sm, p.a_sk, p.a_sl);
        ++pack->n;
    }
    if (pack->b && !pack->shared) {
        pack->floats[pack->n] = plan_pack(&pack->job[pack->n], p.B, p.N, p.K, p.L, p.b_sn, p.b_sk, p.b_sl);
        ++pack->n;
    }
    const long long floats = pack->floats[0] + pack->floats[1];
    if (pairs * p.K * gain < 1.5 * pack_seconds(floats) || floats * 4 > PACK_MAX_BYTES) pack->n = 0;
}

// The same call on the operands packed into `scratch` (plan.swapped: the kernel's A is the caller's b).
KmBuildArgs packed_arguments(const KmBuildArgs& args, const BuildPlan& plan, PackPlan* pack, void* scratch) {
    pack->job[0].dst = static_cast<float*>(scratch);
    pack->job[1].dst = pack->job[0].dst + pack->floats[0];
    KmBuildArgs packed = args;
    auto use_a = [&](const PackJob& j) { packed.a = j.dst; packed.a_stride_m = 1; packed.a_stride_k = j.pitch; packed.a_stride_l = j.dst_l; };
    auto use_b = [&](const PackJob& j) { packed.b = j.dst; packed.b_stride_n = 1; packed.b_stride_k = j.pitch; packed.b_stride_l = j.dst_l; };
    if (pack->a) { if (plan.swapped) use_b(pack->job[0]); else use_a(pack->job[0]); }
    if (pack->b) {
        const PackJob& j = pack->job[pack->a && !pack->shared ? 1 : 0];
        if (plan.swapped) use_a(j); else use_b(j);
    }
    return packed;
}

const char* const kInnerNames[IN_COUNT] = {"diff_abs", "diff_square", "diff_pow", "diff_noop", "diff_sqrt", "diff_pow",
                                           "dot_noop", "dot_abs",     "dot_square", "dot_sqrt", "dot_pow"};

}  // namespace
}  // namespace km

namespace km {
namespace {

int launch_plan(const BuildPlan& plan, cudaStream_t st) {
    const BuildParams& p = plan.p;
    if (plan.small) return launch_build_small(p, plan.variant == KM_VARIANT_TMA, st);
    if (plan.variant == KM_VARIANT_TMA) return launch_build_tma(p, st);

    BuildKernelFn fn = cpasync_kernel(kernel_inner(p), plan.avec, plan.bvec, p.symmetric != 0);
    if (!fn) return fail(KM_ERR_INTERNAL, "no kernel for inner id %d", p.inner_id);
    if (int rc = cuda_status(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, BUILD_CPA_SMEM_BYTES),
                             "cudaFuncSetAttribute(build_cpasync_kernel)"))
        return rc;
    const int total_l = p.L;
    for (int l0 = 0; l0 < total_l; l0 += 65535) {
        BuildParams q = p;
        q.L           = (total_l - l0 < 65535) ? (total_l - l0) : 65535;
        q.A += (long long)l0 * p.a_sl;
        q.B += (long long)l0 * p.b_sl;
        q.C += (long long)l0 * p.c_sl;
        if (q.p_inner.ptr) q.p_inner.ptr += (long long)l0 * q.p_inner.batch_stride;
        if (q.p_outer.ptr) q.p_outer.ptr += (long long)l0 * q.p_outer.batch_stride;
        if (q.bandwidth.ptr) q.bandwidth.ptr += (long long)l0 * q.bandwidth.batch_stride;
        if (q.regularization.ptr) q.regularization.ptr += (long long)l0 * q.regularization.batch_stride;
        dim3 grid((unsigned)q.tile_count, (unsigned)q.L, 1);
        if (int rc = cuda_status(launch_overlapped(fn, grid, BUILD_CPA_THREADS, BUILD_CPA_SMEM_BYTES, st, q),
                                 "launch of build_cpasync_kernel"))
            return rc;
    }
    return 0;
}

}  // namespace
}  // namespace km

extern "C" int kermac_b200_build_kernel(const KmBuildArgs* args, void* stream) {
    using namespace km;
    BuildPlan plan;
    if (int rc = make_plan(args, &plan)) return rc;
    if (plan.p.M == 0 || plan.p.N == 0 || plan.p.tile_count == 0) return 0;
    if (int rc = require_sm100()) return rc;
    return launch_plan(plan, static_cast<cudaStream_t>(stream));
}

extern "C" int64_t kermac_b200_build_scratch_bytes(const KmBuildArgs* args) {
    using namespace km;
    BuildPlan plan;
    if (make_plan(args, &plan)) return 0;
    PackPlan pack;
    plan_pack_operands(plan, &pack);
    return pack.n ? (int64_t)(pack.floats[0] + pack.floats[1]) * 4 : 0;
}

extern "C" int kermac_b200_build_kernel_scratch(const KmBuildArgs* args, void* scratch, int64_t scratch_bytes, void* stream) {
    using namespace km;
    BuildPlan plan;
    if (int rc = make_plan(args, &plan)) return rc;
    if (plan.p.M == 0 || plan.p.N == 0 || plan.p.tile_count == 0) return 0;
    if (int rc = require_sm100()) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    PackPlan pack;
    plan_pack_operands(plan, &pack);
    const int64_t need = (int64_t)(pack.floats[0] + pack.floats[1]) * 4;
    if (!pack.n || !scratch || !aligned16(scratch) || scratch_bytes < need) return launch_plan(plan, st);

    KmBuildArgs packed = packed_arguments(*args, plan, &pack, scratch);
    if (int rc = launch_pack(pack.job, pack.n, plan.p.K, st)) return rc;
    if (int rc = make_plan(&packed, &plan)) return rc;
    return launch_plan(plan, st);
}

extern "C" int64_t kermac_b200_build_tile_count(const KmBuildArgs* args) {
    using namespace km;
    if (!args) return fail(KM_ERR_NULL_POINTER, "args is NULL");
    KmBuildArgs whole = *args;
    whole.tile_first = whole.tile_count = 0;
    BuildPlan plan;
    if (int rc = make_plan(&whole, &plan)) return rc;
    return (int64_t)plan.p.tiles_m * plan.p.tiles_n;
}

extern "C" int kermac_b200_describe_variant(const KmBuildArgs* args, char* buf, int32_t buf_len) {
    using namespace km;
    if (!buf || buf_len <= 0) return fail(KM_ERR_NULL_POINTER, "buf is NULL or empty");
    BuildPlan plan;
    if (int rc = make_plan(args, &plan)) return rc;
    const BuildParams& p = plan.p;
    auto name  = [](const BuildPlan& q) { return q.variant == KM_VARIANT_TMA ? "tma" : "cpasync"; };
    int length = snprintf(buf, (size_t)buf_len,
             "build_kernel variant=%s inner=%s outer_power=%d kernel_type=%d exchanged=%d a_vec16=%d b_vec16=%d "
             "out_vec16=%d tiles=%dx%d batches=%d symmetric=%d tile_range=%d+%d kernel_tile=%d%s",
             name(plan), kInnerNames[p.inner_id], p.outer_power, p.kernel_type,
             plan.swapped ? 1 : 0, plan.avec ? 1 : 0, plan.bvec ? 1 : 0, p.c_vec4, p.tiles_m, p.tiles_n, p.L, p.symmetric,
             p.tile_first, p.tile_count, plan.small ? 64 : BUILD_TILE,
             plan.variant != KM_VARIANT_TMA && kernel_inner(p) == IN_DIFF_POW_TABLE ? " pow=table" : "");
    // what kermac_b200_build_kernel_scratch does with as much scratch as it asks for (any aligned address stands for it)
    PackPlan pack;
    plan_pack_operands(plan, &pack);
    if (!pack.n || length < 0 || length >= buf_len) return 0;
    const long long bytes = (pack.floats[0] + pack.floats[1]) * 4;
    KmBuildArgs packed    = packed_arguments(*args, plan, &pack, reinterpret_cast<void*>(uintptr_t{256}));
    if (int rc = make_plan(&packed, &plan)) return rc;
    snprintf(buf + length, (size_t)(buf_len - length), "; with %lld bytes of scratch: operands packed, variant=%s kernel_tile=%d",
             bytes, name(plan), plan.small ? 64 : BUILD_TILE);
    return 0;
}
