// Rewrites points held as torch rows (k contiguous, or any layout that cannot be copied 16 bytes at a time
// along the points) k-major into scratch, which the TMA-staged kernels read.
//
// Bound by memory: every element is read and written once, 64 points x 32 k per block through shared
// memory, so that both sides move whole 128-byte lines.
#include "km_common.cuh"
#include "km_pack.h"

namespace km {
namespace {

constexpr int PK_POINTS  = 64;
constexpr int PK_K       = 32;
constexpr int PK_THREADS = 256;

struct PackParams {
    PackJob job[2];
    int first_blocks;      // blocks of job[0]
    int K, ktiles;
};

__global__ void __launch_bounds__(PK_THREADS) pack_kernel(const __grid_constant__ PackParams p) {
    __shared__ float tile[PK_K][PK_POINTS + 1];
    after_previous_grid();
    const bool second  = static_cast<int>(blockIdx.x) >= p.first_blocks;
    const PackJob& job = p.job[second ? 1 : 0];
    const int block    = second ? blockIdx.x - p.first_blocks : blockIdx.x;
    const int l        = blockIdx.y;
    if (l >= job.L) return;
    const int t0 = (block / p.ktiles) * PK_POINTS, k0 = (block % p.ktiles) * PK_K;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float* src = job.src + static_cast<long long>(l) * job.s_l;
    float* dst       = job.dst + static_cast<long long>(l) * job.dst_l;
    if (job.s_k == 1) {
#pragma unroll
        for (int r = 0; r < PK_POINTS / 8; ++r) {
            const int t = warp + r * 8;
            if (t0 + t < job.count && k0 + lane < p.K)
                tile[lane][t] = src[static_cast<long long>(t0 + t) * job.s_t + k0 + lane];
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < PK_K / 8; ++r) {
        const int k = warp + r * 8;
        if (k0 + k >= p.K) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int t = lane + h * 32;
            if (t0 + t >= job.count) continue;
            const float v = (job.s_k == 1) ? tile[k][t]
                                           : src[static_cast<long long>(t0 + t) * job.s_t + static_cast<long long>(k0 + k) * job.s_k];
            dst[static_cast<long long>(k0 + k) * job.pitch + t0 + t] = v;
        }
    }
}

}  // namespace

long long plan_pack(PackJob* job, const float* src, int count, int K, int L, long long s_t, long long s_k, long long s_l) {
    job->src = src; job->s_t = s_t; job->s_k = s_k; job->s_l = s_l;
    job->dst   = nullptr;
    job->count = count;
    job->L     = (s_l == 0) ? 1 : L;
    job->pitch = ceil_div_ll(count, 32) * 32;
    job->dst_l = (s_l == 0) ? 0 : job->pitch * K;
    return job->pitch * K * job->L;
}

double pack_seconds(long long floats) { return 4e-6 + static_cast<double>(floats) * 8.0 / 4e12; }

int launch_pack(const PackJob* jobs, int n, int K, cudaStream_t stream) {
    PackParams p;
    p.K      = K;
    p.ktiles = (int)ceil_div_ll(K, PK_K);
    long long blocks = 0;
    int L = 1;
    p.first_blocks = 0;
    for (int i = 0; i < 2; ++i) {
        p.job[i] = jobs[i < n ? i : 0];
        if (i >= n) continue;
        blocks += ceil_div_ll(jobs[i].count, PK_POINTS) * p.ktiles;
        if (i == 0) p.first_blocks = (int)blocks;
        if (jobs[i].L > L) L = jobs[i].L;
    }
    return cuda_status(launch_overlapped(pack_kernel, dim3((unsigned)blocks, (unsigned)L, 1), PK_THREADS, 0, stream, p),
                       "launch of pack_kernel");
}

}  // namespace km
