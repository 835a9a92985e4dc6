// Operands rewritten k-major (declarations; implementation in km_pack.cu).
#pragma once

#include "km_host.h"

namespace km {

// One operand: `count` points of K features, element (l, t, k) at src[l * s_l + t * s_t + k * s_k] (s_l 0: one
// batch entry for all), to be written to dst[l * dst_l + k * pitch + t].
struct PackJob {
    const float* src; long long s_t, s_k, s_l;
    float*       dst; long long pitch, dst_l;
    int count, L;
};

// Fills the destination's geometry (dst itself stays NULL) and returns its size in floats: rows of a multiple
// of 32 floats, so a 16-byte aligned dst satisfies what TMA and 16-byte copies need.
long long plan_pack(PackJob* job, const float* src, int count, int K, int L, long long s_t, long long s_k, long long s_l);

// Packs one or two operands in one launch; K >= 1.
int launch_pack(const PackJob* jobs, int n, int K, cudaStream_t stream);

// Packing takes at most this much scratch (0.6 % of the device), so that a call on a few points against very many
// does not take a copy of its data set from a caller who counts on the memory; larger operands are read as they lie.
constexpr long long PACK_MAX_BYTES = 1LL << 30;

// Seconds a pack of `floats` elements adds to a call.
double pack_seconds(long long floats);

}  // namespace km
