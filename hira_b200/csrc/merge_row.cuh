// Log-sum-exp merge of the softmax partials of one query head, by one thread block.
#pragma once
#include <math_constants.h>

namespace hira {

constexpr int MERGE_PARTS = 64;    // partials whose weights are staged together
constexpr int MERGE_FLIGHT = 16;   // output rows a thread loads ahead of its additions

// part_o / part_ml point at the head's row of part 0; part s lies s * {o,ml}_part_stride floats on.
//   out = sum_s e^{m_s-M} o_s / sum_s e^{m_s-M} l_s      (o_s unnormalised), or with normalised o_s
//   (sequence shards) o_s first scaled back by l_s.
// The partials are read past L1 (ld.global.cg): they may have been written by another GPU.
// Called by all threads of a block of whole warps (at most 32 of them).  The sums run over the parts one
// after another; the loads must not: each weight is fetched and exponentiated by one thread of the block
// and handed round through shared memory, and a thread has MERGE_FLIGHT rows of its channel in flight.
// 32 heads x 23 parts x 128 channels took 15.6 us when every thread walked the (m, l) list itself and waited
// for each row: the decode step around it (8 heads of 32,768 keys) went from 53.6 to 42.1 us.
__device__ __forceinline__ void merge_row(const float* part_o, const float* part_ml, long long o_part_stride,
                                          long long ml_part_stride, int n_parts, int vdim, int normalised,
                                          float* __restrict__ out, float* __restrict__ out_ml) {
    __shared__ float s_max[32];
    __shared__ float s_w[MERGE_PARTS], s_l[MERGE_PARTS];   // e^{m-M} (negative: the part is empty), l
    const int tid = threadIdx.x;
    float M = -CUDART_INF_F;
    for (int s = tid; s < n_parts; s += blockDim.x) M = fmaxf(M, __ldcg(part_ml + s * ml_part_stride));
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    if ((tid & 31) == 0) s_max[tid >> 5] = M;
    __syncthreads();
    for (int w = 0; w < (int)blockDim.x / 32; ++w) M = fmaxf(M, s_max[w]);
    for (int d0 = 0; d0 < vdim; d0 += blockDim.x) {
        const int d = d0 + tid;
        float L = 0.f, o = 0.f;
        for (int p0 = 0; p0 < n_parts; p0 += MERGE_PARTS) {
            const int np = min(n_parts - p0, MERGE_PARTS);
            __syncthreads();   // the weights of the parts before are consumed
            for (int i = tid; i < np; i += blockDim.x) {
                const float ms = __ldcg(part_ml + (p0 + i) * ml_part_stride);
                s_l[i] = __ldcg(part_ml + (p0 + i) * ml_part_stride + 1);
                s_w[i] = ms > -CUDART_INF_F ? __expf(ms - M) : -1.f;
            }
            __syncthreads();
            for (int b = 0; b < np; b += MERGE_FLIGHT) {
                float x[MERGE_FLIGHT];
#pragma unroll
                for (int u = 0; u < MERGE_FLIGHT; ++u)
                    x[u] = (b + u < np && d < vdim) ? __ldcg(part_o + (p0 + b + u) * o_part_stride + d) : 0.f;
#pragma unroll
                for (int u = 0; u < MERGE_FLIGHT; ++u) {
                    if (b + u < np && !(s_w[b + u] < 0.f)) {
                        const float w = s_w[b + u], l = s_l[b + u];
                        L = __fmaf_rn(l, w, L);
                        o = __fmaf_rn(normalised ? w * l : w, x[u], o);
                    }
                }
            }
        }
        if (d < vdim) out[d] = L > 0.f ? o / L : 0.f;
        if (out_ml && d == 0) {
            out_ml[0] = M;
            out_ml[1] = L;
        }
    }
}

}  // namespace hira
