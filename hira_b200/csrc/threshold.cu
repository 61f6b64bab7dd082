// Threshold (tau) finders, on device.
//
// The reference declares sample_max(samples, query) and
// sample_mean_topk(samples, query, k) (cache/threshold_finder.py:1-14, selected
// by HiraConfig.threshold_method / sample_size, cache/hira_config.py:22-23) but
// both raise NotImplementedError; the meaning implemented here is the one the
// names state: score a sample of keys against the query, then take the maximum
// or the mean of the k largest scores.  hira_kth_score gives the exact k-th
// largest score over a whole head (used to set tau so that a given number of
// keys survives).
#include "common.cuh"
#include <type_traits>
#include <math_constants.h>

namespace hira {

constexpr int TAU_MAX_SAMPLES = 4096;
constexpr int TAU_LIST = 32;   // longest list the merge tree keeps: one entry per lane

// descending sort of one key per lane
__device__ __forceinline__ uint32_t warp_sort_desc(uint32_t v, int wl) {
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            const uint32_t o = __shfl_xor_sync(0xffffffffu, v, stride);
            const bool want_max = ((wl & size) == 0) == ((wl & stride) == 0);
            v = want_max ? max(v, o) : min(v, o);
        }
    }
    return v;
}
// the 32 largest of two descending lists of 32, descending: max(a[i], b[31 - i]) is bitonic and holds them
__device__ __forceinline__ uint32_t warp_merge_top(uint32_t a, uint32_t b, int wl) {
    uint32_t v = max(a, __shfl_sync(0xffffffffu, b, 31 - wl));
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1) {
        const uint32_t o = __shfl_xor_sync(0xffffffffu, v, stride);
        v = (wl & stride) == 0 ? max(v, o) : min(v, o);
    }
    return v;
}

// One CTA per query head: every sample scored (canonical dot product), then the k largest scores in
// descending order.  The work is a chain of latencies, not bytes (1000 bf16 samples of 128 channels are
// 256 KB out of L2): ROWS rows per group are loaded together, and 1024 threads leave two such rounds.
// Up to 32 wanted scores need no sort of all samples: each warp sorts its scores 32 at a time in
// registers and keeps the 32 largest, and the warps' lists are merged pairwise (5 rounds for 32 warps);
// only a larger k goes through the bitonic sort of the whole array.
// Scores travel as order-preserving integers; a NaN score sorts last.
// Measured, 1000 bf16 samples, D = 128, k = 16: 32.3 -> 8.4 us for 32 query heads (256 threads, one row in
// flight per group and a 55-step bitonic sort before), 42.0 -> 8.9 us for 64.
template <typename T, int NCH, int TH, int PER_SM>
__global__ void __launch_bounds__(TH, PER_SM)
threshold_kernel(const T* __restrict__ samples, long long head_stride, int n_samples, int dim,
                 const float* __restrict__ q, const int32_t* __restrict__ q2kv, int group, int method, int k,
                 float* __restrict__ tau_out) {
    constexpr int HW = TH / GROUP;
    // 128 bytes of rows in flight per lane; 64 of wide bf16 rows where four CTAs are to fit an SM
    constexpr int ROWS = NCH == 4 && PER_SM == 4 ? 1 : 16 / ((int)sizeof(T) * NCH);
    __shared__ uint32_t s[TAU_MAX_SAMPLES];
    const int tid = threadIdx.x, lane = tid & (GROUP - 1), hw = tid / GROUP, warp = tid >> 5, wl = tid & 31;
    grid_wait();
    grid_trigger();
    const int qh = blockIdx.x;
    const int h = q2kv ? q2kv[qh] : qh / group;
    const T* rows = samples + (size_t)h * head_stride;
    float qreg[NCH][8];
    load_vec_f32<NCH>(q + (size_t)qh * dim, qreg, lane, dim);
    int n2 = TAU_LIST;
    while (n2 < n_samples) n2 <<= 1;
    for (int b = 0; b < n2; b += HW * ROWS) {  // uniform trip count
        RawChunk<T> raw[ROWS][NCH];
#pragma unroll
        for (int u = 0; u < ROWS; ++u) {
            const int i = b + u * HW + hw;
#pragma unroll
            for (int ci = 0; ci < NCH; ++ci) {
                const int c = lane + GROUP * ci;
                if (i < n_samples && c * 8 < dim) raw[u][ci] = load_chunk<T>(rows + (size_t)i * dim, c);
                else raw[u][ci] = zero_chunk<T>();
            }
        }
#pragma unroll
        for (int u = 0; u < ROWS; ++u) {
            const int i = b + u * HW + hw;
            Acc2 acc{0.f, 0.f};
#pragma unroll
            for (int ci = 0; ci < NCH; ++ci) {
                if ((lane + GROUP * ci) * 8 < dim) {
                    float a[8];
                    to_float(raw[u][ci], a);
                    chunk_fma(acc, a, qreg[ci]);
                }
            }
            const float d = group_sum(__fadd_rn(acc.e, acc.o));
            if (lane == 0 && i < n2) s[i] = (i < n_samples && d == d) ? order_key(d) : 0u;  // padding sorts last
        }
    }
    __syncthreads();
    const int want = method == HIRA_TAU_SAMPLE_MAX ? 1 : k;
    if (want <= TAU_LIST) {
        constexpr int WARPS = TH / 32;
        uint32_t best = 0u;
        for (int i = warp * 32; i < n2; i += TH) best = warp_merge_top(best, warp_sort_desc(s[i + wl], wl), wl);
        int live = n2 / 32 < WARPS ? n2 / 32 : WARPS;   // warps that hold a list: a power of two
        for (; live > 1; live >>= 1) {
            __syncthreads();
            if (warp >= live / 2 && warp < live) s[(warp - live / 2) * 32 + wl] = best;
            __syncthreads();
            if (warp < live / 2) best = warp_merge_top(best, s[warp * 32 + wl], wl);
        }
        __syncthreads();
        if (warp == 0) s[wl] = best;
    } else {
        // bitonic sort, descending
        for (int size = 2; size <= n2; size <<= 1) {
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int i = tid; i < n2; i += TH) {
                    const int j = i ^ stride;
                    if (j > i) {
                        const bool desc = (i & size) == 0;
                        const uint32_t a = s[i], b = s[j];
                        if (desc ? (a < b) : (a > b)) { s[i] = b; s[j] = a; }
                    }
                }
                __syncthreads();
            }
        }
    }
    __syncthreads();
    if (tid == 0) {
        float t;
        if (method == HIRA_TAU_SAMPLE_MAX) {
            t = key_to_float(s[0]);
        } else if (method == HIRA_TAU_SAMPLE_KTH) {
            t = key_to_float(s[k - 1]);
        } else {
            float sum = 0.f;
            for (int i = 0; i < k; ++i) sum = __fadd_rn(sum, key_to_float(s[i]));
            t = __fdiv_rn(sum, (float)k);
        }
        tau_out[qh] = t;
    }
}

// radix select, 8 bits per pass, over the compacted scores of one query head
__global__ void __launch_bounds__(1024)
kth_kernel(const float* __restrict__ score, const int32_t* __restrict__ count, long long cap_children,
           int n_tiles, int n_tiles_active, int tile_rows, const int32_t* __restrict__ kk,
           float* __restrict__ tau_out) {
    __shared__ unsigned int hist[256];
    __shared__ unsigned int s_prefix, s_remaining;
    const int qh = blockIdx.x;
    const int tid = threadIdx.x;
    const float* sc = score + (size_t)qh * cap_children;
    const int32_t* cnt = count + (size_t)qh * n_tiles;
    uint32_t prefix = 0, prefix_mask = 0;
    uint32_t remaining = (uint32_t)kk[qh];
    bool fail = kk[qh] < 1;
    for (int pass = 0; pass < 4 && !fail; ++pass) {
        const int shift = 24 - 8 * pass;
        if (tid < 256) hist[tid] = 0;
        __syncthreads();
        for (int t = 0; t < n_tiles_active; ++t) {
            const int c = cnt[t];
            for (int i = tid; i < c; i += blockDim.x) {
                const uint32_t key = order_key(sc[(size_t)t * tile_rows + i]);
                if ((key & prefix_mask) == prefix) atomicAdd(&hist[(key >> shift) & 0xff], 1u);
            }
        }
        __syncthreads();
        if (tid == 0) {
            uint32_t acc = 0;
            int d = 255;
            for (; d >= 0; --d) {
                if (acc + hist[d] >= remaining) break;
                acc += hist[d];
            }
            if (d < 0) {
                s_prefix = 0xffffffffu; s_remaining = 0;  // fewer than k scores
            } else {
                s_prefix = (uint32_t)d; s_remaining = remaining - acc;
            }
        }
        __syncthreads();
        if (s_remaining == 0) { fail = true; }
        else {
            prefix |= s_prefix << shift;
            prefix_mask |= 0xffu << shift;
            remaining = s_remaining;
        }
        __syncthreads();
    }
    if (tid == 0) tau_out[qh] = fail ? -CUDART_INF_F : key_to_float(prefix);
}

// q_hat = q / ||q|| (fp32) and the per-head logit scale ||q|| * softmax_scale: the unit query
// and `scaling` the reference's searchers expect (searcher/cpu.py:58-63), in one launch.
template <typename T>
__global__ void __launch_bounds__(128)
prepare_query_kernel(const T* __restrict__ q, int dim, float sm_scale, float* __restrict__ q_hat,
                     float* __restrict__ logit_scale) {
    __shared__ float s_part[4];
    grid_trigger();   // launched plainly: everything before it is complete
    const int qh = blockIdx.x, tid = threadIdx.x;
    const T* row = q + (size_t)qh * dim;
    float acc = 0.f;
    for (int d = tid; d < dim; d += 128) {
        const float v = (float)row[d];
        acc = __fmaf_rn(v, v, acc);
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((tid & 31) == 0) s_part[tid >> 5] = acc;
    __syncthreads();
    const float nrm = fmaxf(__fsqrt_rn(s_part[0] + s_part[1] + s_part[2] + s_part[3]), 1e-20f);
    for (int d = tid; d < dim; d += 128) q_hat[(size_t)qh * dim + d] = __fdiv_rn((float)row[d], nrm);
    if (tid == 0) logit_scale[qh] = nrm * sm_scale;
}

}  // namespace hira

using namespace hira;

extern "C" int hira_prepare_query(const void* q, int32_t dtype, int32_t n_qheads, int32_t dim, float sm_scale,
                                  float* q_hat, float* logit_scale, void* stream) {
    HIRA_CHECK_ARG(q && q_hat && logit_scale, HIRA_ERR_ARG, "hira_prepare_query: NULL argument");
    HIRA_CHECK_ARG(dtype == HIRA_F32 || dtype == HIRA_BF16, HIRA_ERR_DTYPE, "hira_prepare_query: dtype %d", dtype);
    HIRA_CHECK_ARG(n_qheads >= 1 && dim >= 1, HIRA_ERR_SHAPE, "hira_prepare_query: n_qheads=%d dim=%d", n_qheads, dim);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (dtype == HIRA_BF16)
        prepare_query_kernel<<<n_qheads, 128, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(q), dim, sm_scale, q_hat, logit_scale);
    else
        prepare_query_kernel<<<n_qheads, 128, 0, s>>>(reinterpret_cast<const float*>(q), dim, sm_scale, q_hat, logit_scale);
    HIRA_CHECK_LAUNCH("hira_prepare_query launch");
    return HIRA_OK;
}


extern "C" int hira_threshold(const void* samples, int32_t dtype, int32_t n_heads, int32_t n_samples,
                              int32_t dim, int64_t head_stride, const float* q, const int32_t* q2kv,
                              int32_t n_qheads, int32_t method, int32_t k, float* tau_out, void* stream) {
    HIRA_CHECK_ARG(samples && q && tau_out, HIRA_ERR_ARG, "hira_threshold: NULL argument");
    HIRA_CHECK_ARG(dtype == HIRA_F32 || dtype == HIRA_BF16, HIRA_ERR_DTYPE, "hira_threshold: dtype %d", dtype);
    HIRA_CHECK_ARG(n_samples >= 1 && n_samples <= TAU_MAX_SAMPLES, HIRA_ERR_CAPACITY,
                   "hira_threshold: n_samples=%d outside 1..%d", n_samples, TAU_MAX_SAMPLES);
    HIRA_CHECK_ARG(dim >= 8 && dim <= 256 && dim % 8 == 0, HIRA_ERR_SHAPE, "hira_threshold: dim=%d", dim);
    HIRA_CHECK_ARG(n_heads >= 1 && n_qheads >= 1 && (q2kv || n_qheads % n_heads == 0), HIRA_ERR_SHAPE,
                   "hira_threshold: n_heads=%d n_qheads=%d", n_heads, n_qheads);
    HIRA_CHECK_ARG(method >= 0 && method <= 2, HIRA_ERR_ARG, "hira_threshold: unknown method %d", method);
    HIRA_CHECK_ARG(method == HIRA_TAU_SAMPLE_MAX || (k >= 1 && k <= n_samples), HIRA_ERR_ARG,
                   "hira_threshold: k=%d outside 1..n_samples=%d", k, n_samples);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int group = q2kv ? 1 : n_qheads / n_heads;
    const bool wide = dim > 128;  // chunks per lane: 2 up to 128 elements, else 4
    const dim3 grid((unsigned)n_qheads);
    cudaError_t e;
    auto run = [&](auto kern, const auto* rows, int threads) {
        e = launch_chained(kern, grid, dim3((unsigned)threads), 0, s, rows, (long long)head_stride, (int)n_samples, (int)dim, q, q2kv,
                           group, (int)method, (int)k, tau_out);
    };
    // One CTA a query head, and as many threads as leave all CTAs resident: 1024 while there is an SM for each,
    // smaller ones beyond that and for few samples.  bf16 samples of 128 channels, us with 1024, 512 and 256 threads:
    // 128 heads x 1,000, k = 16: 8.3, 9.1, 12.4;  256 heads 15.5, 12.6, 13.9;  512 heads 29.7, 23.4, 21.4 (k = 33,
    // 62.6, 51.0, 47.1);  512 heads x 16: 14.6, 7.3, 4.1;  32 heads x 100: 4.7, 3.8, 3.5;  384 heads x 4,096 64, 67,
    // 76 (k = 82, 174, 179, 212).  Rows above 128 channels (200): 512 heads x 1,000, k = 33 85 with 512 threads, 73
    // with 256 of three CTAs an SM, 57 with four;  384 heads 64, 45, 56.
    auto sized = [&](const auto* rows) {
        typedef typename std::remove_const<typename std::remove_pointer<decltype(rows)>::type>::type T;
        if (wide) {
            if (n_qheads > 3 * SM_COUNT) run(threshold_kernel<T, 4, 256, 4>, rows, 256);
            else if (n_qheads > (n_samples <= 128 ? 1 : 2) * SM_COUNT) run(threshold_kernel<T, 4, 256, 3>, rows, 256);
            else run(threshold_kernel<T, 4, 512, sizeof(T) == 4 ? 2 : 1>, rows, 512);   // bf16 would spill at two
        } else {
            if (n_samples <= 128 || n_qheads > (n_samples > 1024 ? 3 : 2) * SM_COUNT) run(threshold_kernel<T, 2, 256, 4>, rows, 256);
            else if (n_qheads > SM_COUNT) run(threshold_kernel<T, 2, 512, 2>, rows, 512);
            else run(threshold_kernel<T, 2, 1024, 1>, rows, 1024);
        }
    };
    if (dtype == HIRA_BF16) sized(reinterpret_cast<const __nv_bfloat16*>(samples));
    else sized(reinterpret_cast<const float*>(samples));
    if (e != cudaSuccess) {
        set_error("hira_threshold launch: %s", cudaGetErrorString(e));
        return HIRA_ERR_CUDA;
    }
    return HIRA_OK;
}

extern "C" int hira_kth_score(const hira_index_t* ix, int32_t n_qheads, int32_t tile_parents,
                              const float* score, const int32_t* count, const int32_t* k, float* tau_out,
                              void* stream) {
    int rc = validate_index(ix, false);
    if (rc != HIRA_OK) return rc;
    HIRA_CHECK_ARG(score && count && k && tau_out, HIRA_ERR_ARG, "hira_kth_score: NULL argument");
    HIRA_CHECK_ARG(n_qheads >= 1 && tile_parents >= 1, HIRA_ERR_SHAPE, "hira_kth_score: n_qheads=%d tile_parents=%d",
                   n_qheads, tile_parents);
    const int n_tiles = (ix->cap_parents + tile_parents - 1) / tile_parents;
    kth_kernel<<<n_qheads, 1024, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        score, count, (long long)ix->cap_parents * ix->bf, n_tiles, active_tiles(ix, tile_parents), tile_parents * ix->bf, k,
        tau_out);
    HIRA_CHECK_LAUNCH("hira_kth_score launch");
    return HIRA_OK;
}
