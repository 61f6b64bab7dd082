// Index build: per head, per level, nearest-centroid assignment, capacity-bf
// grouping closest-first with overflow into free slots, blocked layout, radii.
//
// Follows CUDAIndexer.build (indexer/cuda.py:56-108):
//   _build_random_bf_level_batched (:200-336): K = ceil(n/bf) centres taken from
//     the points themselves, one nearest-centre assignment (cdist + argmin,
//     :244-245), each centre keeps its bf closest points in distance order
//     (:252-303), the overflow goes to the free slots (:309-334);
//   _build_parents_children_from_keys (:338-426) and
//   _build_grandparents_parents_children_from_keys (:428-538): blocked layout,
//     second level over the parent centres, child blocks move with their parent;
//   _compute_parent_radii_from_layout / _compute_grandparent_radii_from_layout
//     (:114-198).
// Differences by design: the (n, K) distance matrix is never materialised (the
// arg-min runs inside the contraction), the overflow fill is deterministic
// (ascending free slot <- overflow in (centre, distance) order) instead of a
// per-head randperm, optional Lloyd mean updates precede the final assignment,
// and counts/validity are written as explicit state.
#include "common.cuh"
#include <cub/block/block_scan.cuh>
#include <math_constants.h>
#include <string.h>

namespace hira {

int q8_refresh(const hira_index_t* ix, cudaStream_t s, long long parents_bound);
int launch_assign_tc(const void* points, long long p_head_stride, const void* cents, const float* csq,
                     int n_heads, int n, int k, int dim, int32_t* out_idx, float* out_d2, cudaStream_t s);
bool assign_tc_supported(int dtype, int n, int k, int dim);

// ---------------------------------------------------------------------------
// The assignment's arithmetic: one fp32 FMA chain over d = 0..D-1 starting from 0.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void memcpy_chunk(RawChunk<T>& raw, const T* src) {
    T e[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) e[j] = src[j];
    memcpy(&raw, e, sizeof(raw));
}

// One row per thread: the chain over d is serial by definition, so what counts is that the row's pieces are
// on their way before the chain needs them.  Eight 16-byte pieces are loaded ahead (before: one element per
// load; 8 x 1,024 bf16 centres of 128 channels: 18.5 -> 3.1 us).
constexpr int SQ_THREADS = 64;
constexpr int MEMBER_LISTS = 2;   // words behind the member counts, see member_starts_kernel
template <typename T>
__global__ void __launch_bounds__(SQ_THREADS)
sqnorm_seq_kernel(const T* __restrict__ rows, long long n_rows, int dim, float* __restrict__ out,
                  int32_t* __restrict__ zero) {
    const long long i = (long long)blockIdx.x * SQ_THREADS + threadIdx.x;
    if (i >= n_rows) return;
    constexpr int FLIGHT = 16 / (int)sizeof(T);   // 8-element chunks: 128 bytes of bf16, 128 of fp32
    const T* r = rows + i * dim;
    float acc = 0.f;
    const int chunks = dim / 8;
    const bool aligned = ((uintptr_t)r & 15) == 0;   // hira_assign takes rows at any address
    for (int c0 = 0; c0 < chunks; c0 += FLIGHT) {
        RawChunk<T> raw[FLIGHT];
#pragma unroll
        for (int u = 0; u < FLIGHT; ++u)
            if (c0 + u < chunks) {
                if (aligned) raw[u] = load_chunk<T>(r, c0 + u);
                else memcpy_chunk<T>(raw[u], r + (c0 + u) * 8);
            }
#pragma unroll
        for (int u = 0; u < FLIGHT; ++u) {
            if (c0 + u < chunks) {
                float f[8];
                to_float(raw[u], f);
#pragma unroll
                for (int e = 0; e < 8; ++e) acc = __fmaf_rn(f[e], f[e], acc);
            }
        }
    }
    out[i] = acc;
    if (zero) {   // the centre's member count and, behind the counts, the work lists' lengths, for the assignment that follows
        zero[i] = 0;
        if (i == 0)
            for (int u = 0; u < MEMBER_LISTS; ++u) zero[n_rows + u] = 0;
    }
}

// ---------------------------------------------------------------------------
// CUDA-core assignment: 128 points x 64 centres per step, 4 x 8 per thread.
//
// Every (point, centre) product is one FMA chain over d, so the chains of a thread are its only
// parallelism and shared memory has to keep up with them: both operands are staged transposed ([d][row]),
// a thread reads its 4 points and 8 centres of one d with three 128-bit loads and does 32 FMAs as 16
// packed ones.  (4 x 4 per thread out of row-major tiles, eight 32-bit loads for 16 FMAs, ran at 13 TFLOP/s;
// 8 x 4,096 fp32 points, 64 centres, D = 128: 39.8 -> 25.1 us.)
// ---------------------------------------------------------------------------
constexpr int AS_PTS = 128, AS_CTS = 64, AS_THREADS = 256;
constexpr int AS_LDX = AS_PTS + 4, AS_LDC = AS_CTS + 4;   // 16-byte rows whose 4-row stride is half the banks

// rows [r0, r0 + ROWS) of `src`, transposed into dst[d][row]; rows beyond n are zero.  16 lanes take 16 rows,
// the other half-warp the next chunk of them: 32-byte reads, and stores that meet no bank twice (fp32).
template <typename T, int ROWS, int LD>
__device__ __forceinline__ void stage_transposed(const T* __restrict__ src, int r0, int n, int dim, float* dst) {
    constexpr int E = 16 / (int)sizeof(T);   // elements of a 16-byte piece
    const int pieces = dim / E;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pairs = (pieces + 1) / 2;
    const bool aligned = ((uintptr_t)src & 15) == 0;   // rows are whole 16-byte pieces
    for (int t = warp; t < pairs * (ROWS / 16); t += AS_THREADS / 32) {
        const int r = (t % (ROWS / 16)) * 16 + (lane & 15);
        const int pc = (t / (ROWS / 16)) * 2 + (lane >> 4);
        if (pc >= pieces) continue;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (r0 + r < n) {
            const T* at = src + (size_t)(r0 + r) * dim + pc * E;
            if (aligned) {
                v = __ldg(reinterpret_cast<const uint4*>(at));
            } else {   // hira_assign takes rows at any address
                T e[E];
#pragma unroll
                for (int j = 0; j < E; ++j) e[j] = at[j];
                memcpy(&v, e, 16);
            }
        }
        float* w = dst + (size_t)pc * E * LD + r;
        if constexpr (sizeof(T) == 4) {
            w[0] = __uint_as_float(v.x); w[LD] = __uint_as_float(v.y); w[2 * LD] = __uint_as_float(v.z); w[3 * LD] = __uint_as_float(v.w);
        } else {
            float f[8];
            unpack_bf16x8(v, f);
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e * LD] = f[e];
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(AS_THREADS)
assign_kernel(const T* __restrict__ points, long long p_head_stride, const T* __restrict__ cents,
              const float* __restrict__ csq, int n, int k, int dim, int32_t* __restrict__ out_idx,
              float* __restrict__ out_d2) {
    extern __shared__ __align__(16) float sm[];
    float* xs = sm;                  // [dim][AS_LDX]
    float* cs = sm + dim * AS_LDX;   // [dim][AS_LDC]
    const int h = blockIdx.y;
    const int p0 = blockIdx.x * AS_PTS;
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;   // points 4 ty .. + 3, centres 4 tx .. + 3 and 32 + 4 tx .. + 3
    const T* C = cents + (size_t)h * k * dim;
    const float* CS = csq + (size_t)h * k;

    stage_transposed<T, AS_PTS, AS_LDX>(points + (size_t)h * p_head_stride, p0, n, dim, xs);
    float best_s[4];
    int best_i[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { best_s[i] = CUDART_INF_F; best_i[i] = 0x7fffffff; }

    for (int c0 = 0; c0 < k; c0 += AS_CTS) {
        __syncthreads();
        stage_transposed<T, AS_CTS, AS_LDC>(C, c0, k, dim, cs);
        __syncthreads();
        float2 acc[4][4];   // [point][centre pair]
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
        const float* xp = xs + 4 * ty;
        const float* cp = cs + 4 * tx;
#pragma unroll 4
        for (int d = 0; d < dim; ++d) {
            const float4 x = *reinterpret_cast<const float4*>(xp + d * AS_LDX);
            const float4 a = *reinterpret_cast<const float4*>(cp + d * AS_LDC);
            const float4 b = *reinterpret_cast<const float4*>(cp + d * AS_LDC + 32);
            const float xv[4] = {x.x, x.y, x.z, x.w};
            const float2 cv[4] = {make_float2(a.x, a.y), make_float2(a.z, a.w), make_float2(b.x, b.y), make_float2(b.z, b.w)};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = __ffma2_rn(make_float2(xv[i], xv[i]), cv[j], acc[i][j]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = c0 + (j >> 2) * 32 + 4 * tx + (j & 3);
            if (c < k) {
                const float cq = CS[c];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 p = acc[i][j >> 1];
                    const float s = __fsub_rn(cq, __fmul_rn(2.0f, (j & 1) ? p.y : p.x));
                    if (s < best_s[i] || (s == best_s[i] && c < best_i[i])) { best_s[i] = s; best_i[i] = c; }
                }
            }
        }
    }
    // the 8 threads (tx) that share a point; then its own squared norm, one point per thread
    float* rs = cs;                               // [AS_PTS]
    int* ri = reinterpret_cast<int*>(cs + AS_PTS);   // [AS_PTS]
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const float s = __shfl_xor_sync(0xffffffffu, best_s[i], o);
            const int c = __shfl_xor_sync(0xffffffffu, best_i[i], o);
            if (s < best_s[i] || (s == best_s[i] && c < best_i[i])) { best_s[i] = s; best_i[i] = c; }
        }
        if (tx == 0) { rs[4 * ty + i] = best_s[i]; ri[4 * ty + i] = best_i[i]; }
    }
    __syncthreads();
    if (tid < AS_PTS && p0 + tid < n) {
        float xsq = 0.f;
#pragma unroll 8
        for (int d = 0; d < dim; ++d) xsq = __fmaf_rn(xs[d * AS_LDX + tid], xs[d * AS_LDX + tid], xsq);
        out_idx[(size_t)h * n + p0 + tid] = ri[tid];
        out_d2[(size_t)h * n + p0 + tid] = fmaxf(__fadd_rn(xsq, rs[tid]), 0.f);
    }
}

template <typename T>
static int launch_assign_cc(const T* points, long long p_head_stride, const T* cents, const float* csq,
                            int n_heads, int n, int k, int dim, int32_t* out_idx, float* out_d2, cudaStream_t s) {
    const size_t smem = (size_t)dim * (AS_LDX + AS_LDC) * sizeof(float);   // dim >= 8: room for the 2 x [AS_PTS] of the end
    auto kern = assign_kernel<T>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) { set_error("assign: cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return HIRA_ERR_CUDA; }
    }
    dim3 grid((unsigned)((n + AS_PTS - 1) / AS_PTS), (unsigned)n_heads);
    kern<<<grid, AS_THREADS, smem, s>>>(points, p_head_stride, cents, csq, n, k, dim, out_idx, out_d2);
    HIRA_CHECK_LAUNCH("assign launch");
    return HIRA_OK;
}

static int run_assign(int dtype, const void* points, long long p_head_stride, const void* cents, float* csq,
                      int n_heads, int n, int k, int dim, int use_tc, int32_t* out_idx, float* out_d2,
                      cudaStream_t s, bool csq_ready = false, int32_t* zero = nullptr) {
    const long long rows = (long long)n_heads * k;
    const int blocks = (int)((rows + SQ_THREADS - 1) / SQ_THREADS);
    if (!csq_ready) {
        if (dtype == HIRA_BF16)
            sqnorm_seq_kernel<<<blocks, SQ_THREADS, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(cents), rows, dim, csq, zero);
        else
            sqnorm_seq_kernel<<<blocks, SQ_THREADS, 0, s>>>(reinterpret_cast<const float*>(cents), rows, dim, csq, zero);
        HIRA_CHECK_LAUNCH("sqnorm launch");
    }
    if (use_tc && assign_tc_supported(dtype, n, k, dim))
        return launch_assign_tc(points, p_head_stride, cents, csq, n_heads, n, k, dim, out_idx, out_d2, s);
    if (dtype == HIRA_BF16)
        return launch_assign_cc(reinterpret_cast<const __nv_bfloat16*>(points), p_head_stride,
                                reinterpret_cast<const __nv_bfloat16*>(cents), csq, n_heads, n, k, dim, out_idx, out_d2, s);
    return launch_assign_cc(reinterpret_cast<const float*>(points), p_head_stride,
                            reinterpret_cast<const float*>(cents), csq, n_heads, n, k, dim, out_idx, out_d2, s);
}

// ---------------------------------------------------------------------------
// Level build pieces.
// ---------------------------------------------------------------------------
// chunk c (8 elements) of a row; rows of a build lie on 16-byte boundaries
template <typename T>
__device__ __forceinline__ void copy_chunk(T* dst, const T* src, int c) {
    reinterpret_cast<RawChunk<T>*>(dst)[c] = load_chunk<T>(src, c);
}

template <typename T>
__global__ void gather_centres_kernel(const T* __restrict__ points, long long p_head_stride, int n,
                                      const int32_t* __restrict__ cent_idx, int k, int dim, T* __restrict__ cents) {
    // one thread per (head, centre, 8-element chunk)
    const int chunks = dim / 8;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int h = blockIdx.y;
    if (t >= (long long)k * chunks) return;
    const int c = (int)(t / chunks), ch = (int)(t % chunks);
    int src;
    if (cent_idx) {
        src = cent_idx[(size_t)h * k + c];
        src = src < 0 ? 0 : (src >= n ? n - 1 : src);
    } else {
        src = (int)(((long long)c * n) / k);  // evenly strided
    }
    copy_chunk(cents + ((size_t)h * k + c) * dim, points + (size_t)h * p_head_stride + (size_t)src * dim, ch);
}

// ---------------------------------------------------------------------------
// Members of every centre in (distance, point) order.
//
// The points of a head are counted per centre, the counts scanned, the points dropped into their centre's
// range in arrival order and each range sorted by itself.  The sort key is (distance bits, point), which no two
// members share, so the result does not depend on the arrival order.  A range is bf points on average and most are
// sorted by one warp in registers, but any of them can be anything up to all the points of a head (hubs, padding
// rows, constant keys): ranges of more than SORT_WARP members go to a work list in pieces of SORT_CTA, a piece is
// sorted by one CTA, and ranges of several pieces are merged MERGE_WAYS runs at a time by the whole GPU.
// (A device-wide radix sort of (centre, distance) before: 5 or 6 passes of about 9 us whatever the size.  8 x 4,096
// points in 64 centres, an iteration with all of the kernels around the sort: 73 -> 16 us; a build of 8 x 32,768
// points, both levels: radix sort 101 us, this 22 with 25 of small kernels.)
// ---------------------------------------------------------------------------
constexpr int SORT_THREADS = 256, SORT_RANGES = SORT_THREADS / 32, SORT_WARP = 128, SORT_CTA = 4096;
constexpr int SORT_PIECE_CTAS = 2 * SM_COUNT;   // CTAs of the sort that serve the work list
constexpr int MERGE_WAYS = 16, MERGE_UNIT = 1024, MERGE_FLIGHT = 5;
struct MemberLists {       // pieces as range << 32 | piece: of ranges above SORT_WARP, of ranges above SORT_CTA
    uint64_t *pieces, *merges;
    int32_t* len;          // [MEMBER_LISTS]: entries of the two
};
static size_t pieces_bound(size_t total) { return total / SORT_WARP + total / SORT_CTA + 1; }   // ceil(m / SORT_CTA) for every m > SORT_WARP
static size_t merges_bound(size_t total) { return 2 * (total / SORT_CTA) + 1; }                 // the same for every m > SORT_CTA

// An assignment outside [0, k) -- the tensor-core kernel writes -1 for the points of a CTA whose
// bounded barrier wait ran out -- must not reach the segment arithmetic below: the point goes to
// centre 0 at distance 0 (so that every later index stays in range) and the caller is told through
// the status word.
// `placed` (balanced rounds): points that already have a slot belong to no centre any more (arrival -1).
// The lanes of a warp that chose the same centre count it together: a centre that draws every point of a head
// would otherwise be one chain of n atomics.
__global__ void __launch_bounds__(256)
count_members_kernel(int32_t* __restrict__ idx, float* __restrict__ d2, int n, int k, long long total,
                     const int32_t* __restrict__ placed, int32_t* __restrict__ cnt, int32_t* __restrict__ arrival,
                     int32_t* __restrict__ status) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool counts = i < total && !(placed && placed[i] >= 0);
    int seg = -1;
    if (counts) {
        int c = idx[i];
        if (c < 0 || c >= k || !(d2[i] >= 0.f)) {
            if (status) atomicOr(status, HIRA_STATUS_ASSIGN_FAILED);
            idx[i] = c = 0;
            d2[i] = 0.f;
        }
        seg = (int)(i / n) * k + c;
    }
    const unsigned same = __match_any_sync(0xffffffffu, seg);
    const int wl = threadIdx.x & 31, leader = __ffs(same) - 1;
    int at = 0;
    if (counts && wl == leader) at = atomicAdd(cnt + seg, __popc(same));
    at = __shfl_sync(0xffffffffu, at, leader);
    if (i < total) arrival[i] = counts ? at + __popc(same & ((1u << wl) - 1u)) : -1;
}

// start[h][c] = h n + members of the centres before c; and the work lists
constexpr int SCAN_ITEMS = 4;
__global__ void __launch_bounds__(1024)
member_starts_kernel(const int32_t* __restrict__ cnt, int n, int k, int32_t* __restrict__ start, const MemberLists lists) {
    typedef cub::BlockScan<int, 1024> Scan;
    __shared__ typename Scan::TempStorage tmp;
    const int h = blockIdx.x;
    int carry = h * n;
    for (int c0 = 0; c0 < k; c0 += 1024 * SCAN_ITEMS) {
        int v[SCAN_ITEMS], total;
        const int c = c0 + threadIdx.x * SCAN_ITEMS;
#pragma unroll
        for (int u = 0; u < SCAN_ITEMS; ++u) {
            v[u] = c + u < k ? cnt[(size_t)h * k + c + u] : 0;
            if (v[u] > SORT_WARP) {
                const int np = (v[u] + SORT_CTA - 1) / SORT_CTA;
                const uint64_t range = (uint64_t)((size_t)h * k + c + u) << 32;
                int at = atomicAdd(lists.len, np);
                for (int p = 0; p < np; ++p) lists.pieces[at + p] = range | (uint32_t)p;
                if (np > 1) {
                    at = atomicAdd(lists.len + 1, np);
                    for (int p = 0; p < np; ++p) lists.merges[at + p] = range | (uint32_t)p;
                }
            }
        }
        Scan(tmp).ExclusiveSum(v, v, total);
        __syncthreads();
#pragma unroll
        for (int u = 0; u < SCAN_ITEMS; ++u)
            if (c + u < k) start[(size_t)h * k + c + u] = carry + v[u];
        carry += total;
    }
}

__global__ void drop_members_kernel(const int32_t* __restrict__ idx, const float* __restrict__ d2, int n, int k,
                                    long long total, const int32_t* __restrict__ start, const int32_t* __restrict__ arrival,
                                    uint64_t* __restrict__ keys) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int a = arrival[i];
    if (a < 0) return;
    const long long h = i / n;
    // d2 >= 0: bits order like values
    keys[start[h * k + idx[i]] + a] = ((uint64_t)__float_as_uint(d2[i]) << 32) | (uint32_t)(i - h * n);
}

// The first SORT_PIECE_CTAS (or fewer) CTAs take the pieces of the work list, each sorted in shared memory
// (bitonic): the whole range, or a run to be merged.  The CTAs behind them take SORT_RANGES ranges each, a warp
// a range: the rank of a member is the number of smaller keys.  Writes the member list and the rank of every
// point inside its range.
__global__ void __launch_bounds__(SORT_THREADS)
sort_members_kernel(const int32_t* __restrict__ cnt, const int32_t* __restrict__ start, int n, int k, long long n_seg,
                    int piece_ctas, const MemberLists lists, uint64_t* __restrict__ keys, uint32_t* __restrict__ sorted_ids,
                    int32_t* __restrict__ rank) {
    __shared__ uint64_t sk[SORT_CTA];   // SORT_RANGES x SORT_WARP of it while the warps work
    const int tid = threadIdx.x, warp = tid >> 5, wl = tid & 31;
    if ((int)blockIdx.x >= piece_ctas) {
        const long long seg = (long long)(blockIdx.x - piece_ctas) * SORT_RANGES + warp;
        const int m = seg < n_seg ? cnt[seg] : 0;
        if (m > 0 && m <= SORT_WARP) {
            const int b = start[seg];
            const size_t head = (size_t)(seg / k) * n;
            uint64_t* mine = sk + warp * SORT_WARP;
            for (int i = wl; i < m; i += 32) mine[i] = keys[b + i];
            __syncwarp();
            for (int i = wl; i < m; i += 32) {
                const uint64_t key = mine[i];
                int r = 0;
                for (int j = 0; j < m; ++j) r += mine[j] < key ? 1 : 0;
                const uint32_t id = (uint32_t)key;
                sorted_ids[b + r] = id;
                rank[head + id] = r;
            }
        }
        return;
    }
    const int n_pieces = lists.len[0];
    for (int e = blockIdx.x; e < n_pieces; e += piece_ctas) {   // every test below is uniform over the CTA
        const long long seg = (long long)(lists.pieces[e] >> 32);
        const int p0 = (int)(uint32_t)lists.pieces[e] * SORT_CTA;
        const int m = cnt[seg], np = min(m - p0, SORT_CTA);
        const int b = start[seg] + p0;
        const size_t head = (size_t)(seg / k) * n;
        int n2 = 2 * SORT_WARP;
        while (n2 < np) n2 <<= 1;
        __syncthreads();   // the piece before is written out
        for (int i = tid; i < n2; i += SORT_THREADS) sk[i] = i < np ? keys[b + i] : ~0ull;
        __syncthreads();
        for (int size = 2; size <= n2; size <<= 1) {
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int t = tid; t < n2 / 2; t += SORT_THREADS) {
                    const int i = 2 * t - (t & (stride - 1)), j = i + stride;
                    const bool up = (i & size) == 0;
                    const uint64_t x = sk[i], y = sk[j];
                    if ((x > y) == up) { sk[i] = y; sk[j] = x; }
                }
                __syncthreads();
            }
        }
        if (m <= SORT_CTA) {
            for (int i = tid; i < np; i += SORT_THREADS) {
                const uint32_t id = (uint32_t)sk[i];
                sorted_ids[b + i] = id;
                rank[head + id] = i;
            }
        } else {
            for (int i = tid; i < np; i += SORT_THREADS) keys[b + i] = sk[i];
        }
    }
}

// Ranges of more than `len` members, sorted in runs of `len`: up to MERGE_WAYS neighbouring runs become one.  A
// member's place is its place in its own run and, for each of the others, the number of smaller keys there, found
// by MERGE_FLIGHT bisections at a time; neighbouring lanes look for neighbouring keys, so most of their reads
// meet.  The pass that makes a range one run writes the member list and the ranks instead of keys.
// Bound by the latency of the bisections; what they cost is little beside the build around them: 8 x 131,072 equal
// bf16 keys, one range a head, 2.31 ms against 2.07 ms of random keys (7.29 ms when the CTA that sorted the pieces
// of a range also merged them in pairs; 2.75 ms with the radix sort), 8 x 32,768 0.51 and 0.48 ms (1.33; 0.98).
__global__ void __launch_bounds__(SORT_THREADS)
merge_members_kernel(const int32_t* __restrict__ cnt, const int32_t* __restrict__ start, int n, int k, int len,
                     const MemberLists lists, const uint64_t* __restrict__ from_all, uint64_t* __restrict__ to_all,
                     uint32_t* __restrict__ sorted_ids, int32_t* __restrict__ rank) {
    grid_wait();
    const int units = lists.len[1] * (SORT_CTA / MERGE_UNIT);
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
        const uint64_t entry = lists.merges[u / (SORT_CTA / MERGE_UNIT)];
        const long long seg = (long long)(entry >> 32);
        const int m = cnt[seg];
        if (m <= len) continue;   // one run already
        const int i0 = (int)(uint32_t)entry * SORT_CTA + u % (SORT_CTA / MERGE_UNIT) * MERGE_UNIT;
        const int b = start[seg];
        const uint64_t* from = from_all + b;
        const int run = i0 / len, first = run / MERGE_WAYS * MERGE_WAYS;
        const int runs = min(MERGE_WAYS, (m + len - 1) / len - first);
        const bool last = (long long)len * MERGE_WAYS >= m;
        const size_t head = (size_t)(seg / k) * n;
        for (int i = i0 + threadIdx.x; i < min(i0 + MERGE_UNIT, m); i += SORT_THREADS) {
            const uint64_t key = from[i];
            int at = first * len + (i - run * len);
            for (int s0 = 0; s0 < runs; s0 += MERGE_FLIGHT) {
                int lo[MERGE_FLIGHT], left[MERGE_FLIGHT];   // what is left to search: left[] keys from lo[] on
#pragma unroll
                for (int j = 0; j < MERGE_FLIGHT; ++j) {
                    const int s = first + s0 + j;
                    lo[j] = s * len;
                    left[j] = s0 + j < runs && s != run ? min(len, m - lo[j]) : 0;
                    at -= left[j] ? lo[j] : 0;
                }
                for (int reach = len; reach > 0; reach >>= 1) {
#pragma unroll
                    for (int j = 0; j < MERGE_FLIGHT; ++j) {
                        if (left[j] > 0) {
                            const int half = left[j] >> 1;
                            const bool below = from[lo[j] + half] < key;
                            lo[j] += below ? half + 1 : 0;
                            left[j] = below ? left[j] - half - 1 : half;
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < MERGE_FLIGHT; ++j) {
                    const int s = first + s0 + j;
                    if (s0 + j < runs && s != run) at += lo[j];
                }
            }
            if (last) {
                const uint32_t id = (uint32_t)key;
                sorted_ids[b + at] = id;
                rank[head + id] = at;
            } else {
                to_all[b + at] = key;
            }
        }
    }
}

// Lloyd mean update.  The members of a centre are added one after another in sorted order, so a centre is
// a serial chain; what it must not be is a chain of memory latencies.  One warp owns a slab of the
// channels of one centre (32 of fp32, 64 of bf16: one 128-byte piece of every member row) and keeps a ring of
// STAGES batches of 32 member rows in flight in shared memory ahead of the additions (each lane reads
// only what it copied itself).  Random centres have hubs -- thousands of members after the first assignment --
// and the longest chain is the time of the kernel.  8 x 4,096 fp32 keys of 128 channels, 64 centres: 42.1 us
// a call on average with one row of an 8-lane group in flight, 17.6 us with 32 rows in registers, 9.8 us
// with the ring.
constexpr int MEANS_BATCH = 32, MEANS_WARPS = 4;
template <typename T> struct MeansElem;
template <> struct MeansElem<float> {
    typedef float raw; static constexpr int N = 1;
    static __device__ __forceinline__ void get(raw r, float (&f)[1]) { f[0] = r; }
    static __device__ __forceinline__ raw put(const float (&f)[1]) { return f[0]; }
};
template <> struct MeansElem<__nv_bfloat16> {
    typedef uint32_t raw; static constexpr int N = 2;
    static __device__ __forceinline__ void get(raw r, float (&f)[2]) {
        f[0] = __uint_as_float(r << 16);
        f[1] = __uint_as_float(r & 0xffff0000u);
    }
    static __device__ __forceinline__ raw put(const float (&f)[2]) {
        const __nv_bfloat162 p = __floats2bfloat162_rn(f[0], f[1]);
        return *reinterpret_cast<const uint32_t*>(&p);
    }
};
template <typename T, int STAGES>
__global__ void __launch_bounds__(MEANS_WARPS * 32)
means_kernel(const T* __restrict__ points, long long p_head_stride, int n, const uint32_t* __restrict__ sorted_ids,
             const int32_t* __restrict__ start, const int32_t* __restrict__ count, int k, int dim, int slabs,
             long long n_seg, T* __restrict__ cents) {
    typedef MeansElem<T> E;
    typedef typename E::raw raw_t;
    extern __shared__ __align__(16) uint32_t ring_all[];
    const int wl = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long w = (long long)blockIdx.x * MEANS_WARPS + warp;
    const long long seg = w / slabs;
    if (seg >= n_seg) return;   // the whole warp
    const int d = ((int)(w - seg * slabs) * 32 + wl) * E::N;
    const int h = (int)(seg / k);
    const int b = start[seg], e = b + count[seg];
    if (e <= b) return;  // empty cluster keeps its centre
    const bool on = d < dim;
    const T* P = points + (size_t)h * p_head_stride + (on ? d : 0);
    uint32_t* ring = ring_all + warp * (STAGES * MEANS_BATCH * 32) + wl;   // [stage][row][lane]
    const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(ring);
    float sum[E::N];
#pragma unroll
    for (int j = 0; j < E::N; ++j) sum[j] = 0.f;
    const int batches = (e - b + MEANS_BATCH - 1) / MEANS_BATCH;   // uniform over the warp, as every test below
    auto load_ids = [&](int t) { const int m = b + t * MEANS_BATCH + wl; return m < e ? sorted_ids[m] : 0u; };
    auto issue = [&](int t, uint32_t ids) {
        if (t < batches) {
            const int np = min(MEANS_BATCH, e - b - t * MEANS_BATCH);
            const uint32_t dst = ring_s + (uint32_t)(t % STAGES) * (MEANS_BATCH * 128);
#pragma unroll
            for (int u = 0; u < MEANS_BATCH; ++u) {
                const uint32_t id = __shfl_sync(0xffffffffu, ids, u);
                if (u < np)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst + u * 128), "l"(P + (size_t)id * dim) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    uint32_t ids = load_ids(0);
#pragma unroll
    for (int t = 0; t < STAGES - 1; ++t) {
        const uint32_t next = load_ids(t + 1);
        issue(t, ids);
        ids = next;
    }
    for (int t = 0; t < batches; ++t) {
        const uint32_t next = load_ids(t + STAGES);
        issue(t + STAGES - 1, ids);
        ids = next;
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 1) : "memory");
        const int np = min(MEANS_BATCH, e - b - t * MEANS_BATCH);
        const uint32_t* src = ring + (t % STAGES) * (MEANS_BATCH * 32);
        if (np == MEANS_BATCH) {
#pragma unroll
            for (int u = 0; u < MEANS_BATCH; ++u) {
                float a[E::N];
                E::get(reinterpret_cast<const raw_t*>(src)[u * 32], a);
#pragma unroll
                for (int j = 0; j < E::N; ++j) sum[j] = __fadd_rn(sum[j], a[j]);
            }
        } else {
            for (int u = 0; u < np; ++u) {
                float a[E::N];
                E::get(reinterpret_cast<const raw_t*>(src)[u * 32], a);
#pragma unroll
                for (int j = 0; j < E::N; ++j) sum[j] = __fadd_rn(sum[j], a[j]);
            }
        }
    }
    if (!on) return;
    const float cnt = (float)(e - b);
#pragma unroll
    for (int j = 0; j < E::N; ++j) sum[j] = __fdiv_rn(sum[j], cnt);
    *reinterpret_cast<raw_t*>(cents + (size_t)seg * dim + d) = E::put(sum);
}

// Balanced rounds: centres that are full drop out of the next assignment (score +inf).
__global__ void mask_full_centres_kernel(const float* __restrict__ csq, const int32_t* __restrict__ filled, int bf,
                                         long long n_seg, float* __restrict__ csq_masked) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_seg) return;
    csq_masked[c] = filled[c] < bf ? csq[c] : CUDART_INF_F;
}

// An intermediate balanced round: every centre accepts, closest first, as many of the points that
// chose it as it still has room for; the rest stay unplaced for the next round.
__global__ void accept_kernel(const int32_t* __restrict__ idx, const int32_t* __restrict__ rank,
                              const int32_t* __restrict__ filled, int n, int k, int bf, long long total,
                              int32_t* __restrict__ slot) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total || slot[i] >= 0) return;   // placed earlier
    const int c = idx[i], r = rank[i];
    const int have = filled[(i / n) * k + c];
    if (r < bf - have) slot[i] = c * bf + have + r;
}
__global__ void accept_counts_kernel(const int32_t* __restrict__ count, int bf, long long n_seg,
                                     int32_t* __restrict__ filled) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_seg) return;
    const int cnt = count[c], room = bf - filled[c];
    filled[c] += cnt < room ? cnt : room;
}

// per head: exclusive scans of free slots and overflow counts over the centres; `filled` = slots
// taken in earlier balanced rounds (NULL without them)
__global__ void __launch_bounds__(1024)
capacity_scan_kernel(const int32_t* __restrict__ count, const int32_t* __restrict__ filled, int k, int bf,
                     int32_t* __restrict__ free_base, int32_t* __restrict__ left_base, int32_t* __restrict__ fill_cnt) {
    typedef cub::BlockScan<int, 1024> Scan;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ int s_total_left;
    const int h = blockIdx.x;
    const int32_t* ct = count + (size_t)h * k;
    auto fl = [&](int c) { return filled ? filled[(size_t)h * k + c] : 0; };
    int32_t* fb = free_base + (size_t)h * (k + 1);
    int32_t* lb = left_base + (size_t)h * (k + 1);
    int carry_f = 0, carry_l = 0;
    for (int c0 = 0; c0 < k; c0 += 1024) {
        const int c = c0 + threadIdx.x;
        int cnt = 0, room = 0;
        if (c < k) { cnt = ct[c]; room = bf - fl(c); }
        const int fr = (c < k) ? max(room - cnt, 0) : 0;
        const int lf = (c < k) ? max(cnt - room, 0) : 0;
        int ef, el, tf, tl;
        Scan(tmp).ExclusiveSum(fr, ef, tf);
        __syncthreads();
        Scan(tmp).ExclusiveSum(lf, el, tl);
        __syncthreads();
        if (c < k) { fb[c] = carry_f + ef; lb[c] = carry_l + el; }
        carry_f += tf; carry_l += tl;
    }
    if (threadIdx.x == 0) { fb[k] = carry_f; lb[k] = carry_l; s_total_left = carry_l; }
    __syncthreads();
    const int total_left = s_total_left;
    for (int c = threadIdx.x; c < k; c += 1024) {
        const int cnt = ct[c], room = bf - fl(c);
        const int fr = max(room - cnt, 0);
        int recv = total_left - fb[c];
        recv = recv < 0 ? 0 : (recv > fr ? fr : recv);
        fill_cnt[(size_t)h * k + c] = fl(c) + min(cnt, room) + recv;
    }
}

// slot (centre*bf + rank) of every point inside its level (the last round: everything is placed)
__global__ void placement_kernel(const int32_t* __restrict__ idx, const int32_t* __restrict__ rank,
                                 const int32_t* __restrict__ count, const int32_t* __restrict__ filled,
                                 const int32_t* __restrict__ free_base, const int32_t* __restrict__ left_base, int n,
                                 int k, int bf, long long total, bool some_placed, int32_t* __restrict__ slot) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total || (some_placed && slot[i] >= 0)) return;   // placed in an earlier balanced round
    const int h = (int)(i / n);
    const int c = idx[i], r = rank[i];
    auto fl = [&](int x) { return filled ? filled[(size_t)h * k + x] : 0; };
    const int room = bf - fl(c);
    int s;
    if (r < room) {
        s = c * bf + fl(c) + r;
    } else {
        const int32_t* fb = free_base + (size_t)h * (k + 1);
        const int L = left_base[(size_t)h * (k + 1) + c] + (r - room);
        // largest c2 with fb[c2] <= L and a free slot there: upper_bound(fb, L) - 1
        int lo = 0, hi = k;  // search in fb[0..k]
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (fb[mid] <= L) lo = mid; else hi = mid - 1;
        }
        // skip centres without free slots (fb equal runs): lo is the last index with fb[lo] <= L,
        // which has fb[lo+1] > L, hence at least one free slot
        const int cnt2 = count[(size_t)h * k + lo];
        s = lo * bf + fl(lo) + min(cnt2, bf - fl(lo)) + (L - fb[lo]);
    }
    slot[i] = s;
}

// Keys and values of every point to their slot, whole 16-byte pieces.  16 lanes share SCATTER_POINTS points:
// the slot of a point is looked up once for its key and its value row, and the pieces of all of them are in
// flight together.  8 x 32,768 bf16 keys and values of 128 channels: 38.7 us, 6.9 TB/s (62.9 us as two kernels).
constexpr int SCATTER_THREADS = 256, SCATTER_LANES = 16, SCATTER_POINTS = 2;
__global__ void __launch_bounds__(SCATTER_THREADS)
scatter_kv_kernel(const uint4* __restrict__ keys, long long k_head_pieces, int k_pieces, const uint4* __restrict__ values,
                  long long v_head_pieces, int v_pieces, int n, const int32_t* __restrict__ slot1,
                  const int32_t* __restrict__ slot2, int k1, int bf, uint4* __restrict__ children,
                  uint4* __restrict__ values_out, long long dst_head_rows, int32_t* __restrict__ slot2token, int token_base) {
    const int lane = threadIdx.x % SCATTER_LANES;
    const int i0 = (blockIdx.x * (SCATTER_THREADS / SCATTER_LANES) + threadIdx.x / SCATTER_LANES) * SCATTER_POINTS;
    const int h = blockIdx.y;
    size_t dst[SCATTER_POINTS];
    bool on[SCATTER_POINTS];
#pragma unroll
    for (int u = 0; u < SCATTER_POINTS; ++u) {
        on[u] = i0 + u < n;
        int s = on[u] ? slot1[(size_t)h * n + i0 + u] : 0;
        if (slot2) {
            const int c = s / bf, r = s - c * bf;
            s = slot2[(size_t)h * k1 + c] * bf + r;
        }
        dst[u] = (size_t)h * dst_head_rows + s;
        if (slot2token && on[u] && lane == 0) slot2token[dst[u]] = token_base + i0 + u;
    }
    const int most = k_pieces > v_pieces ? k_pieces : v_pieces;
    for (int p = lane; p < most; p += SCATTER_LANES) {
        const bool kp = p < k_pieces, vp = p < v_pieces;
        uint4 k[SCATTER_POINTS], v[SCATTER_POINTS];
#pragma unroll
        for (int u = 0; u < SCATTER_POINTS; ++u) {
            if (on[u] && kp) k[u] = __ldcs(keys + (size_t)h * k_head_pieces + (size_t)(i0 + u) * k_pieces + p);
            if (on[u] && vp) v[u] = __ldcs(values + (size_t)h * v_head_pieces + (size_t)(i0 + u) * v_pieces + p);
        }
#pragma unroll
        for (int u = 0; u < SCATTER_POINTS; ++u) {
            if (on[u] && kp) children[dst[u] * k_pieces + p] = k[u];
            if (on[u] && vp) __stcs(values_out + dst[u] * v_pieces + p, v[u]);
        }
    }
}

// parents (and their counts) into their final slots
template <typename T>
__global__ void scatter_parents_kernel(const T* __restrict__ cents1, const int32_t* __restrict__ fill1,
                                       const int32_t* __restrict__ slot2, int k1, int dim, T* __restrict__ parents,
                                       int32_t* __restrict__ child_counts, int cap_parents) {
    const int chunks = dim / 8;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int h = blockIdx.y;
    if (t >= (long long)k1 * chunks) return;
    const int c = (int)(t / chunks), ch = (int)(t % chunks);
    const int s = slot2 ? slot2[(size_t)h * k1 + c] : c;
    copy_chunk(parents + ((size_t)h * cap_parents + s) * dim, cents1 + ((size_t)h * k1 + c) * dim, ch);
    if (ch == 0) child_counts[(size_t)h * cap_parents + s] = fill1[(size_t)h * k1 + c];
}

template <typename T>
__global__ void scatter_gps_kernel(const T* __restrict__ cents2, const int32_t* __restrict__ fill2, int k2, int dim,
                                   T* __restrict__ gps, int32_t* __restrict__ gp_counts, int cap_gp) {
    const int chunks = dim / 8;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int h = blockIdx.y;
    if (t >= (long long)k2 * chunks) return;
    const int g = (int)(t / chunks), ch = (int)(t % chunks);
    copy_chunk(gps + ((size_t)h * cap_gp + g) * dim, cents2 + ((size_t)h * k2 + g) * dim, ch);
    if (ch == 0) gp_counts[(size_t)h * cap_gp + g] = fill2[(size_t)h * k2 + g];
}

// Child slots that hold no key: zero rows, token -1.  One warp per parent; the free slots of a parent
// are its last ones, so they are one run of whole 16-byte pieces per array.
constexpr int UNFILLED_THREADS = 256;
__global__ void __launch_bounds__(UNFILLED_THREADS)
clear_unfilled_kernel(const int32_t* __restrict__ child_counts, int cap_parents, int n_parents, int bf,
                      uint4* __restrict__ children, int row_pieces, uint4* __restrict__ values, int vrow_pieces,
                      int32_t* __restrict__ slot2token) {
    const int p = blockIdx.x * (UNFILLED_THREADS / 32) + (threadIdx.x >> 5), wl = threadIdx.x & 31;
    if (p >= n_parents) return;
    const size_t hp = (size_t)blockIdx.y * cap_parents + p;
    const int cnt = child_counts[hp];
    if (cnt >= bf) return;
    const size_t slot = hp * bf + cnt;
    const int n = bf - cnt;
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    for (int i = wl; i < n * row_pieces; i += 32) children[slot * row_pieces + i] = z;
    for (int i = wl; i < n * vrow_pieces; i += 32) values[slot * vrow_pieces + i] = z;
    if (slot2token)
        for (int i = wl; i < n; i += 32) slot2token[slot + i] = -1;
}

__global__ void set_used_kernel(int32_t* used, int n_heads, int used_p, int used_g, int n_keys) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= n_heads) return;
    used[h * 4 + 0] = used_p; used[h * 4 + 1] = used_g; used[h * 4 + 2] = n_keys; used[h * 4 + 3] = 0;
}

// ---------------------------------------------------------------------------
// Radii from the layout.
// ---------------------------------------------------------------------------
// One warp per ball.  Its four 8-lane groups take every fourth member, RADII_FLIGHT rows each in flight; a
// maximum does not depend on the order.  8 heads of 1,024 balls of 32 bf16 rows: 53.4 -> 16.4 us, the 32 balls
// of 32 balls above them: 42.1 -> 5.6 us (one group walked a ball with one row in flight before).
constexpr int RADII_THREADS = 256;
// max over the members c < cnt of  ||centre - row_c|| (+ extra[c]), the same in every lane of the warp
template <typename T, int NCH>
__device__ __forceinline__ float ball_radius(const T* rows, const float* extra, int cnt, const float (&px)[NCH][8], int dim) {
    constexpr int FLIGHT = NCH * (int)sizeof(T) > 4 ? 2 : 4;
    const int lane = threadIdx.x & (GROUP - 1), grp = (threadIdx.x >> 3) & 3;
    float r = 0.f;
    for (int c0 = 0; c0 < cnt; c0 += 4 * FLIGHT) {   // uniform over the warp
        RawChunk<T> raw[FLIGHT][NCH];
        float ex[FLIGHT];
#pragma unroll
        for (int u = 0; u < FLIGHT; ++u) {
            const int c = c0 + u * 4 + grp;
#pragma unroll
            for (int i = 0; i < NCH; ++i) {
                const int ch = lane + GROUP * i;
                raw[u][i] = (c < cnt && ch * 8 < dim) ? load_chunk_coherent<T>(rows + (size_t)c * dim, ch) : zero_chunk<T>();
            }
            ex[u] = extra && c < cnt ? extra[c] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < FLIGHT; ++u) {
            Acc2 acc{0.f, 0.f};
#pragma unroll
            for (int i = 0; i < NCH; ++i) {
                if ((lane + GROUP * i) * 8 < dim) {
                    float a[8], d[8];
                    to_float(raw[u][i], a);
#pragma unroll
                    for (int j = 0; j < 8; ++j) d[j] = __fsub_rn(px[i][j], a[j]);
                    chunk_fma(acc, d, d);
                }
            }
            const float dist = __fsqrt_rn(group_sum(__fadd_rn(acc.e, acc.o)));
            if (c0 + u * 4 + grp < cnt) r = fmaxf(r, extra ? __fadd_rn(dist, ex[u]) : dist);
        }
    }
    r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, 8));
    return fmaxf(r, __shfl_xor_sync(0xffffffffu, r, 16));
}

template <typename T, int NCH>
__global__ void __launch_bounds__(RADII_THREADS)
parent_radii_kernel(const hira_index_t ix) {
    const int lane = threadIdx.x & (GROUP - 1);
    const long long w = ((long long)blockIdx.x * RADII_THREADS + threadIdx.x) >> 5;  // (head, parent)
    if (w >= (long long)ix.n_heads * ix.cap_parents) return;
    const int h = (int)(w / ix.cap_parents), p = (int)(w % ix.cap_parents);
    const int bf = ix.bf, dim = ix.dim;
    bool valid;
    if (ix.depth == 3) {
        const int g = p / bf;
        valid = g < ix.used[h * 4 + 1] && (p - g * bf) < ix.gp_counts[(size_t)h * ix.cap_gp + g];
    } else {
        valid = p < ix.used[h * 4 + 0];
    }
    float r = 0.f, sq = 0.f;
    if (valid) {   // the whole warp
        int cnt = ix.child_counts[w];
        cnt = cnt > bf ? bf : cnt;
        float px[NCH][8];
        load_vec<T, NCH>(reinterpret_cast<const T*>(ix.parents) + (size_t)w * dim, px, lane, dim);
        sq = reg_sqnorm<NCH>(px);
        r = ball_radius<T, NCH>(reinterpret_cast<const T*>(ix.children) + (size_t)w * bf * dim, nullptr, cnt, px, dim);
    }
    if ((threadIdx.x & 31) == 0) {
        ix.parent_radii[w] = r;
        if (ix.parent_sqnorm) ix.parent_sqnorm[w] = sq;
    }
}

template <typename T, int NCH>
__global__ void __launch_bounds__(RADII_THREADS)
gp_radii_kernel(const hira_index_t ix) {
    const int lane = threadIdx.x & (GROUP - 1);
    const long long w = ((long long)blockIdx.x * RADII_THREADS + threadIdx.x) >> 5;  // (head, gp)
    if (w >= (long long)ix.n_heads * ix.cap_gp) return;
    const int h = (int)(w / ix.cap_gp), g = (int)(w % ix.cap_gp);
    const int bf = ix.bf, dim = ix.dim;
    float r = 0.f, sq = 0.f;
    if (g < ix.used[h * 4 + 1]) {   // the whole warp
        const size_t first = (size_t)h * ix.cap_parents + (size_t)g * bf;
        int cnt = ix.gp_counts[w];
        cnt = cnt > bf ? bf : cnt;
        float gx[NCH][8];
        load_vec<T, NCH>(reinterpret_cast<const T*>(ix.grand_parents) + (size_t)w * dim, gx, lane, dim);
        sq = reg_sqnorm<NCH>(gx);
        r = ball_radius<T, NCH>(reinterpret_cast<const T*>(ix.parents) + first * dim, ix.parent_radii + first, cnt, gx, dim);
    }
    if ((threadIdx.x & 31) == 0) {
        ix.gp_radii[w] = r;
        if (ix.gp_sqnorm) ix.gp_sqnorm[w] = sq;
    }
}

template <typename T>
static int launch_radii(const hira_index_t* ix, cudaStream_t s) {
    const long long blocks_p = ((long long)ix->n_heads * ix->cap_parents * 32 + RADII_THREADS - 1) / RADII_THREADS;
    HIRA_CHECK_ARG(blocks_p <= 0x7fffffffll, HIRA_ERR_SHAPE, "radii: %d heads x %d parents exceed the grid limit", ix->n_heads,
                   ix->cap_parents);
    if (ix->dim > 128) parent_radii_kernel<T, 4><<<(unsigned)blocks_p, RADII_THREADS, 0, s>>>(*ix);
    else parent_radii_kernel<T, 2><<<(unsigned)blocks_p, RADII_THREADS, 0, s>>>(*ix);
    HIRA_CHECK_LAUNCH("parent radii launch");
    if (ix->depth == 3) {
        const long long blocks_g = ((long long)ix->n_heads * ix->cap_gp * 32 + RADII_THREADS - 1) / RADII_THREADS;
        if (ix->dim > 128) gp_radii_kernel<T, 4><<<(unsigned)blocks_g, RADII_THREADS, 0, s>>>(*ix);
        else gp_radii_kernel<T, 2><<<(unsigned)blocks_g, RADII_THREADS, 0, s>>>(*ix);
        HIRA_CHECK_LAUNCH("grandparent radii launch");
    }
    return HIRA_OK;
}

// ---------------------------------------------------------------------------
// Export (slot order -> token order).
// ---------------------------------------------------------------------------
// Whole 16-byte pieces, keys and values of a slot together (before: two passes of 8 two-byte copies per
// thread; 8 x 65,664 bf16 keys and values: 391 -> 162 us).
// V: uint4, or 2-byte pieces for outputs that are not 16-byte aligned.
template <typename V>
__global__ void __launch_bounds__(256)
export_kv_kernel(const V* __restrict__ children, int k_pieces, const V* __restrict__ values, int v_pieces,
                 const int32_t* __restrict__ slot2token, long long head_rows, long long visit_rows, int token_base, int n_out,
                 V* __restrict__ out_k, V* __restrict__ out_v) {
    const int lane = threadIdx.x % 16;
    const long long s = (long long)blockIdx.x * 16 + threadIdx.x / 16;
    const int h = blockIdx.y;
    if (s >= visit_rows) return;
    const size_t at = (size_t)h * head_rows + s;
    const int tok = slot2token[at];
    if (tok < 0) return;
    const int o = tok - token_base;
    if (o < 0 || o >= n_out) return;
    const size_t to = (size_t)h * n_out + o;
    for (int p = lane; p < k_pieces; p += 16) out_k[to * k_pieces + p] = children[at * k_pieces + p];
    for (int p = lane; p < v_pieces; p += 16) out_v[to * v_pieces + p] = values[at * v_pieces + p];
}

// ---------------------------------------------------------------------------
// Workspace carving.
// ---------------------------------------------------------------------------
struct BuildWs {
    size_t total = 0;
    size_t cents1, cents2, csq, csq_masked, filled, a_idx, a_d2, keys, keys2, rank, sorted, start, count, pieces, merges, fill1,
        fill2, fbase, lbase, slot1, slot2;
};

static size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

static BuildWs carve(const hira_index_t* ix, int n_keys) {
    BuildWs w;
    const size_t H = ix->n_heads, n = n_keys, bf = ix->bf, D = ix->dim, es = elem_size(ix->dtype);
    const size_t k1 = (n + bf - 1) / bf, k2 = (k1 + bf - 1) / bf;
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off += align_up(bytes); return o; };
    w.cents1 = take(H * k1 * D * es);
    w.cents2 = take(H * k2 * D * es);
    w.csq = take(H * k1 * 4);
    w.csq_masked = take(H * k1 * 4);
    w.filled = take(H * k1 * 4);
    w.a_idx = take(H * n * 4);
    w.a_d2 = take(H * n * 4);
    w.keys = take(H * n * 8);
    w.keys2 = take(H * n * 8);
    w.rank = take(H * n * 4);
    w.sorted = take(H * n * 4);
    w.start = take(H * k1 * 4);
    w.count = take((H * k1 + MEMBER_LISTS) * 4);
    w.pieces = take(pieces_bound(H * n) * 8);
    w.merges = take(merges_bound(H * n) * 8);
    w.fill1 = take(H * k1 * 4);
    w.fill2 = take(H * k2 * 4);
    w.fbase = take(H * (k1 + 1) * 4);
    w.lbase = take(H * (k1 + 1) * 4);
    w.slot1 = take(H * n * 4);
    w.slot2 = take(H * k1 * 4);
    w.total = off;
    return w;
}

// One level: points -> K centres (in `cents`), per-point slot (centre*bf+rank)
// and per-centre filled count.
template <typename T>
static int build_level(int dtype, const T* points, long long p_head_stride, int n_heads, int n, int k, int bf,
                       int dim, const int32_t* cent_idx, int n_iters, int balance_rounds, int use_tc, T* cents, char* base,
                       const BuildWs& w, int32_t* slot, int32_t* fill, int32_t* status, cudaStream_t s) {
    const long long total = (long long)n_heads * n;
    const long long n_seg = (long long)n_heads * k;
    float* csq = reinterpret_cast<float*>(base + w.csq);
    int32_t* a_idx = reinterpret_cast<int32_t*>(base + w.a_idx);
    float* a_d2 = reinterpret_cast<float*>(base + w.a_d2);
    uint64_t* keys = reinterpret_cast<uint64_t*>(base + w.keys);
    uint64_t* keys2 = reinterpret_cast<uint64_t*>(base + w.keys2);
    int32_t* rank = reinterpret_cast<int32_t*>(base + w.rank);
    uint32_t* sorted = reinterpret_cast<uint32_t*>(base + w.sorted);
    int32_t* start = reinterpret_cast<int32_t*>(base + w.start);
    int32_t* count = reinterpret_cast<int32_t*>(base + w.count);
    int32_t* fbase = reinterpret_cast<int32_t*>(base + w.fbase);
    int32_t* lbase = reinterpret_cast<int32_t*>(base + w.lbase);
    const int chunks = dim / 8;
    {
        dim3 grid((unsigned)(((long long)k * chunks + 255) / 256), (unsigned)n_heads);
        gather_centres_kernel<T><<<grid, 256, 0, s>>>(points, p_head_stride, n, cent_idx, k, dim, cents);
        HIRA_CHECK_LAUNCH("gather centres launch");
    }
    const int blocks = (int)((total + 255) / 256);
    const MemberLists lists{reinterpret_cast<uint64_t*>(base + w.pieces), reinterpret_cast<uint64_t*>(base + w.merges), count + n_seg};
    const size_t most = pieces_bound((size_t)total);
    const int piece_ctas = most < (size_t)SORT_PIECE_CTAS ? (int)most : SORT_PIECE_CTAS;
    // counts, ranges and ranks of the points' latest assignment; `placed`: the slots of the points to leave out
    auto sort_members = [&](const int32_t* placed) -> int {
        if (placed) cudaMemsetAsync(count, 0, ((size_t)n_seg + MEMBER_LISTS) * 4, s);   // else cleared with the norms of the centres
        count_members_kernel<<<blocks, 256, 0, s>>>(a_idx, a_d2, n, k, total, placed, count, rank, status);
        member_starts_kernel<<<n_heads, 1024, 0, s>>>(count, n, k, start, lists);
        drop_members_kernel<<<blocks, 256, 0, s>>>(a_idx, a_d2, n, k, total, start, rank, keys);
        const long long sblocks = piece_ctas + (n_seg + SORT_RANGES - 1) / SORT_RANGES;
        sort_members_kernel<<<(unsigned)sblocks, SORT_THREADS, 0, s>>>(count, start, n, k, n_seg, piece_ctas, lists, keys, sorted, rank);
        HIRA_CHECK_LAUNCH("member sort launch");
        uint64_t *from = keys, *to = keys2;
        for (long long len = SORT_CTA; len < n; len *= MERGE_WAYS) {   // what a range of all the points would take
            const cudaError_t e = launch_chained(merge_members_kernel, dim3(4 * SM_COUNT), dim3(SORT_THREADS), 0, s, (const int32_t*)count,
                                                 (const int32_t*)start, n, k, (int)len, lists, (const uint64_t*)from, to, sorted, rank);
            if (e != cudaSuccess) { set_error("member merge launch: %s", cudaGetErrorString(e)); return HIRA_ERR_CUDA; }
            uint64_t* t = from; from = to; to = t;
        }
        return HIRA_OK;
    };
    const int iters = n_iters < 1 ? 1 : n_iters;
    for (int it = 0; it < iters; ++it) {
        int rc = run_assign(dtype, points, p_head_stride, cents, csq, n_heads, n, k, dim, use_tc, a_idx, a_d2, s, false, count);
        if (rc != HIRA_OK) return rc;
        rc = sort_members(nullptr);
        if (rc != HIRA_OK) return rc;
        if (it + 1 < iters) {
            const int per_warp = 32 * MeansElem<T>::N;
            const int slabs = (dim + per_warp - 1) / per_warp;
            const long long mblocks = (n_seg * slabs + MEANS_WARPS - 1) / MEANS_WARPS;
            auto means = [&](auto kern, int stages) -> int {
                const int smem = MEANS_WARPS * stages * MEANS_BATCH * 128;
                const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
                if (e != cudaSuccess) { set_error("means: cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return HIRA_ERR_CUDA; }
                kern<<<(unsigned)mblocks, MEANS_WARPS * 32, smem, s>>>(points, p_head_stride, n, sorted, start, count, k, dim, slabs,
                                                                       n_seg, cents);
                return HIRA_OK;
            };
            // crowded centres: a deep ring for their chains; many small ones: twice the warps per SM instead
            rc = n >= 48ll * k ? means(means_kernel<T, 4>, 4) : means(means_kernel<T, 2>, 2);
            if (rc != HIRA_OK) return rc;
            HIRA_CHECK_LAUNCH("means launch");
        }
    }
    // ---- capacity-aware rounds: points that did not fit under their nearest centre choose again
    // among the centres that still have room, closest first, `balance_rounds` times; what is left
    // after that (and everything beyond the bf closest when balance_rounds == 0, the reference's
    // rule, indexer/cuda.py:252-334) goes to the free slots in (centre, distance) order.
    int32_t* filled = reinterpret_cast<int32_t*>(base + w.filled);
    float* csq_masked = reinterpret_cast<float*>(base + w.csq_masked);
    const int seg_blocks = (int)((n_seg + 255) / 256);
    if (balance_rounds > 0) {
        cudaMemsetAsync(filled, 0, (size_t)n_seg * 4, s);
        cudaMemsetAsync(slot, 0xff, (size_t)total * 4, s);
    }
    const int32_t* taken = balance_rounds > 0 ? filled : nullptr;   // NULL: every centre starts empty
    for (int r = 0; r < balance_rounds; ++r) {
        accept_kernel<<<blocks, 256, 0, s>>>(a_idx, rank, filled, n, k, bf, total, slot);
        accept_counts_kernel<<<seg_blocks, 256, 0, s>>>(count, bf, n_seg, filled);
        mask_full_centres_kernel<<<seg_blocks, 256, 0, s>>>(csq, filled, bf, n_seg, csq_masked);
        HIRA_CHECK_LAUNCH("balanced round launch");
        int rc = run_assign(dtype, points, p_head_stride, cents, csq_masked, n_heads, n, k, dim, use_tc, a_idx, a_d2, s, true);
        if (rc != HIRA_OK) return rc;
        rc = sort_members(slot);
        if (rc != HIRA_OK) return rc;
    }
    capacity_scan_kernel<<<n_heads, 1024, 0, s>>>(count, taken, k, bf, fbase, lbase, fill);
    HIRA_CHECK_LAUNCH("capacity scan launch");
    placement_kernel<<<blocks, 256, 0, s>>>(a_idx, rank, count, taken, fbase, lbase, n, k, bf, total, balance_rounds > 0, slot);
    HIRA_CHECK_LAUNCH("placement launch");
    return HIRA_OK;
}

template <typename T>
static int build_impl(const hira_index_t* ix, const void* keys_v, const void* values, int n_keys,
                      long long k_head_stride, long long v_head_stride, int token_base, const int32_t* cent_idx1,
                      const int32_t* cent_idx2, int n_iters, int balance_rounds, int use_tc, char* base, const BuildWs& w,
                      int32_t* status, cudaStream_t s) {
    const T* keys = reinterpret_cast<const T*>(keys_v);
    const int H = ix->n_heads, bf = ix->bf, dim = ix->dim;
    const int k1 = (n_keys + bf - 1) / bf;
    const int k2 = (k1 + bf - 1) / bf;
    const size_t es = elem_size(ix->dtype);
    const size_t capP = ix->cap_parents, capC = capP * bf;
    // ---- clear the index -----------------------------------------------------
    // Everything, or -- when the host vouches through active_parents that no slot beyond that bound
    // was ever used -- the slots up to the larger of that bound and what this build fills.  The child
    // rows, the bulk of the index, are not cleared here: the scatter below writes the filled ones and
    // clear_unfilled_kernel the rest, each once.
    size_t clearP = capP;
    if (ix->active_parents > 0) {
        const size_t fills = ix->depth == 3 ? (size_t)k2 * bf : (size_t)k1;
        clearP = (size_t)ix->active_parents > fills ? (size_t)ix->active_parents : fills;
        if (clearP > capP) clearP = capP;
    }
    {
        const size_t clearG = ix->depth == 3 ? (clearP + bf - 1) / bf : 0;
        auto clear = [&](void* ptr, int value, size_t row_bytes, size_t rows_cap, size_t rows_clear) {
            if (ptr) cudaMemset2DAsync(ptr, rows_cap * row_bytes, value, rows_clear * row_bytes, (size_t)H, s);
        };
        clear(ix->parents, 0, dim * es, capP, clearP);
        clear(ix->child_counts, 0, 4, capP, clearP);
        if (ix->depth == 3) {
            clear(ix->grand_parents, 0, dim * es, ix->cap_gp, clearG);
            clear(ix->gp_counts, 0, 4, ix->cap_gp, clearG);
        }
        if (n_keys == 0) {   // otherwise written by the radii kernels
            clear(ix->parent_radii, 0, 4, capP, clearP);
            clear(ix->parent_sqnorm, 0, 4, capP, clearP);
            if (ix->depth == 3) {
                clear(ix->gp_radii, 0, 4, ix->cap_gp, clearG);
                clear(ix->gp_sqnorm, 0, 4, ix->cap_gp, clearG);
            }
        }
    }
    HIRA_CHECK_LAUNCH("index clear");
    auto clear_unfilled = [&]() -> int {
        const int warps = UNFILLED_THREADS / 32;
        dim3 grid((unsigned)((clearP + warps - 1) / warps), (unsigned)H);
        clear_unfilled_kernel<<<grid, UNFILLED_THREADS, 0, s>>>(
            ix->child_counts, (int)capP, (int)clearP, bf, reinterpret_cast<uint4*>(ix->children), (int)(dim * es / 16),
            reinterpret_cast<uint4*>(ix->values), ix->values ? (int)(ix->vdim * elem_size(ix->vdtype) / 16) : 0,
            ix->slot2token);
        HIRA_CHECK_LAUNCH("clear unfilled launch");
        return HIRA_OK;
    };
    if (n_keys == 0) {
        set_used_kernel<<<(H + 127) / 128, 128, 0, s>>>(ix->used, H, 0, 0, 0);
        HIRA_CHECK_LAUNCH("set used launch");
        return clear_unfilled();
    }
    T* cents1 = reinterpret_cast<T*>(base + w.cents1);
    T* cents2 = reinterpret_cast<T*>(base + w.cents2);
    int32_t* slot1 = reinterpret_cast<int32_t*>(base + w.slot1);
    int32_t* slot2 = reinterpret_cast<int32_t*>(base + w.slot2);
    int32_t* fill1 = reinterpret_cast<int32_t*>(base + w.fill1);
    int32_t* fill2 = reinterpret_cast<int32_t*>(base + w.fill2);
    int rc = build_level<T>(ix->dtype, keys, k_head_stride, H, n_keys, k1, bf, dim, cent_idx1, n_iters, balance_rounds, use_tc,
                            cents1, base, w, slot1, fill1, status, s);
    if (rc != HIRA_OK) return rc;
    const int32_t* slot2_used = nullptr;
    if (ix->depth == 3) {
        rc = build_level<T>(ix->dtype, cents1, (long long)k1 * dim, H, k1, k2, bf, dim, cent_idx2, n_iters, balance_rounds, use_tc,
                            cents2, base, w, slot2, fill2, status, s);
        if (rc != HIRA_OK) return rc;
        slot2_used = slot2;
        const int chunks = dim / 8;
        dim3 grid((unsigned)(((long long)k2 * chunks + 255) / 256), (unsigned)H);
        scatter_gps_kernel<T><<<grid, 256, 0, s>>>(cents2, fill2, k2, dim, reinterpret_cast<T*>(ix->grand_parents),
                                                   ix->gp_counts, ix->cap_gp);
        HIRA_CHECK_LAUNCH("scatter gps launch");
    }
    {
        const int chunks = dim / 8;
        dim3 grid((unsigned)(((long long)k1 * chunks + 255) / 256), (unsigned)H);
        scatter_parents_kernel<T><<<grid, 256, 0, s>>>(cents1, fill1, slot2_used, k1, dim,
                                                       reinterpret_cast<T*>(ix->parents), ix->child_counts,
                                                       ix->cap_parents);
        HIRA_CHECK_LAUNCH("scatter parents launch");
    }
    {
        const int per_block = SCATTER_THREADS / SCATTER_LANES * SCATTER_POINTS;
        dim3 grid((unsigned)((n_keys + per_block - 1) / per_block), (unsigned)H);
        const size_t ves = ix->values ? elem_size(ix->vdtype) : 0;
        scatter_kv_kernel<<<grid, SCATTER_THREADS, 0, s>>>(
            reinterpret_cast<const uint4*>(keys), k_head_stride * (long long)es / 16, (int)(dim * es / 16),
            reinterpret_cast<const uint4*>(values), v_head_stride * (long long)ves / 16, ix->values ? (int)(ix->vdim * ves / 16) : 0,
            n_keys, slot1, slot2_used, k1, bf, reinterpret_cast<uint4*>(ix->children), reinterpret_cast<uint4*>(ix->values),
            (long long)capC, ix->slot2token, token_base);
        HIRA_CHECK_LAUNCH("scatter keys and values launch");
    }
    rc = clear_unfilled();
    if (rc != HIRA_OK) return rc;
    set_used_kernel<<<(H + 127) / 128, 128, 0, s>>>(ix->used, H, ix->depth == 3 ? k2 * bf : k1,
                                                     ix->depth == 3 ? k2 : 0, n_keys);
    HIRA_CHECK_LAUNCH("set used launch");
    rc = launch_radii<T>(ix, s);
    if (rc != HIRA_OK) return rc;
    // the int8 side copy of the children, when the index carries one: over the slots this build filled
    return q8_refresh(ix, s, ix->depth == 3 ? (long long)k2 * bf : (long long)k1);
}

// ---------------------------------------------------------------------------
// A larger copy of an index: every head's part of every array copied and the room behind it filled, all arrays
// in one launch (a copy and a fill per array before, some forty launches of a few microseconds).
// ---------------------------------------------------------------------------
struct GrowItem { const char* src; char* dst; long long src_bytes, dst_bytes; uint32_t fill; };   // bytes per head
constexpr int GROW_ITEMS = 16;
struct GrowItems { GrowItem it[GROW_ITEMS]; };
__global__ void __launch_bounds__(256)
grow_kernel(const GrowItems items) {
    const GrowItem g = items.it[blockIdx.z];
    const char* src = g.src + (size_t)blockIdx.y * g.src_bytes;
    char* dst = g.dst + (size_t)blockIdx.y * g.dst_bytes;
    const long long first = (long long)blockIdx.x * 256 + threadIdx.x, step = (long long)gridDim.x * 256;
    if ((((uintptr_t)src | (uintptr_t)dst | (uintptr_t)g.src_bytes | (uintptr_t)g.dst_bytes) & 15) == 0) {
        const uint4 f = make_uint4(g.fill, g.fill, g.fill, g.fill);
        for (long long i = first; i < g.dst_bytes / 16; i += step)
            reinterpret_cast<uint4*>(dst)[i] = i < g.src_bytes / 16 ? reinterpret_cast<const uint4*>(src)[i] : f;
    } else {   // the arrays of single words, where a head's part may start at any of them
        for (long long i = first; i < g.dst_bytes / 4; i += step)
            reinterpret_cast<uint32_t*>(dst)[i] = i < g.src_bytes / 4 ? reinterpret_cast<const uint32_t*>(src)[i] : g.fill;
    }
}

// point drawn by u in [0, 1) out of stride c of k equal strides of n points
__global__ void stratified_kernel(const float* __restrict__ u, int n, int k, long long total, int32_t* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const long long c = i % k, lo = c * n / k, width = (c + 1) * n / k - lo;
    long long j = (long long)__fmul_rn(u[i], (float)width);
    const long long last = width > 1 ? width - 1 : 0;
    out[i] = (int32_t)(lo + (j < last ? j : last));
}

}  // namespace hira

using namespace hira;

extern "C" int hira_grow(const hira_index_t* from, const hira_index_t* to, void* stream) {
    int rc = validate_index(from, false);
    if (rc == HIRA_OK) rc = validate_index(to, false);
    if (rc != HIRA_OK) return rc;
    HIRA_CHECK_ARG(from->dtype == to->dtype && from->vdtype == to->vdtype && from->depth == to->depth && from->bf == to->bf &&
                   from->dim == to->dim && from->vdim == to->vdim && from->n_heads == to->n_heads, HIRA_ERR_SHAPE,
                   "hira_grow: the two indexes differ in more than their capacity");
    HIRA_CHECK_ARG(from->cap_parents <= to->cap_parents, HIRA_ERR_CAPACITY, "hira_grow: capacity %d does not fit into %d",
                   from->cap_parents, to->cap_parents);
    HIRA_CHECK_ARG(to->n_heads <= 65535, HIRA_ERR_SHAPE, "hira_grow: %d heads exceed the grid limit", to->n_heads);
    GrowItems items;
    int n = 0;
    auto add = [&](const void* src, void* dst, long long row, long long rows_from, long long rows_to, uint32_t fill) {
        if (src && dst) items.it[n++] = GrowItem{(const char*)src, (char*)dst, row * rows_from, row * rows_to, fill};
    };
    const long long es = (long long)elem_size(to->dtype), ves = (long long)elem_size(to->vdtype), p0 = from->cap_parents,
                    p1 = to->cap_parents, c0 = p0 * to->bf, c1 = p1 * to->bf, g0 = from->cap_gp, g1 = to->cap_gp;
    add(from->children, to->children, to->dim * es, c0, c1, 0);
    add(from->values, to->values, to->vdim * ves, c0, c1, 0);
    add(from->slot2token, to->slot2token, 4, c0, c1, 0xffffffffu);
    add(from->parents, to->parents, to->dim * es, p0, p1, 0);
    add(from->parent_radii, to->parent_radii, 4, p0, p1, 0);
    add(from->parent_sqnorm, to->parent_sqnorm, 4, p0, p1, 0);
    add(from->child_counts, to->child_counts, 4, p0, p1, 0);
    if (to->depth == 3) {
        add(from->grand_parents, to->grand_parents, to->dim * es, g0, g1, 0);
        add(from->gp_radii, to->gp_radii, 4, g0, g1, 0);
        add(from->gp_sqnorm, to->gp_sqnorm, 4, g0, g1, 0);
        add(from->gp_counts, to->gp_counts, 4, g0, g1, 0);
    }
    add(from->used, to->used, 4, 4, 4, 0);
    add(from->children_q8, to->children_q8, 128, c0, c1, 0);
    add(from->children_q8_meta, to->children_q8_meta, 4, c0, c1, 0);
    add(from->q8_chan_scale, to->q8_chan_scale, 4, HIRA_Q8_CHAN, HIRA_Q8_CHAN, 0);
    grow_kernel<<<dim3(64, (unsigned)to->n_heads, (unsigned)n), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(items);
    HIRA_CHECK_LAUNCH("hira_grow launch");
    return HIRA_OK;
}

extern "C" int hira_stratified(const float* u, int32_t n_heads, int32_t n, int32_t k, int32_t* out, void* stream) {
    HIRA_CHECK_ARG(u && out, HIRA_ERR_ARG, "hira_stratified: NULL argument");
    HIRA_CHECK_ARG(n_heads >= 1 && n >= 1 && k >= 1, HIRA_ERR_SHAPE, "hira_stratified: n_heads=%d n=%d k=%d", n_heads, n, k);
    const long long total = (long long)n_heads * k;
    stratified_kernel<<<(unsigned)((total + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(u, n, k, total, out);
    HIRA_CHECK_LAUNCH("hira_stratified launch");
    return HIRA_OK;
}

extern "C" size_t hira_build_workspace_bytes(const hira_index_t* ix, int32_t n_keys) {
    if (validate_index(ix, false) != HIRA_OK || n_keys < 0) return 0;
    return carve(ix, n_keys > 0 ? n_keys : 1).total;
}

extern "C" int hira_build(const hira_index_t* ix, const void* keys, const void* values, int32_t n_keys,
                          int64_t k_head_stride, int64_t v_head_stride, int32_t token_base,
                          const int32_t* cent_idx1, const int32_t* cent_idx2, int32_t n_iters,
                          int32_t balance_rounds, int32_t use_tensor_cores, int32_t* status, void* workspace,
                          size_t workspace_bytes, void* stream) {
    int rc = validate_index(ix, false);
    if (rc != HIRA_OK) return rc;
    HIRA_CHECK_ARG(n_keys >= 0, HIRA_ERR_SHAPE, "hira_build: n_keys=%d", n_keys);
    HIRA_CHECK_ARG(balance_rounds >= 0 && balance_rounds <= 64, HIRA_ERR_ARG, "hira_build: balance_rounds=%d", balance_rounds);
    HIRA_CHECK_ARG(n_keys == 0 || keys, HIRA_ERR_ARG, "hira_build: keys is NULL");
    HIRA_CHECK_ARG((ix->values == nullptr) == (values == nullptr) || n_keys == 0, HIRA_ERR_ARG,
                   "hira_build: values must be given iff the index stores values");
    const long long bf = ix->bf;
    const long long k1 = (n_keys + bf - 1) / bf, k2 = (k1 + bf - 1) / bf;
    if (ix->depth == 3)
        HIRA_CHECK_ARG(k2 <= ix->cap_gp, HIRA_ERR_CAPACITY, "hira_build: %d keys need %lld grandparents, capacity %d",
                       n_keys, k2, ix->cap_gp);
    else
        HIRA_CHECK_ARG(k1 <= ix->cap_parents, HIRA_ERR_CAPACITY, "hira_build: %d keys need %lld parents, capacity %d",
                       n_keys, k1, ix->cap_parents);
    const BuildWs w = carve(ix, n_keys > 0 ? n_keys : 1);
    HIRA_CHECK_ARG(n_keys == 0 || (workspace && workspace_bytes >= w.total), HIRA_ERR_CAPACITY,
                   "hira_build: workspace of %zu bytes given, %zu needed", workspace_bytes, w.total);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    char* base = reinterpret_cast<char*>(workspace);
    if (ix->dtype == HIRA_BF16)
        return build_impl<__nv_bfloat16>(ix, keys, values, n_keys, k_head_stride, v_head_stride, token_base, cent_idx1,
                                         cent_idx2, n_iters, balance_rounds, use_tensor_cores, base, w, status, s);
    return build_impl<float>(ix, keys, values, n_keys, k_head_stride, v_head_stride, token_base, cent_idx1, cent_idx2,
                             n_iters, balance_rounds, use_tensor_cores, base, w, status, s);
}

extern "C" int hira_recompute_radii(const hira_index_t* ix, void* stream) {
    int rc = validate_index(ix, false);
    if (rc != HIRA_OK) return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    return ix->dtype == HIRA_BF16 ? launch_radii<__nv_bfloat16>(ix, s) : launch_radii<float>(ix, s);
}

extern "C" int hira_export(const hira_index_t* ix, int32_t token_base, int32_t n_out, void* out_k, void* out_v,
                           void* stream) {
    int rc = validate_index(ix, false);
    if (rc != HIRA_OK) return rc;
    HIRA_CHECK_ARG(ix->slot2token, HIRA_ERR_ARG, "hira_export: the index has no slot2token map");
    HIRA_CHECK_ARG(out_k && n_out >= 1, HIRA_ERR_ARG, "hira_export: out_k is NULL or n_out < 1");
    HIRA_CHECK_ARG(!out_v || ix->values, HIRA_ERR_ARG, "hira_export: out_v given but the index stores no values");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const long long rows = (long long)ix->cap_parents * ix->bf;
    // only the slots that can hold keys are visited (the host's bound, hira_index_t::active_parents)
    const long long visit = (ix->active_parents > 0 ? (long long)ix->active_parents : (long long)ix->cap_parents) * ix->bf;
    dim3 grid((unsigned)((visit + 15) / 16), (unsigned)ix->n_heads);
    auto launch = [&](auto piece) {
        using V = decltype(piece);
        export_kv_kernel<V><<<grid, 256, 0, s>>>(
            reinterpret_cast<const V*>(ix->children), (int)(ix->dim * elem_size(ix->dtype) / sizeof(V)),
            reinterpret_cast<const V*>(ix->values), out_v ? (int)(ix->vdim * elem_size(ix->vdtype) / sizeof(V)) : 0,
            ix->slot2token, rows, visit, token_base, n_out, reinterpret_cast<V*>(out_k), reinterpret_cast<V*>(out_v));
    };
    if ((((uintptr_t)out_k | (uintptr_t)out_v) & 15) == 0) launch(uint4{});
    else launch((uint16_t)0);
    HIRA_CHECK_LAUNCH("export launch");
    return HIRA_OK;
}

extern "C" int hira_assign(const void* points, const void* cents, int32_t dtype, int32_t n_heads, int32_t n,
                           int32_t k, int32_t dim, int32_t use_tensor_cores, float* csq_scratch, int32_t* out_idx,
                           float* out_dist2, void* stream) {
    HIRA_CHECK_ARG(points && cents && csq_scratch && out_idx && out_dist2, HIRA_ERR_ARG, "hira_assign: NULL argument");
    HIRA_CHECK_ARG(dtype == HIRA_F32 || dtype == HIRA_BF16, HIRA_ERR_DTYPE, "hira_assign: dtype %d", dtype);
    HIRA_CHECK_ARG(n_heads >= 1 && n >= 1 && k >= 1, HIRA_ERR_SHAPE, "hira_assign: n_heads=%d n=%d k=%d", n_heads, n, k);
    HIRA_CHECK_ARG(dim >= 8 && dim <= 256 && dim % 8 == 0, HIRA_ERR_SHAPE, "hira_assign: dim=%d", dim);
    return run_assign(dtype, points, (long long)n * dim, cents, csq_scratch, n_heads, n, k, dim, use_tensor_cores,
                      out_idx, out_dist2, reinterpret_cast<cudaStream_t>(stream));
}
