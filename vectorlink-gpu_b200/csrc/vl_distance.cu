// Gathered fp32 distance kernels: the operator-level replacements of the reference's
// cuda_distances_kernel (vectorlink_gpu/kernels.py:130-171) and
// cuda_search_from_seeds_kernel (kernels.py:204-257).
//
// The reference launches one CTA per (row, neighbour) pair and re-reads the query row for
// every pair.  Here one warp owns a (query row, run of candidates) task: the query row
// is loaded once into registers, and the warp walks its candidates 32/LPR at a time, each
// candidate row fetched by LPR lanes with 128-bit loads (a contiguous LPR*16-byte span per
// load instruction), several steps in flight.  The kernels are bound by the gather of
// candidate rows: 4*dim + 12 bytes per evaluated pair, from HBM or, where rows repeat, from L2.
// 1,000,000 rows of 128 dimensions, 32 scattered neighbours each (a load): 2.69 ms with one step of four lanes per
// row in flight, 2.42 ms with four steps of eight lanes (17.2 GB; copy bandwidth alone: 2.6 ms, some of
// the rows repeat in L2).
#include "vl_common.cuh"
#include "vlgpu.h"

namespace {

constexpr int kWarpsPerBlock = 4;

struct GatherArgs {
    const float* vectors;      // [n, dim]
    int64_t n;
    int dim;
    const float* queries;      // [rows, dim]
    int64_t rows;
    int segs, seg_len;         // candidates of a row: segs segments of seg_len
    int span, spans;           // a segment is walked in `spans` runs of at most `span` candidates
    // where a candidate's id comes from, one of:
    const int32_t* ids;        //   [rows, segs*seg_len]
    const int32_t* visit;      //   [rows, segs]: ids of visited nodes, the candidates are their rows of `graph` [n, seg_len]
    const int32_t* graph;
    const int32_t* offsets;    //   [seg_len]: (first_row + row + offset) mod modulo, in 32 bits (utils.py:26-32)
    int32_t first_row, modulo;
    int32_t* idx_out;          // [rows, segs*seg_len] or null
    float* dist_out;           // [rows, segs*seg_len]
    int* status;
};

// JU > 0: exact-fit rows (dim == 4*LPR*JU, aligned); JU == 0: any dimension.
template <int LPR, int JP, int JU, int METRIC, bool ALIGNED>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
gather_distance_kernel(const GatherArgs a)
{
    constexpr int G = 32 / LPR;                      // candidates per warp step
    constexpr int JQ = JU > 0 ? JU : JP;
    constexpr int U = JU > 0 ? (JU <= 4 ? 4 : 2) : (JP <= 4 ? 2 : 1);   // steps in flight
    const int lane = threadIdx.x & 31;
    const int g = lane / LPR, lg = lane % LPR;
    const int64_t per_row = (int64_t)a.segs * a.spans;
    const int64_t total = a.rows * per_row;
    const int64_t warp0 = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    const int64_t nwarps = (int64_t)gridDim.x * kWarpsPerBlock;
    for (int64_t task = warp0; task < total; task += nwarps) {
        const int64_t r = task / per_row;
        const int part = (int)(task - r * per_row);
        const int s = part / a.spans;
        const int m_lo = (part - s * a.spans) * a.span;
        const int m_hi = m_lo + a.span < a.seg_len ? m_lo + a.span : a.seg_len;
        const float* q = a.queries + r * (int64_t)a.dim;
        float4 qr[JQ];
        if constexpr (JU > 0) vl_load_exact<LPR, JU>(q, lg, qr);
        else vl_load_query<LPR, JP, ALIGNED>(q, a.dim, lg, qr);
        int32_t node = 0;
        if (a.visit) {
            node = __ldg(a.visit + r * a.segs + s);
            if (node != VL_MAXINT && (node < 0 || (int64_t)node >= a.n)) {
                if (lane == 0) atomicOr(a.status, VL_STATUS_BAD_ID);
                node = VL_MAXINT;
            }
        }
        const int64_t out0 = r * (int64_t)a.segs * a.seg_len + (int64_t)s * a.seg_len;
        for (int m0 = m_lo; m0 < m_hi; m0 += U * G) {
            int32_t id[U];
            bool live[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int m = m0 + u * G + g;
                id[u] = VL_MAXINT;
                if (m < m_hi) {
                    if (a.offsets) {
                        const int32_t x = (int32_t)((uint32_t)a.first_row + (uint32_t)r + (uint32_t)__ldg(a.offsets + m)) % a.modulo;
                        id[u] = x < 0 ? x + a.modulo : x;
                    } else if (a.visit) id[u] = (node == VL_MAXINT) ? VL_MAXINT : __ldg(a.graph + (int64_t)node * a.seg_len + m);
                    else id[u] = __ldg(a.ids + out0 + m);
                }
                live[u] = (id[u] != VL_MAXINT);
                if (live[u] && (id[u] < 0 || (int64_t)id[u] >= a.n)) {
                    live[u] = false;
                    if (lg == 0) atomicOr(a.status, VL_STATUS_BAD_ID);
                }
            }
            float d[U];
            float4 xr[U][JQ];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float* row = a.vectors + (int64_t)(live[u] ? id[u] : 0) * a.dim;
                if constexpr (JU > 0) vl_load_exact<LPR, JU>(row, lg, xr[u]);
                else vl_load_row<LPR, JP, ALIGNED>(row, a.dim, lg, live[u], xr[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if constexpr (JU > 0) d[u] = vl_exact_distance<LPR, JP, JU, METRIC>(xr[u], qr);
                else {
                    const float* row = a.vectors + (int64_t)(live[u] ? id[u] : 0) * a.dim;
                    d[u] = vl_row_distance<LPR, JP, METRIC, ALIGNED>(xr[u], qr, row, q, a.dim, lg, live[u]);
                }
            }
            if (lg == 0) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int m = m0 + u * G + g;
                    if (m < m_hi) {
                        a.dist_out[out0 + m] = live[u] ? d[u] : VL_MAXFLOAT;
                        if (a.idx_out) a.idx_out[out0 + m] = live[u] ? id[u] : VL_MAXINT;
                    }
                }
            }
        }
    }
}

template <int LPR, int JP, int JU, int METRIC, bool ALIGNED>
int gather_launch(GatherArgs a, cudaStream_t stream)
{
    // a few thousand warps fill the device: with fewer (row, segment) pairs, a segment is divided among
    // warps, in multiples of the 32 candidates that keep their loads in flight
    const int64_t pairs = a.rows * a.segs, sms = vl_sm_count();
    a.span = a.seg_len;
    if (pairs < sms * 32) {
        const int64_t want = (sms * 32 + pairs - 1) / pairs;
        const int64_t span = (a.seg_len + want - 1) / want;
        a.span = (int)((span + 31) / 32 * 32);
    }
    a.spans = (a.seg_len + a.span - 1) / a.span;
    int64_t blocks = (pairs * a.spans + kWarpsPerBlock - 1) / kWarpsPerBlock;
    const int64_t cap = sms * 64;  // grid-stride beyond that
    if (blocks > cap) blocks = cap;
    gather_distance_kernel<LPR, JP, JU, METRIC, ALIGNED><<<(unsigned)blocks, kWarpsPerBlock * 32, 0, stream>>>(a);
    VL_CHECK_LAUNCH("gather_distance_kernel");
    return 0;
}

template <int METRIC>
int launch_gather(const GatherArgs& a, cudaStream_t stream)
{
    const bool aligned = (a.dim % 4 == 0) && (((uintptr_t)a.vectors | (uintptr_t)a.queries) % 16 == 0);
    if (aligned && a.n > 0) {      // the exact fit loads row 0 for a candidate that is none, so there has to be one
#define VL_EXACT(L, J, U) if (a.dim == 4 * L * U) return gather_launch<L, J, U, METRIC, true>(a, stream);
        VL_EXACT(4, 4, 4)     // dim 64
        VL_EXACT(8, 4, 3)     // dim 96
        VL_EXACT(8, 4, 4)     // dim 128
        VL_EXACT(16, 4, 4)    // dim 256
        VL_EXACT(32, 4, 3)    // dim 384
        VL_EXACT(32, 4, 4)    // dim 512
        VL_EXACT(32, 8, 6)    // dim 768
        VL_EXACT(32, 8, 8)    // dim 1024
#undef VL_EXACT
    }
    VlShape shape = vl_pick_shape(a.dim);
    VL_DISPATCH_SHAPE(shape, {
        return aligned ? gather_launch<LPR, JP, 0, METRIC, true>(a, stream) : gather_launch<LPR, JP, 0, METRIC, false>(a, stream);
    });
}

}  // namespace

extern "C" int vl_calculate_distances(const float* vectors, int64_t n, int dim, const float* queries,
                                      int64_t rows, const int32_t* ids, int w, float* dist_out, int metric,
                                      int* status, void* stream)
{
    VL_CHECK_ARG(dim > 0 && w >= 0 && rows >= 0 && n >= 0, "vl_calculate_distances: bad size");
    if (rows == 0 || w == 0) return 0;
    VL_CHECK_ARG(vectors && queries && ids && dist_out && status, "vl_calculate_distances: null pointer");
    VL_CHECK_ARG(metric == VL_METRIC_COSINE || metric == VL_METRIC_SQL2, "vl_calculate_distances: unknown metric %d", metric);
    GatherArgs a = {vectors, n, dim, queries, rows, 1, w, 0, 0, ids, nullptr, nullptr, nullptr, 0, 0, nullptr, dist_out, status};
    return metric == VL_METRIC_COSINE ? launch_gather<VL_METRIC_COSINE>(a, (cudaStream_t)stream)
                                      : launch_gather<VL_METRIC_SQL2>(a, (cudaStream_t)stream);
}

extern "C" int vl_circulant_seeds(const float* vectors, int64_t n, int dim, const float* queries, int64_t rows,
                                  const int32_t* offsets, int w, int64_t first_row, int64_t modulo, int32_t* idx_out,
                                  float* dist_out, int metric, int* status, void* stream)
{
    VL_CHECK_ARG(dim > 0 && w >= 0 && rows >= 0 && n >= 0, "vl_circulant_seeds: bad size");
    if (rows == 0 || w == 0) return 0;
    VL_CHECK_ARG(vectors && queries && offsets && idx_out && dist_out && status, "vl_circulant_seeds: null pointer");
    VL_CHECK_ARG(modulo > 0 && modulo <= n && modulo < (1ll << 31), "vl_circulant_seeds: modulo %lld outside 1..%lld", (long long)modulo, (long long)n);
    VL_CHECK_ARG(metric == VL_METRIC_COSINE || metric == VL_METRIC_SQL2, "vl_circulant_seeds: unknown metric %d", metric);
    GatherArgs a = {vectors, n, dim, queries, rows, 1, w, 0, 0, nullptr, nullptr, nullptr, offsets, (int32_t)first_row, (int32_t)modulo,
                    idx_out, dist_out, status};
    return metric == VL_METRIC_COSINE ? launch_gather<VL_METRIC_COSINE>(a, (cudaStream_t)stream)
                                      : launch_gather<VL_METRIC_SQL2>(a, (cudaStream_t)stream);
}

extern "C" int vl_search_from_seeds(const float* queries, int64_t b, const int32_t* visit, int v,
                                    const int32_t* graph, int w, const float* vectors, int64_t n, int dim,
                                    int32_t* idx_out, float* dist_out, int metric, int* status, void* stream)
{
    VL_CHECK_ARG(dim > 0 && w >= 0 && v >= 0 && b >= 0 && n >= 0, "vl_search_from_seeds: bad size");
    if (b == 0 || v == 0 || w == 0) return 0;
    VL_CHECK_ARG(vectors && queries && visit && graph && idx_out && dist_out && status, "vl_search_from_seeds: null pointer");
    VL_CHECK_ARG(metric == VL_METRIC_COSINE || metric == VL_METRIC_SQL2, "vl_search_from_seeds: unknown metric %d", metric);
    GatherArgs a = {vectors, n, dim, queries, b, v, w, 0, 0, nullptr, visit, graph, nullptr, 0, 0, idx_out, dist_out, status};
    return metric == VL_METRIC_COSINE ? launch_gather<VL_METRIC_COSINE>(a, (cudaStream_t)stream)
                                      : launch_gather<VL_METRIC_SQL2>(a, (cudaStream_t)stream);
}
