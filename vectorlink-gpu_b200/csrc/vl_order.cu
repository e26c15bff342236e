// Order in which a build's rows are searched.  Rows are independent (a round reads the previous
// round's graph only), so any order gives the same lists; what the order decides is which rows are
// in flight together.  About 2,400 are, and each gathers several thousand candidate rows from its
// own neighbourhood: taken by row number their neighbourhoods have nothing in common, taken
// neighbourhood by neighbourhood they gather the same rows and L2 serves them.
//
// A row's key is the smallest hashed id within two steps of the graph (high word) and within one
// step (low word): rows that share most of their neighbourhood mostly share the minimum, so
// sorting by key groups them.  Two passes over the lists, bound by reading them (4 * w bytes per row and
// pass) and by the second pass's 4-byte gathers: 0.13 + 0.28 ms on 1,000,000 lists of 96.
// Whole builds without / with the order, ms: 1,000,000 x 128 from near neighbours 959 / 893, 60,007 x 768
// 155 / 141 (one warp per row: rounds of 729 / 660, 172 / 155, and 104 / 98 on 150,000 x 128).
#include "vl_common.cuh"
#include "vlgpu.h"

namespace {

constexpr int kThreads = 256;

// a bijection of the ids below 2^31, so distinct ids never tie and a key is a non-negative int64
__device__ __forceinline__ uint32_t hashed_id(uint32_t id) { return (id * 2654435761u) & 0x7fffffffu; }

// STEP 1: near[x] = min hashed id over x and its list.  STEP 2: key[x - lo] = (min of near over the
// same nodes) << 32 | near[x].  One warp per row.
template <int STEP>
__global__ void __launch_bounds__(kThreads)
locality_kernel(const int32_t* __restrict__ graph, int64_t n, int w, int64_t lo, int64_t hi,
                uint32_t* __restrict__ near, long long* __restrict__ keys)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp0 = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * kThreads) >> 5;
    for (int64_t x = lo + warp0; x < hi; x += nwarps) {
        const uint32_t own = STEP == 1 ? hashed_id((uint32_t)x) : near[x];
        uint32_t best = own;
        for (int j = lane; j < w; j += 32) {
            const int32_t y = __ldg(graph + x * w + j);
            if (y < 0 || (int64_t)y >= n) continue;      // MAXINT padding; a bad id is reported by the search itself
            const uint32_t h = STEP == 1 ? hashed_id((uint32_t)y) : near[y];
            best = h < best ? h : best;
        }
        best = __reduce_min_sync(0xffffffffu, best);
        if (lane == 0) {
            if (STEP == 1) near[x] = best;
            else keys[x - lo] = ((long long)best << 32) | own;
        }
    }
}

}  // namespace

extern "C" int vl_locality_keys(const int32_t* graph, int64_t n, int w, int64_t row_lo, int64_t row_hi, uint32_t* near,
                                long long* keys_out, void* stream)
{
    VL_CHECK_ARG(graph && near && keys_out, "vl_locality_keys: null pointer");
    VL_CHECK_ARG(w > 0 && n > 0 && 0 <= row_lo && row_lo <= row_hi && row_hi <= n, "vl_locality_keys: bad size");
    if (row_hi == row_lo) return 0;
    const int64_t cap = (int64_t)vl_sm_count() * 32, per = kThreads / 32;
    const int64_t all = (n + per - 1) / per, part = (row_hi - row_lo + per - 1) / per;
    locality_kernel<1><<<(unsigned)(all < cap ? all : cap), kThreads, 0, (cudaStream_t)stream>>>(graph, n, w, 0, n, near, keys_out);
    locality_kernel<2><<<(unsigned)(part < cap ? part : cap), kThreads, 0, (cudaStream_t)stream>>>(graph, n, w, row_lo, row_hi, near, keys_out);
    VL_CHECK_LAUNCH("locality_kernel");
    return 0;
}
