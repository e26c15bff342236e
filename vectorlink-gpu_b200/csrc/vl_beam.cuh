// Shared parts of the fused beam search (vl_beam.cu): the visited set and the distance memo of a row.
#pragma once
#include "vl_common.cuh"

namespace {

constexpr int32_t kHashEmpty = -1;

__device__ __forceinline__ unsigned hash_slot(int32_t id, int shift) { return ((uint32_t)id * 2654435761u) >> shift; }

__device__ __noinline__ void hash_insert(int32_t* table, int slots, int shift, int32_t id, int* status)
{
    unsigned s = hash_slot(id, shift);
#pragma unroll 1
    for (int probe = 0; probe < slots; ++probe) {
        int32_t prev = atomicCAS(&table[s], kHashEmpty, id);
        if (prev == kHashEmpty || prev == id) return;
        s = (s + 1) & (slots - 1);
    }
    atomicOr(status, VL_STATUS_OVERFLOW);
}

__device__ __noinline__ bool hash_contains(const int32_t* table, int slots, int shift, int32_t id)
{
    unsigned s = hash_slot(id, shift);
#pragma unroll 1
    for (int probe = 0; probe < slots; ++probe) {
        int32_t v = table[s];
        if (v == id) return true;
        if (v == kHashEmpty) return false;
        s = (s + 1) & (slots - 1);
    }
    return false;
}

// Distance memo: 2-entry buckets of (ordered distance << 32 | id) keys, newest first.
__device__ __forceinline__ unsigned memo_bucket(uint32_t id, int shift, int buckets)
{
    return buckets > 1 ? (id * 2654435761u) >> shift : 0u;
}
// A new key goes to way `way` of its bucket (the caller alternates the way between
// iterations: first-in-first-out over two ways without reading the bucket).  An entry is one
// aligned 64-bit word, so lanes that collide on a slot can only lose an entry, never pair an
// id with another id's distance.
__device__ __forceinline__ void memo_put(vl_key_t* memo, int buckets, int shift, vl_key_t key, int way)
{
    memo[2 * (size_t)memo_bucket((uint32_t)key, shift, buckets) + way] = key;
}

}  // namespace

// Two warps per query row (vl_beam_pair.cu) or one (vl_beam_solo.cu).  Each plans the launch and, with `launch`, runs it;
// `blocks`: CTAs = rows in flight, `smem`: bytes of shared memory of one.
bool vl_beam_one_warp(const vl_beam_params& p);          // which of the two a launch takes
int64_t vl_beam_solo_rows(const vl_beam_params& p);      // rows that one warp each keeps in flight
int vl_beam_pair_launch(const vl_beam_params& p, const int64_t* row_order, bool launch, int* blocks, int* smem, cudaStream_t stream);
int vl_beam_solo_launch(const vl_beam_params& p, const int64_t* row_order, bool launch, int* blocks, int* smem, cudaStream_t stream);

// The same with two warps per row and cycle counters (vl_beam_timed.cu), if the launch asks for them and its rows fit.
bool vl_beam_timed_fits(const vl_beam_params& p);
int vl_beam_timed_launch(const vl_beam_params& p, const int64_t* row_order, bool launch, int* blocks, int* smem, cudaStream_t stream);

// A CTA of up to 16 warps per query row (vl_beam_team.cu), for launches of few rows; `arrivals` as in
// vl_beam_search_rows.  The memo is on chip, no scratch is needed.
bool vl_beam_team_fits(const vl_beam_params& p);
int vl_beam_team_launch(const vl_beam_params& p, unsigned int* arrivals, cudaStream_t stream);

// Calls LAUNCH<LPR, JP, JU, METRIC, ALIGNED>(args) for the launch's rows and returns its result: exact-fit
// instantiations (no per-chunk bounds tests) for the row sizes that matter, the smallest fitting shape otherwise.
#define VL_BEAM_EXACT(P, LAUNCH, L, J, U, ...)                                                     \
    if ((P).dim == 4 * L * U) {                                                                    \
        if ((P).metric == VL_METRIC_COSINE) return LAUNCH<L, J, U, VL_METRIC_COSINE, true>(__VA_ARGS__); \
        return LAUNCH<L, J, U, VL_METRIC_SQL2, true>(__VA_ARGS__);                                 \
    }
#define VL_BEAM_DISPATCH(P, LAUNCH, ...)                                                           \
    do {                                                                                           \
        const bool aligned__ = (P).dim % 4 == 0 && ((uintptr_t)(P).vectors | (uintptr_t)(P).queries) % 16 == 0; \
        if (aligned__) {                                                                           \
            VL_BEAM_EXACT(P, LAUNCH, 4, 4, 4, __VA_ARGS__)     /* dim 64 */                        \
            VL_BEAM_EXACT(P, LAUNCH, 4, 8, 6, __VA_ARGS__)     /* dim 96 */                        \
            VL_BEAM_EXACT(P, LAUNCH, 8, 4, 4, __VA_ARGS__)     /* dim 128: one 128-byte line per 8-lane load */ \
            VL_BEAM_EXACT(P, LAUNCH, 8, 8, 8, __VA_ARGS__)     /* dim 256 */                       \
            VL_BEAM_EXACT(P, LAUNCH, 16, 8, 6, __VA_ARGS__)    /* dim 384 */                       \
            VL_BEAM_EXACT(P, LAUNCH, 16, 8, 8, __VA_ARGS__)    /* dim 512 */                       \
            VL_BEAM_EXACT(P, LAUNCH, 32, 8, 6, __VA_ARGS__)    /* dim 768 */                       \
            VL_BEAM_EXACT(P, LAUNCH, 32, 8, 8, __VA_ARGS__)    /* dim 1024 */                      \
        }                                                                                          \
        const VlShape shape__ = vl_pick_shape((P).dim);                                            \
        VL_DISPATCH_SHAPE(shape__, {                                                               \
            if (aligned__) {                                                                       \
                if ((P).metric == VL_METRIC_COSINE) return LAUNCH<LPR, JP, 0, VL_METRIC_COSINE, true>(__VA_ARGS__); \
                return LAUNCH<LPR, JP, 0, VL_METRIC_SQL2, true>(__VA_ARGS__);                      \
            }                                                                                      \
            if ((P).metric == VL_METRIC_COSINE) return LAUNCH<LPR, JP, 0, VL_METRIC_COSINE, false>(__VA_ARGS__); \
            return LAUNCH<LPR, JP, 0, VL_METRIC_SQL2, false>(__VA_ARGS__);                         \
        });                                                                                        \
    } while (0)
