// Launches of the fused beam search that keep as many rows in flight as fit, memos in global memory, one or two
// warps per row: shared by vl_beam_pair.cu, vl_beam_solo.cu and vl_beam_timed.cu.
#pragma once
#include "vl_beam_team.cuh"

namespace {

template <int TEAM, int LPR, int JP>
TeamSmem many_layout(const vl_beam_params& p)
{
    return team_layout(p.pvc * p.graph_w, p.sq_len, p.vq_len, p.seen_cap, LPR * JP * 16, p.memo ? p.memo_entries : 0, false, TEAM > 1);
}

// CTAs = rows of this launch that the device keeps in flight at once; 0 if a row does not fit, -1 on an error
template <int TEAM, int LPR, int JP, int JU, int METRIC, bool ALIGNED, bool TIMED = false>
int64_t rows_in_flight(const vl_beam_params& p)
{
    auto kernel = beam_team_kernel<LPR, JP, JU, METRIC, ALIGNED, TEAM, TIMED>;
    const TeamSmem lay = many_layout<TEAM, LPR, JP>(p);
    if (lay.total > vl_smem_limit()) return 0;
    int per_sm = 0;
    if (vl_allow_smem(kernel) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * TEAM, lay.total) != cudaSuccess) return -1;
    return (int64_t)vl_sm_count() * per_sm;
}

template <int TEAM, int LPR, int JP, int JU, int METRIC, bool ALIGNED, bool TIMED = false>
int many_launch(const vl_beam_params& p, const int64_t* row_order, bool launch, int* blocks, int* smem, cudaStream_t stream)
{
    const TeamSmem lay = many_layout<TEAM, LPR, JP>(p);
    VL_CHECK_ARG(lay.total <= vl_smem_limit(), "vl_beam_search: one row needs %d bytes of shared memory, the device offers %d", lay.total,
                 vl_smem_limit());
    const int64_t resident = rows_in_flight<TEAM, LPR, JP, JU, METRIC, ALIGNED, TIMED>(p);   // one wave; further rows are drawn as CTAs finish
    VL_CHECK_ARG(resident > 0, "vl_beam_search: occupancy query failed");
    const int grid = (int)(p.rows < resident ? p.rows : resident);
    *blocks = grid;
    *smem = lay.total;
    if (!launch) return 0;
    VL_CHECK_ARG(!p.memo || p.memo_slots >= grid, "vl_beam_search: memo has %lld slots, the launch keeps %d rows in flight",
                 (long long)p.memo_slots, grid);
    beam_team_kernel<LPR, JP, JU, METRIC, ALIGNED, TEAM, TIMED><<<grid, 32 * TEAM, lay.total, stream>>>(p, lay, row_order, nullptr);
    VL_CHECK_LAUNCH("beam_team_kernel");
    return 0;
}

}  // namespace
