// Fused beam search with up to 16 warps per query row: launches of few rows.
//
// A launch of r rows keeps r CTAs busy, and a row's iteration is a chain of memory round trips (graph
// rows, memo, as many steps of candidate rows as the warps' registers need) and queue steps.  With rows to
// spare SMs, a row gets more warps, so that all candidate rows of an iteration are in flight together,
// and its distance memo moves into shared memory.
//
// Ending together: the reference's loop leaves at the first check at which no row of the batch
// changed (ann.py:85-91).  When every row of the batch is in flight at once (a cooperative launch), the CTAs
// agree on that check through one counter per check, so neither the iterations behind it nor a second
// run up to it are spent.  A row that changed does not wait; one that did not waits until one that did or
// all have reported.  The wait is bounded by wall time: when it runs out the row sets
// VL_STATUS_TIMEOUT and goes on as if the batch had changed.  Rows that saw the last report just before may then
// have stopped, so the launch's results are of no use: the caller runs the batch again without `arrivals`.
#include "vl_beam_team.cuh"

namespace {

struct TeamPlan { TeamSmem lay; int warps, per_sm; };

// Warps per row by rows per SM: a CTA of T warps takes T / 16 of an SM's registers, so T warps per row are
// free as long as every row is in flight.  Beyond 8 rows per SM two warps per row with the memo in global
// memory (vl_beam_pair.cu) keep 16 in flight.  With one row per SM, 16 warps pay for their barriers only where an
// iteration has 256 candidates.  Measured, ms with 2 / 4 / 8 / 16 warps (whole search, memo on chip):
//   1 row of 128 dimensions, 81 iterations of 128 candidates:    0.50 / 0.44 / 0.45 / 0.46  (one warp: 0.76)
//   16 rows of 768 dimensions, 161 iterations of 256 candidates: 5.0 / 2.03 / 1.39 / 1.25   (4.9)
//   1,000 rows of 96 dimensions, 91 iterations of 96 candidates: 0.78 / 1.19 / 2.24 / 3.9   (1.26; vl_beam_pair.cu 0.86)
bool team_plan(const vl_beam_params& p, TeamPlan& plan)
{
    const int64_t per_sm = (p.rows + vl_sm_count() - 1) / vl_sm_count();
    const int64_t m = (int64_t)p.pvc * p.graph_w;
    if (per_sm <= 1) plan.warps = m >= 256 ? 16 : 8;
    else if (per_sm <= 2) plan.warps = 8;
    else if (per_sm <= 4) plan.warps = 4;
    else if (per_sm <= 8) plan.warps = 2;
    else return false;
    plan.per_sm = kMaxTeam / plan.warps;
    const VlShape shape = vl_pick_shape(p.dim);
    const int budget = vl_smem_limit() / plan.per_sm - 1024;
    // the memo holds the ids a row gathers: about a quarter of the neighbours it looks at
    int entries = 1024;
    while (entries < 16384 && entries < (int64_t)p.seen_cap * p.graph_w / 4) entries <<= 1;
    // (with less than a quarter of that, gathers repeated cost more than the warps save: 1,000 rows of 768
    // dimensions with 1,024 of 16,384 entries 7.7 ms, vl_beam_pair.cu 3.6 ms)
    for (const int least = entries / 4 > 1024 ? entries / 4 : 1024; entries >= least; entries >>= 1) {
        plan.lay = team_layout((int)m, p.sq_len, p.vq_len, p.seen_cap, shape.lpr * shape.jp * 16, entries, true, true);
        if (plan.lay.total <= budget) return true;
    }
    return false;
}

template <int LPR, int JP, int JU, int METRIC, bool ALIGNED>
int team_launch(const vl_beam_params& p, const TeamPlan& plan, unsigned int* arrivals, cudaStream_t stream)
{
    auto kernel = beam_team_kernel<LPR, JP, JU, METRIC, ALIGNED, kMaxTeam>;
    TeamSmem lay = plan.lay;
    cudaError_t e = vl_allow_smem(kernel);
    VL_CHECK_ARG(e == cudaSuccess, "vl_beam_search: %s", cudaGetErrorString(e));
    const int64_t slots = (int64_t)vl_sm_count() * plan.per_sm;
    const unsigned grid = (unsigned)(p.rows < slots ? p.rows : slots);
    if (arrivals) {
        int per_sm = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, plan.warps * 32, lay.total);
        const bool one_batch = p.group_rows <= 0 || p.group_row0 / p.group_rows == (p.group_row0 + p.rows - 1) / p.group_rows;
        if (e != cudaSuccess || (int64_t)per_sm * vl_sm_count() < p.rows || grid < p.rows || !one_batch || p.dump_last ||
            p.out_cols < p.sq_len + p.pvc * p.graph_w)
            arrivals = nullptr;
    }
    if (arrivals) {
        vl_beam_params pv = p;
        const int64_t* order = nullptr;
        void* args[] = {&pv, &lay, &order, &arrivals};
        e = cudaLaunchCooperativeKernel((const void*)kernel, dim3(grid), dim3(plan.warps * 32), args, (size_t)lay.total, stream);
        VL_CHECK_ARG(e == cudaSuccess, "beam_team_kernel: %s", cudaGetErrorString(e));
    } else {
        kernel<<<grid, plan.warps * 32, lay.total, stream>>>(p, lay, nullptr, nullptr);
    }
    VL_CHECK_LAUNCH("beam_team_kernel");
    return 0;
}

}  // namespace

bool vl_beam_team_fits(const vl_beam_params& p)
{
    TeamPlan plan;
    return p.rows > 0 && team_plan(p, plan);
}

int vl_beam_team_launch(const vl_beam_params& p, unsigned int* arrivals, cudaStream_t stream)
{
    TeamPlan plan;
    VL_CHECK_ARG(team_plan(p, plan), "vl_beam_search: rows do not fit a CTA each");
    VL_BEAM_DISPATCH(p, team_launch, p, plan, arrivals, stream);
}
