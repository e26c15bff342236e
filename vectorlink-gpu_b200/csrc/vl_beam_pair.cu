// Fused beam search with two warps per query row and 16 rows in flight per SM, or one warp and 20 rows:
// launches of many rows.
//
// A row's iteration is a chain of memory round trips and queue steps, so a launch is bound by latency
// at the number of rows that can be in flight.  That number is bound in turn by the rows' memos
// (64 KB each at a build's 30,720 evaluations, 155 MB in all, already more than the 126 MB L2), not by
// registers: a second warp per row halves the id, memo and gather phases and runs the two queue steps side
// by side at 64 registers per thread, without another row's memo.  Build rounds, ms, one warp per row with
// the queue merges of before (128 registers) / this, rows in neighbourhood order, on one B200:
//   1,000,000 x 128, lists of 96 from near neighbours: 660 / 526
//   60,007 x 768, lists of 192:                        155 / 121
//   150,000 x 128, rounds 2 and 3:                  98, 97 / 76, 78
// 10,000 searches of 1,000,000 x 128: 6.6 / 5.3; 2,500 of 200,000 x 256: 2.33 / 1.55.  12 rows per SM at 80
// registers (two gather steps in flight): 541, 119, 81; one warp per row with the same queue step at 16 rows per
// SM: 528, 137, 75, at 24 rows per SM: 740, 144, 108.
//
// One warp per row and 20 rows per SM (vl_beam_solo) is better where a row's memo is small (32 KB or none, so that
// 2,960 of them do not push each other out of L2) and its rows are short: searches of 30,000 x 96 (clusters)
// 10.0 / 8.9 ms, 10,000 of 1,000,000 x 128 5.2 / 4.8, the first build round (no memo) of 150,000 x 128 253 / 227.  Rows
// of 256 dimensions gain only where 20 rows per SM save a wave (2,500 searches, memos of 64 KB: 1.54 / 1.08; first round of
// 20,000: 44.8 / 46.9); 768 dimensions lose (3,000 searches: 3.3 / 4.9).
#include "vl_beam_team.cuh"

namespace {

template <int TEAM, int LPR, int JP>
TeamSmem many_layout(const vl_beam_params& p)
{
    return team_layout(p.pvc * p.graph_w, p.sq_len, p.vq_len, p.seen_cap, LPR * JP * 16, p.memo ? p.memo_entries : 0, false, TEAM > 1);
}

template <int TEAM, int LPR, int JP, int JU, int METRIC, bool ALIGNED>
int many_launch(const vl_beam_params& p, const int64_t* row_order, bool launch, int* blocks, int* smem, cudaStream_t stream)
{
    auto kernel = beam_team_kernel<LPR, JP, JU, METRIC, ALIGNED, TEAM>;
    const TeamSmem lay = many_layout<TEAM, LPR, JP>(p);
    int per_sm = 0;
    VL_CHECK_ARG(lay.total <= vl_smem_limit(), "vl_beam_search: one row needs %d bytes of shared memory, the device offers %d", lay.total,
                 vl_smem_limit());
    cudaError_t e = vl_allow_smem(kernel);
    VL_CHECK_ARG(e == cudaSuccess, "vl_beam_search: %s", cudaGetErrorString(e));
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * TEAM, lay.total);
    VL_CHECK_ARG(e == cudaSuccess && per_sm > 0, "vl_beam_search: occupancy query failed");
    const int64_t resident = (int64_t)vl_sm_count() * per_sm;   // one resident wave; further rows are drawn as CTAs finish
    const int grid = (int)(p.rows < resident ? p.rows : resident);
    *blocks = grid;
    *smem = lay.total;
    if (!launch) return 0;
    VL_CHECK_ARG(!p.memo || p.memo_slots >= grid, "vl_beam_search: memo has %lld slots, the launch keeps %d rows in flight",
                 (long long)p.memo_slots, grid);
    kernel<<<grid, 32 * TEAM, lay.total, stream>>>(p, lay, row_order, nullptr);
    VL_CHECK_LAUNCH("beam_team_kernel");
    return 0;
}

// the choice described above
bool vl_beam_solo(const vl_beam_params& p)
{
    if (p.dim <= 128) return p.memo_entries <= 4096;
    const int64_t sms = vl_sm_count();
    return p.dim <= 256 && p.memo_entries <= 8192 && p.rows > sms * many_per_sm(2) && p.rows <= sms * many_per_sm(1);
}

template <int LPR, int JP, int JU, int METRIC, bool ALIGNED>
int pair_launch(const vl_beam_params& p, const int64_t* row_order, bool launch, int* blocks, int* smem, cudaStream_t stream)
{
    // a single warp needs 10 instead of 14 bytes of shared memory per candidate: rows of more than about 15,000 take it
    if (vl_beam_solo(p) || many_layout<2, LPR, JP>(p).total > vl_smem_limit())
        return many_launch<1, LPR, JP, JU, METRIC, ALIGNED>(p, row_order, launch, blocks, smem, stream);
    return many_launch<2, LPR, JP, JU, METRIC, ALIGNED>(p, row_order, launch, blocks, smem, stream);
}

}  // namespace

int vl_beam_pair_launch(const vl_beam_params& p, const int64_t* row_order, bool launch, int* blocks, int* smem, cudaStream_t stream)
{
    VL_BEAM_DISPATCH(p, pair_launch, p, row_order, launch, blocks, smem, stream);
}
