// Fused beam search with two warps per query row and 16 rows in flight per SM, or one warp (vl_beam_solo.cu) and 20
// rows: launches of many rows.
//
// A row's iteration is a chain of memory round trips and queue steps, so a launch is bound by latency
// at the number of rows that can be in flight.  That number is bound in turn by the rows' memos
// (64 KB each at a build's 30,720 evaluations, 155 MB in all, already more than the 126 MB L2), not by
// registers: a second warp per row halves the id, memo and gather phases and runs the two queue steps side
// by side at 64 registers per thread, without another row's memo.  Build rounds, ms, one warp per row with
// the queue merges of before (128 registers) / this, rows in neighbourhood order, on one B200:
//   1,000,000 x 128, lists of 96 from near neighbours: 660 / 526
//   60,007 x 768, lists of 192:                        155 / 121  (shared memory holds 9 of these rows per SM, also below)
//   150,000 x 128, rounds 2 and 3:                  98, 97 / 76, 78
// 10,000 searches of 1,000,000 x 128: 6.6 / 5.3; 2,500 of 200,000 x 256: 2.33 / 1.55.  12 rows per SM at 80
// registers (two gather steps in flight): 541, 119, 81; one warp per row with the same queue step at 16 rows per
// SM: 528, 137, 75, at 24 rows per SM: 740, 144, 108.
//
// One warp per row and 20 rows per SM is better where a row's memo is small (32 KB or none, so that 2,960 of them do not
// push each other out of L2) and its rows are short: searches of 30,000 x 96 (clusters) 10.0 / 8.9 ms, 10,000 of
// 1,000,000 x 128 5.2 / 4.8, the first build round (no memo) of 150,000 x 128 253 / 227.  That also holds where shared memory
// and not registers bounds the rows in flight (wide lists; first rounds without memo of 10,000 to 60,000 rows, two warps /
// one warp): 128 dimensions at degree 40, 48, 64, 80, 96, 128, 192: 160 / 137, 233 / 205, 441 / 401, 408 / 383, 652 / 602,
// 910 / 912, 1,758 / 1,547; 64 dimensions at 64, 80, 96: 271 / 250, 258 / 238, 410 / 374; 32 and 100 dimensions at 64: 248 / 235,
// 527 / 415.  Only rows of 96 dimensions go the other way from degree 56 on (254 / 261; 64, 80, 96: 333 / 350, 293 / 331, 456 / 522).
// Rows of 256 dimensions gain only where one warp per row keeps a launch in flight that two warps do not: with memos of 64 KB
// 2,368 searches 2.40 / 2.68, 2,500 3.47 / 2.79, 2,960 3.68 / 3.09, 3,100 3.81 / 5.05.  A second wave saved gains nothing (4,800,
// 5,300, 5,900 searches 5.94 / 5.85, 6.05 / 6.21, 6.44 / 6.61; CTAs draw their next row as they finish, so waves blur); first round of
// 20,000: 44.8 / 46.9; 768 dimensions lose (3,000 searches: 3.3 / 4.9).
#include "vl_beam_many.cuh"

namespace {

template <int LPR, int JP, int JU, int METRIC, bool ALIGNED>
bool pair_fits(const vl_beam_params& p)
{
    return many_layout<2, LPR, JP>(p).total <= vl_smem_limit();
}

template <int LPR, int JP, int JU, int METRIC, bool ALIGNED>
int64_t pair_rows(const vl_beam_params& p)
{
    return rows_in_flight<2, LPR, JP, JU, METRIC, ALIGNED>(p);
}

template <int LPR, int JP, int JU, int METRIC, bool ALIGNED>
int pair_launch(const vl_beam_params& p, const int64_t* row_order, bool launch, int* blocks, int* smem, cudaStream_t stream)
{
    return many_launch<2, LPR, JP, JU, METRIC, ALIGNED>(p, row_order, launch, blocks, smem, stream);
}

bool two_warps_fit(const vl_beam_params& p) { VL_BEAM_DISPATCH(p, pair_fits, p); }
int64_t two_warp_rows(const vl_beam_params& p) { VL_BEAM_DISPATCH(p, pair_rows, p); }

}  // namespace

// the choice described above; and a single warp needs 10 instead of 14 bytes of shared memory per candidate, so rows
// of more than about 15,000 candidates take it whatever their dimension
bool vl_beam_one_warp(const vl_beam_params& p)
{
    if (!two_warps_fit(p)) return true;
    if (p.dim <= 128) return p.memo_entries <= 4096;
    return p.dim <= 256 && p.memo_entries <= 8192 && p.rows > two_warp_rows(p) && p.rows <= vl_beam_solo_rows(p);
}

int vl_beam_pair_launch(const vl_beam_params& p, const int64_t* row_order, bool launch, int* blocks, int* smem, cudaStream_t stream)
{
    VL_BEAM_DISPATCH(p, pair_launch, p, row_order, launch, blocks, smem, stream);
}
