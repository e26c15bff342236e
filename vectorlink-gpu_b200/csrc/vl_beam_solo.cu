// Fused beam search with one warp per query row; when it is taken and what it measured stands in vl_beam_pair.cu.
#include "vl_beam_many.cuh"

namespace {

template <int LPR, int JP, int JU, int METRIC, bool ALIGNED>
int64_t solo_rows(const vl_beam_params& p)
{
    return rows_in_flight<1, LPR, JP, JU, METRIC, ALIGNED>(p);
}

template <int LPR, int JP, int JU, int METRIC, bool ALIGNED>
int solo_launch(const vl_beam_params& p, const int64_t* row_order, bool launch, int* blocks, int* smem, cudaStream_t stream)
{
    return many_launch<1, LPR, JP, JU, METRIC, ALIGNED>(p, row_order, launch, blocks, smem, stream);
}

}  // namespace

int64_t vl_beam_solo_rows(const vl_beam_params& p) { VL_BEAM_DISPATCH(p, solo_rows, p); }

int vl_beam_solo_launch(const vl_beam_params& p, const int64_t* row_order, bool launch, int* blocks, int* smem, cudaStream_t stream)
{
    VL_BEAM_DISPATCH(p, solo_launch, p, row_order, launch, blocks, smem, stream);
}
