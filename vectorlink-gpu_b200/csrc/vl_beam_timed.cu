// The fused beam search with cycle counters (vl_beam_params.flags bit 0): two warps per row whatever the number of
// rows, so the counters show the phases of that kernel.  Kernels of their own, because the counters cost the others time
// even when they are off (vl_beam_team.cuh).
#include "vl_beam_many.cuh"

namespace {

template <int LPR, int JP, int JU, int METRIC, bool ALIGNED>
int timed_launch(const vl_beam_params& p, const int64_t* row_order, bool launch, int* blocks, int* smem, cudaStream_t stream)
{
    return many_launch<2, LPR, JP, JU, METRIC, ALIGNED, true>(p, row_order, launch, blocks, smem, stream);
}

template <int LPR, int JP, int JU, int METRIC, bool ALIGNED>
bool timed_fits(const vl_beam_params& p)
{
    return many_layout<2, LPR, JP>(p).total <= vl_smem_limit();
}

}  // namespace

bool vl_beam_timed_fits(const vl_beam_params& p)
{
    if (!(p.flags & 1) || !p.stats) return false;
    VL_BEAM_DISPATCH(p, timed_fits, p);
}

int vl_beam_timed_launch(const vl_beam_params& p, const int64_t* row_order, bool launch, int* blocks, int* smem, cudaStream_t stream)
{
    VL_BEAM_DISPATCH(p, timed_launch, p, row_order, launch, blocks, smem, stream);
}
