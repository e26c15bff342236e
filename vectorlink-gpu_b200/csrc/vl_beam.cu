// Fused beam search: the reference's closest_vectors loop (vectorlink_gpu/ann.py:37-93) as
// ONE kernel.  Per iteration the reference launches pop_n_ids (queue.py:87-95),
// search_from_seeds (kernels.py:204-311), two Queue.insert chains (queue.py:37-61: three
// torch.sort + gathers + dedup kernels each), add_new_to_seen_ (utils.py:61-82) and syncs
// the host; queue state makes a round trip through HBM every time.
//
// Here the warps of one CTA own one query row for the whole search (vl_beam_team.cuh):
//   * the query row, the search queue head, the visit queue and the visited set live in shared
//     memory (two sorted arrays of 64-bit (distance,id) keys and an open-addressing hash set);
//   * per iteration they pop `pvc` ids, read their graph rows, gather the candidate vectors with
//     128-bit loads (32/LPR rows per warp and step), and merge the candidates into the queues,
//     one warp each.
// This file holds the entry points: argument checks and the choice of the launch.
// The only HBM traffic that scales with the work is the gather: 4*dim bytes per candidate
// row + 4 bytes per neighbour id; that is the roofline this kernel is measured against.
//
// Queue semantics reproduced exactly (for capacity == length + candidates per iteration,
// which every queue the reference's drivers create satisfies): after an insert the queue is
// the `length` smallest distinct (distance,id) keys of old head + new candidates minus the
// excluded ids.  "Smallest `length` of a union" can be taken in any grouping, so candidates
// are merged 32 at a time and only those below the current cut-off key are looked at.
// The visited list `seen` (utils.py:61-89) is a set here: a candidate is kept out of the
// visit queue iff its id was popped while the list still had room, and the list's fill level
// (pvc ids per iteration, as for a batch in which at least one row always pops real ids)
// ends the feeding of the visit queue after ceil(E/pvc) iterations, like the reference.
// The two batch-wide decisions of the reference's host loop - "did any row's head change at a
// check iteration" and "was some row's pop always full" - are written to flag arrays for the
// caller, which re-runs a batch with a smaller n_iters or through the operator-level
// path when the reference would have taken a different course.
#include "vl_beam.cuh"

namespace {

int beam_dispatch(const vl_beam_params* pp, const int64_t* row_order, unsigned int* arrivals, int* blocks, int* smem, bool launch,
                  cudaStream_t stream)
{
    VL_CHECK_ARG(pp, "vl_beam_search: null params");
    const vl_beam_params& p = *pp;
    VL_CHECK_ARG(p.vectors && p.graph && p.queries && p.seed_ids && p.seed_dist && p.out_ids && p.out_dist &&
                 p.changed_flags && p.group_full && p.status, "vl_beam_search: null pointer");
    VL_CHECK_ARG(p.n > 0 && p.rows >= 0 && p.dim > 0, "vl_beam_search: bad size");
    VL_CHECK_ARG(p.metric == VL_METRIC_COSINE || p.metric == VL_METRIC_SQL2, "vl_beam_search: unknown metric %d", p.metric);
    VL_CHECK_ARG(p.pvc >= 1 && p.pvc <= 32, "vl_beam_search: parallel_visit_count %d outside 1..32", p.pvc);
    VL_CHECK_ARG(p.graph_w >= 1 && p.sq_len >= 1 && p.sq_len <= 4096, "vl_beam_search: bad queue shape");
    VL_CHECK_ARG(p.vq_len >= p.pvc, "vl_beam_search: visit queue of %d shorter than parallel_visit_count %d", p.vq_len, p.pvc);
    VL_CHECK_ARG(p.seen_cap >= 0 && p.readahead >= 1 && p.n_iters >= 0, "vl_beam_search: bad loop parameters");
    VL_CHECK_ARG(p.seed_cols >= 0 && p.seed_cols <= p.seed_ld, "vl_beam_search: bad seed shape");
    VL_CHECK_ARG(p.out_cols >= p.sq_len && p.out_cols <= p.out_ld, "vl_beam_search: bad output shape");
    VL_CHECK_ARG(!p.dump_last || p.out_cols >= p.sq_len + p.pvc * p.graph_w, "vl_beam_search: dump_last needs out_cols >= length + candidates");
    VL_CHECK_ARG(!p.dump_last || p.n_iters <= (p.seen_cap + p.pvc - 1) / p.pvc + 1, "vl_beam_search: dump_last past the last productive iteration");
    VL_CHECK_ARG(p.exclude_w == 0 || p.exclude, "vl_beam_search: exclusion width without a list");
    VL_CHECK_ARG(p.n_checks >= 0 && p.group_rows >= 0 && p.group_row0 >= 0, "vl_beam_search: bad flag shape");
    VL_CHECK_ARG(p.pvc * (int64_t)p.graph_w <= 65535, "vl_beam_search: %d candidates per iteration exceed 65535", p.pvc * p.graph_w);
    VL_CHECK_ARG(!p.memo || (p.memo_entries >= 2 && (p.memo_entries & (p.memo_entries - 1)) == 0 && (uintptr_t)p.memo % 16 == 0),
                 "vl_beam_search: memo_entries must be a power of two >= 2 and the memo 16-byte aligned");
    *blocks = *smem = 0;
    if (p.rows == 0) return 0;
    if (vl_beam_timed_fits(p)) return vl_beam_timed_launch(p, row_order, launch, blocks, smem, stream);
    if (vl_beam_team_fits(p)) return launch ? vl_beam_team_launch(p, arrivals, stream) : 0;   // no scratch: *blocks stays 0
    if (vl_beam_one_warp(p)) return vl_beam_solo_launch(p, row_order, launch, blocks, smem, stream);
    return vl_beam_pair_launch(p, row_order, launch, blocks, smem, stream);
}

}  // namespace

extern "C" int vl_beam_search(const vl_beam_params* params, void* stream)
{
    int blocks, smem;
    return beam_dispatch(params, nullptr, nullptr, &blocks, &smem, true, (cudaStream_t)stream);
}

extern "C" int vl_beam_search_rows(const vl_beam_params* params, const int64_t* row_order, uint32_t* arrivals, void* stream)
{
    int blocks, smem;
    return beam_dispatch(params, row_order, arrivals, &blocks, &smem, true, (cudaStream_t)stream);
}

extern "C" int vl_beam_search_plan(const vl_beam_params* params, int* smem_per_row, int* rows_per_block, int* blocks)
{
    int b = 0, s = 0;
    int rc = beam_dispatch(params, nullptr, nullptr, &b, &s, false, nullptr);
    if (rc) return rc;
    if (smem_per_row) *smem_per_row = s;
    if (rows_per_block) *rows_per_block = 1;
    if (blocks) *blocks = b;
    return 0;
}
