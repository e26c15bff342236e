"""The launches of the fused beam search - a CTA of several warps per row when rows are few, two warps per
row beyond - against the step-by-step operator path, at the row counts where the launch changes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rows_of(seed, count, dim, metric):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    x = torch.randn((count, dim), generator=g, device=DEV)
    return torch.nn.functional.normalize(x, dim=1) if metric == "cosine" else (x * 40).round_()


def search_both_ways(ann, queries):
    """The whole queues (ids, distances, columns behind the head too) and the loop counts: fused, operator path."""
    from vectorlink_gpu.ann import closest_vectors
    out = []
    for stepwise in (False, True):
        ann.configuration["stepwise"] = stepwise
        queue = ann.search(queries)
        out.append((queue.indices.clone(), queue.distances.clone(), closest_vectors.last_count))
    ann.configuration["stepwise"] = False
    return out


# one row per SM (16 or 8 warps), two (8), four (4), eight (2), more (one or two warps, memo in global memory); 148 SMs
@pytest.mark.parametrize("count", [1, 2, 5, 148, 149, 296, 297, 592, 593, 1184, 1185, 3100])
@pytest.mark.parametrize("metric,dim,degree", [("cosine", 64, 16), ("l2", 100, 24), ("cosine", 768, 64)])
def test_every_split_of_a_row_gives_the_operator_path_queues(count, metric, dim, degree, built_lib):
    from vectorlink_gpu import ANN, _lib
    if degree == 64 and count > 300:
        pytest.skip("the operator path takes long at this width")
    ann = ANN(vectors=rows_of(1, 3001, dim, metric), beam_size=degree, visit_queue_factor=2, recall_search_queue_factor=2,
              metric=metric, init="knn_tile", optimization_loops=1)
    (fused, steps) = search_both_ways(ann, rows_of(2, count, dim, metric))
    assert torch.equal(fused[0], steps[0]) and torch.equal(fused[1], steps[1])
    assert fused[2] == steps[2]
    assert _lib.read_status(DEV) == 0


@pytest.mark.parametrize("count", [2369, 2960, 2961])      # around one wave of either split at 256 dimensions
@pytest.mark.parametrize("memo", [{}, {"memo": False}, {"memo_entries": 2}, {"memo_entries": 4096}, {"memo_entries": 8192}])
def test_one_or_two_warps_per_row_give_the_same_queues(count, memo, built_lib):
    from vectorlink_gpu import ANN
    ann = ANN(vectors=rows_of(1, 3001, 256, "l2"), beam_size=8, visit_queue_factor=2, recall_search_queue_factor=2,
              metric="l2", init="knn_tile", optimization_loops=1)
    ann.configuration.update(memo)
    (fused, steps) = search_both_ways(ann, rows_of(2, count, 256, "l2"))
    assert torch.equal(fused[0], steps[0]) and torch.equal(fused[1], steps[1]) and fused[2] == steps[2]


@pytest.mark.parametrize("count,dim", [(3, 64), (1300, 64), (1300, 512), (1300, 50)])
def test_cycle_counters(count, dim, built_lib):
    """The counters of every phase are there when they are asked for, in 16 words, and change nothing."""
    import vectorlink_gpu.ann as A
    ann = A.ANN(vectors=rows_of(1, 3001, dim, "cosine"), beam_size=16, visit_queue_factor=2, recall_search_queue_factor=2,
                init="knn_tile", optimization_loops=1)
    queries = rows_of(2, count, dim, "cosine")
    want = ann.search(queries).indices.clone()
    stats = {}
    try:
        for timers in (False, True):
            (A.STATS, A.STATS_TIMERS) = (torch.zeros(24, dtype=torch.int64, device=DEV), timers)
            assert torch.equal(ann.search(queries).indices, want)
            stats[timers] = A.STATS.tolist()
    finally:
        (A.STATS, A.STATS_TIMERS) = (None, False)
    assert stats[False][7] > 0 and stats[True][7] > 0
    assert stats[False][8:] == [0] * 16
    assert all(stats[True][i] > 0 for i in (8, 9, 10, 12, 13)) and stats[True][11] == 0 and stats[True][14:] == [0] * 10


@pytest.mark.parametrize("width,memo_entries", [(16, 0), (48, 0), (52, 8192), (64, 0), (128, 0)])
def test_one_warp_per_row_is_chosen_by_the_rows_that_fit(width, memo_entries, built_lib):
    """256 dimensions, where shared memory allows 20 or fewer rows per SM: the plan never leaves rows to a second wave because of
    one warp per row, and keeps all rows in flight where two warps per row would not."""
    import ctypes
    from vectorlink_gpu._lib import BeamParams, check, lib
    some = torch.zeros(4, device=DEV).data_ptr()           # a plan reads no memory

    def planned(rows):
        p = BeamParams(vectors=some, n=20_000, dim=256, graph=some, graph_w=width, pvc=4, queries=some, rows=rows, seed_ids=some,
                       seed_dist=some, seed_ld=2 * width, seed_cols=2 * width, sq_len=2 * width, vq_len=2 * width, seen_cap=10 * width,
                       out_ids=some, out_dist=some, out_ld=2 * width, out_cols=2 * width, n_iters=10, readahead=5, self_base=-1,
                       changed_flags=some, group_full=some, status=some, memo_entries=memo_entries)
        (size, per_block, blocks) = (ctypes.c_int(), ctypes.c_int(), ctypes.c_int())
        check(lib().vl_beam_search_plan(ctypes.byref(p), ctypes.byref(size), ctypes.byref(per_block), ctypes.byref(blocks)), "plan")
        return blocks.value

    two_warps = planned(100_000)                           # rows in flight with two warps per row
    blocks = [planned(rows) for rows in range(1200, 3200, 20)]
    for rows, b in zip(range(1200, 3200, 20), blocks):
        assert b == (rows if b > two_warps else min(rows, two_warps)), rows


@pytest.mark.parametrize("dim,memo", [(64, {}), (64, {"memo": False}), (512, {})])      # two, one and two warps per row
@pytest.mark.parametrize("degree,pvc,exclude_w", [(64, 4, 0), (64, 4, 3), (32, 16, 3), (33, 4, 0)])
def test_wide_lists_with_and_without_exclusions(degree, pvc, exclude_w, dim, memo, built_lib):
    """Iterations of 132 to 512 candidates, with exclusion lists and without, and with 16 ids popped at once (the visit
    queue is then offered every candidate), at a row count of one or two warps per row."""
    import vectorlink_gpu.ann as A
    count = 1300
    ann = A.ANN(vectors=rows_of(1, 3001, dim, "cosine"), beam_size=degree, visit_queue_factor=2, recall_search_queue_factor=2,
                parallel_visit_count=pvc, init="knn_tile", optimization_loops=1)
    queries = rows_of(2, count, dim, "cosine")
    exclude = None
    if exclude_w:
        exclude = ann.search(queries).indices[:, :exclude_w].contiguous()      # the nearest ones may not be found
        exclude[::2, -1] = 2147483647
    got = []
    for more in (memo, {"stepwise": True}):
        queue = A.initial_search_queue(ann.vectors, queries, ann.configuration)
        A.closest_vectors(queries, queue, ann.vectors, ann.beams, dict(ann.configuration, **more), exclude)
        got.append((queue.indices, queue.distances, A.closest_vectors.last_count))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]) and got[0][2] == got[1][2]


@pytest.mark.parametrize("degree,width,dim,visits,exclude", [(128, 384, 32, 3, 5), (128, 384, 300, 3, 5), (520, 520, 32, 1, 1)])
def test_rows_of_many_candidates_per_iteration_are_fused(degree, width, dim, visits, exclude, built_lib):
    """12,288 and 16,640 candidates per iteration, which the operator path refuses, against the oracle.  With lists of
    entrants the last needs more shared memory than a CTA can have.  (The one check comes after the budget: a batch that
    ends early is sorted whole, and rows of this capacity are refused there.)"""
    import oracle
    import vectorlink_gpu.ann as A
    config = oracle.make_config(beam_size=degree, parallel_visit_count=32, visit_queue_factor=visits, exclude_factor=exclude)
    config["speculative_readahead"] = A.loop_bounds(config)[0] + 1
    rng = np.random.default_rng(degree)
    vectors = rng.standard_normal((20_000, dim), dtype=np.float32)
    vectors /= np.linalg.norm(vectors, axis=1, keepdims=True)
    graph = rng.integers(0, 20_000, (20_000, width)).astype(np.int32)
    queries = vectors[:3].copy()
    m = 32 * width
    queue = oracle.Queue(3, width, width + m)
    queue.insert(graph[:3], oracle.calculate_distances(vectors, graph)[:3])
    mine = A.Queue(3, width, width + m)
    mine.indices.copy_(torch.from_numpy(queue.indices))
    mine.distances.copy_(torch.from_numpy(queue.distances))
    A.PROFILE = []
    try:
        A.closest_vectors(torch.from_numpy(queries).to(DEV), mine, torch.from_numpy(vectors).to(DEV), torch.from_numpy(graph).to(DEV), config)
        assert len(A.PROFILE) > 0
    finally:
        A.PROFILE = None
    count = oracle.closest_vectors(queries, queue, vectors, graph, config)
    assert A.closest_vectors.last_count == count
    assert np.array_equal(mine.indices[:, :width].cpu().numpy(), queue.indices[:, :width])
    assert np.array_equal(mine.distances[:, :width].cpu().numpy(), queue.distances[:, :width])


def test_a_batch_that_stops_early_ends_together(built_lib):
    """Few rows stop at the reference's check: one launch, no second run up to it."""
    import vectorlink_gpu.ann as A
    ann = A.ANN(vectors=rows_of(3, 4000, 64, "cosine"), beam_size=16, visit_queue_factor=2, recall_search_queue_factor=2,
                init="knn_tile", optimization_loops=1)
    k_none = A.loop_bounds(ann.configuration)[0]
    early = 0
    for count in (1, 2, 3):
        for seed in range(4):
            queries = rows_of(10 + seed, count, 64, "cosine")
            A.PROFILE = []
            try:
                ann.search(queries)
                launches = len(A.PROFILE)
            finally:
                A.PROFILE = None
            (fused, steps) = search_both_ways(ann, queries)
            assert torch.equal(fused[0], steps[0]) and torch.equal(fused[1], steps[1]) and fused[2] == steps[2]
            assert launches == 1
            early += steps[2] <= k_none
    assert early > 0


def flat_rows(seed, count, dim):
    """Unit vectors of `dim` dimensions in a subspace of six: few neighbours are hard to find there."""
    return torch.nn.functional.pad(rows_of(seed, count, 6, "cosine"), (0, dim - 6)).contiguous()


def converging_index(degree, dim):
    """An index whose searches settle long before their budget is spent: easy rows, a short search queue, a long visit queue."""
    from vectorlink_gpu import ANN
    return ANN(vectors=flat_rows(3, 4000, dim), beam_size=degree, visit_queue_factor=6, recall_search_queue_factor=1,
               init="knn_tile", optimization_loops=1)


def launches_of(ann, queries):
    import vectorlink_gpu.ann as A
    A.PROFILE = []
    try:
        ann.search(queries)
        return len(A.PROFILE)
    finally:
        A.PROFILE = None


# 8 warps per row and one row per SM, 8 and two, 4 and four, 2 and eight; 16 warps where an iteration has 256 candidates
@pytest.mark.parametrize("count,degree", [(100, 16), (200, 16), (500, 16), (1000, 16), (100, 64)])
@pytest.mark.parametrize("exclude_w", [0, 2])
def test_larger_batches_that_stop_early_end_together(count, degree, exclude_w, built_lib):
    import vectorlink_gpu.ann as A
    ann = converging_index(degree, 64)
    queries = flat_rows(4, count, 64)
    exclude = ann.search(queries).indices[:, :exclude_w].contiguous() if exclude_w else None
    got = []
    for more in ({}, {"stepwise": True}):
        queue = A.initial_search_queue(ann.vectors, queries, ann.configuration)
        A.PROFILE = []
        try:
            A.closest_vectors(queries, queue, ann.vectors, ann.beams, dict(ann.configuration, **more), exclude)
            launches = len(A.PROFILE)
        finally:
            A.PROFILE = None
        assert launches == (0 if more else 1)
        got.append((queue.indices, queue.distances, A.closest_vectors.last_count))
    assert got[1][2] <= A.loop_bounds(ann.configuration)[0]
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]) and got[0][2] == got[1][2]


# dimensions whose oracle cases are too few rows for the launches of many
@pytest.mark.parametrize("metric,dim", [("cosine", 384), ("l2", 384), ("cosine", 512), ("l2", 512), ("cosine", 1536), ("l2", 2052), ("cosine", 1024)])
def test_many_rows_of_wide_vectors(metric, dim, built_lib):
    from vectorlink_gpu import ANN
    ann = ANN(vectors=rows_of(1, 2001, dim, metric), beam_size=16, visit_queue_factor=2, recall_search_queue_factor=2,
              metric=metric, init="knn_tile", optimization_loops=1)
    (fused, steps) = search_both_ways(ann, rows_of(2, 1300, dim, metric))
    assert torch.equal(fused[0], steps[0]) and torch.equal(fused[1], steps[1]) and fused[2] == steps[2]


@pytest.mark.parametrize("count", [200, 500, 1000])
def test_a_wait_that_runs_out_is_answered_by_a_second_run(count, built_lib):
    """Rows of a batch wait at most a microsecond for the others: some give up, and the batch is searched again without
    waits.  The queues and the count are the operator path's, and no status bit stays behind."""
    import vectorlink_gpu.ann as A
    from vectorlink_gpu import _lib
    ann = converging_index(16, 64)
    queries = flat_rows(4, count, 64)
    ann.configuration["wait_us"] = 1
    launches = launches_of(ann, queries)
    (fused, steps) = search_both_ways(ann, queries)
    assert steps[2] <= A.loop_bounds(ann.configuration)[0]      # the batch does stop early
    assert launches > 1
    assert torch.equal(fused[0], steps[0]) and torch.equal(fused[1], steps[1]) and fused[2] == steps[2]
    assert _lib.read_status(DEV) == 0


@pytest.mark.parametrize("metric", ["cosine", "l2"])
@pytest.mark.parametrize("dim,offset", [(1, 0), (3, 0), (50, 0), (127, 0), (255, 0), (511, 0), (1023, 0), (1027, 0), (64, 1), (96, 3)])
def test_rows_without_whole_aligned_chunks_give_the_operator_path_results(dim, offset, metric, built_lib):
    """Dimensions that are no multiple of four, and rows whose storage starts off a 16-byte boundary: searches of few
    and of many rows, a build, and the same build without the padded copy."""
    import vectorlink_gpu.ann as A
    n = 1500
    store = torch.empty(n * dim + offset, device=DEV)
    vectors = store[offset:].view(n, dim)
    vectors.copy_(rows_of(5, n, dim, metric))
    assert vectors.is_contiguous() and (dim % 4 or vectors.data_ptr() % 16)
    config = dict(beam_size=8, visit_queue_factor=2, recall_search_queue_factor=2, metric=metric, optimization_loops=1)
    ann = A.ANN(vectors=vectors, **config)
    plain = A.generate_ann(vectors, dict(ann.configuration, stepwise=True))
    assert torch.equal(ann.beams, plain[0]) and torch.equal(ann.distances, plain[1])
    keep = A._chunked_rows
    A._chunked_rows = lambda v: v
    try:
        uncopied = A.generate_ann(vectors, ann.configuration)
    finally:
        A._chunked_rows = keep
    assert torch.equal(uncopied[0], plain[0]) and torch.equal(uncopied[1], plain[1])
    for count in (3, 1300):
        (fused, steps) = search_both_ways(ann, rows_of(6, count, dim, metric))
        assert torch.equal(fused[0], steps[0]) and torch.equal(fused[1], steps[1]) and fused[2] == steps[2]


def test_row_order_of_a_build_changes_nothing(built_lib):
    import vectorlink_gpu.ann as A
    vectors = rows_of(7, 5000, 48, "cosine")
    config = dict(A.ANN(vectors=vectors[:64].contiguous(), beam_size=8).configuration, batch_size=1700)
    keep = A.ORDER_MIN_ROWS
    graphs = []
    try:
        for least in (keep, 1):
            A.ORDER_MIN_ROWS = least
            graphs.append(A.generate_ann(vectors, dict(config, memo=True)))
    finally:
        A.ORDER_MIN_ROWS = keep
    assert torch.equal(graphs[0][0], graphs[1][0]) and torch.equal(graphs[0][1], graphs[1][1])


def test_profiled_launches_include_their_row_order(built_lib):
    import vectorlink_gpu.ann as A
    vectors = rows_of(7, 3000, 48, "cosine")
    config = dict(A.ANN(vectors=vectors[:64].contiguous(), beam_size=8).configuration, memo=True, optimization_loops=1)
    real = A._row_order

    def slow_order(graph, self_base, rows, config):
        if self_base >= 0:
            torch.cuda._sleep(100_000_000)              # 50 ms at 2 GHz
        return real(graph, self_base, rows, config)

    A._row_order = slow_order
    A.PROFILE = []
    try:
        A.generate_ann(vectors, config)
        torch.cuda.synchronize()
        ms = [p["start"].elapsed_time(p["end"]) for p in A.PROFILE if p["tag"] == "round0"]
    finally:
        (A._row_order, A.PROFILE) = (real, None)
    assert ms and ms[0] > 40


def test_first_row_as_a_float(built_lib):
    """Row numbers were and are taken as torch.arange takes them."""
    from vectorlink_gpu import ANN
    ann = ANN(vectors=rows_of(1, 500, 32, "cosine"), beam_size=8, optimization_loops=1)
    queries = rows_of(2, 3, 32, "cosine")
    assert torch.equal(ann.search(queries, first_row=7.0).indices, ann.search(queries, first_row=7).indices)


@pytest.mark.parametrize("n,w,lo,hi", [(1, 1, 0, 1), (50, 7, 10, 50), (3000, 96, 0, 3000)])
def test_locality_keys(n, w, lo, hi, built_lib):
    from vectorlink_gpu._lib import lib, ptr, stream_of
    rng = np.random.default_rng(n)
    graph = rng.integers(0, n, size=(n, w)).astype(np.int32)
    graph[rng.random((n, w)) < 0.2] = 2147483647
    g = torch.from_numpy(graph).to(DEV)
    near = torch.empty(n, dtype=torch.int32, device=DEV)
    keys = torch.empty(hi - lo, dtype=torch.int64, device=DEV)
    assert lib().vl_locality_keys(ptr(g), n, w, lo, hi, ptr(near), ptr(keys), stream_of(g)) == 0
    hashed = (np.arange(n, dtype=np.uint64) * 2654435761 & 0x7fffffff).astype(np.int64)

    def smallest(values):
        padded = np.append(values, 1 << 40)
        return np.minimum(values, padded[np.where(graph < n, graph, n)].min(axis=1))

    one = smallest(hashed)
    two = smallest(one)
    assert np.array_equal(keys.cpu().numpy(), ((two << 32) | one)[lo:hi])


@pytest.mark.parametrize("rows,cands,segments,parts", [((0, 1), (0, 3000), 1, 2), ((0, 129), (0, 3000), 1, 32),
                                                       ((2990, 3000), (100, 2777), 2, 5), ((7, 300), (0, 255), 1, 3)])
@pytest.mark.parametrize("dim", [64, 200])
def test_divided_segments_give_the_same_proposals(rows, cands, segments, parts, dim, built_lib):
    from vectorlink_gpu import knn_tile
    rows_bf16, norms = knn_tile.prepare(rows_of(8, 3000, dim, "l2"), want_norms=True)
    keep = knn_tile._parts
    got = []
    try:
        for count in (1, parts):
            knn_tile._parts = lambda *a: count
            got.append(knn_tile.proposals(rows_bf16, norms, rows, cands, segments).clone())
    finally:
        knn_tile._parts = keep
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("metric", ["cosine", "l2"])
@pytest.mark.parametrize("dim", [1, 50, 64, 96, 128, 250, 256, 384, 512, 768, 1024, 1030])
def test_circulant_seeds_equal_the_operators(dim, metric, built_lib):
    """Seed ids and distances of one kernel against the two operators, rows and widths off every step and run size."""
    from vectorlink_gpu.kernels import calculate_distances, circulant_seeds
    from vectorlink_gpu.utils import generate_queue_circulants, primes, seed_offsets
    vectors = rows_of(9, 701, dim, metric)
    for (rows, w, first_row, modulo) in ((1, 1, 0, 701), (1, 64, 5, 701), (3, 1920, 0, 701), (157, 33, 10_000, 700), (5000, 31, 0, 1)):
        queries = rows_of(10, rows, dim, metric)
        ids = generate_queue_circulants(rows, modulo, primes(w, DEV), first_row)
        want = calculate_distances(vectors, ids, metric=metric, queries=queries)
        (got_ids, got) = circulant_seeds(vectors, queries, seed_offsets(w, DEV), first_row, modulo, metric)
        assert torch.equal(got_ids, ids) and torch.equal(got, want)
