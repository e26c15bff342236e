"""Calls of several host threads, each on a stream of its own: what one of them keeps or shares must not reach the others."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def unit_rows(seed, count, dim):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.nn.functional.normalize(torch.randn((count, dim), generator=g, device=DEV), dim=1)


def serial_and_threaded(calls, passes):
    """What every call gives by itself, and what it gives `passes` times in a thread and stream of its own while the
    others run: each stream is busy for some milliseconds first, so that the launches of a pass start together."""
    serial = []
    for call in calls:
        queue = call()
        serial.append((queue.indices.clone(), queue.distances.clone()))
    torch.cuda.synchronize()
    got = [[] for _ in calls]
    gate = threading.Barrier(len(calls))

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(passes):
                gate.wait(60)
                try:
                    torch.cuda._sleep(20_000_000)
                    queue = calls[i]()
                    got[i].append((queue.indices.clone(), queue.distances.clone()))
                    torch.cuda.current_stream().synchronize()
                except Exception as e:      # the other threads still meet this one at the gate
                    got[i].append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    return serial, got


def assert_threads_change_nothing(calls, passes=10):
    (serial, got) = serial_and_threaded(calls, passes)
    for (want, passes_of_one) in zip(serial, got):
        for one in passes_of_one:
            assert not isinstance(one, Exception), one
            assert torch.equal(one[0], want[0]) and torch.equal(one[1], want[1])


@pytest.mark.parametrize("count", [1300, 2000])     # memos in global memory, and room on the chip for both launches
def test_searches_of_two_streams_share_no_memo(count, built_lib):
    from vectorlink_gpu import ANN
    index = ANN(vectors=unit_rows(1, 3000, 128), beam_size=16, visit_queue_factor=2, recall_search_queue_factor=2,
                init="knn_tile", optimization_loops=1)
    (a, b) = (unit_rows(2, count, 128), unit_rows(3, count, 128))
    assert_threads_change_nothing([lambda: index.search(a), lambda: index.search(b)])


@pytest.mark.parametrize("metric", ["cosine", "l2"])
def test_entry_points_of_two_streams_are_their_own(metric, built_lib):
    from vectorlink_gpu import ANN
    index = ANN(vectors=unit_rows(1, 20_000, 128), beam_size=16, visit_queue_factor=2, recall_search_queue_factor=2,
                metric=metric, init="knn_tile", optimization_loops=1, search_entry_sample=16_384)
    (a, b) = (unit_rows(2, 500, 128), unit_rows(3, 700, 128))
    assert_threads_change_nothing([lambda: index.search(a), lambda: index.search(b)], passes=30)


def test_the_entry_sample_is_complete_before_another_stream_meets_it(built_lib):
    """The first search of an index makes the sample on a stream that is busy; a search on another stream, started right
    after the sample is there, must not read it half made.  (Both streams have met another index first: their memory is
    allocated, which the device would be waited for, and holds other rows.)"""
    from vectorlink_gpu import ANN
    def index_of(seed):
        vectors = unit_rows(seed, 20_000, 128)
        return ANN(vectors=vectors, beams=torch.zeros((20_000, 16), dtype=torch.int32, device=DEV), beam_size=16,
                   search_entry_sample=16_384)

    queries = unit_rows(2, 500, 128)
    (other, index) = (index_of(4), index_of(1))
    want = index._entry_seeds(queries)
    index._entry = None
    (first, second) = (torch.cuda.Stream(), torch.cuda.Stream())
    for stream in (first, second):
        with torch.cuda.stream(stream):
            other._entry = None
            other._entry_seeds(queries)
            stream.synchronize()
    other._entry = None
    torch.cuda.synchronize()
    with torch.cuda.stream(first):
        torch.cuda._sleep(200_000_000)
        index._entry_seeds(queries)
    with torch.cuda.stream(second):
        got = index._entry_seeds(queries)
    torch.cuda.synchronize()
    assert torch.equal(got, want)


def test_a_plan_of_another_thread_does_not_refuse_a_launch(built_lib):
    """One kernel, rows of two sizes: a thread that plans launches of small rows must not take the shared memory from under
    the launches of another thread, whose rows need more than the 48 KB that every kernel may have."""
    import ctypes
    from vectorlink_gpu import ANN
    from vectorlink_gpu._lib import BeamParams, lib
    vectors = unit_rows(1, 20_000, 128)
    index = ANN(vectors=vectors, beam_size=32, visit_queue_factor=25, recall_search_queue_factor=4, init="knn_tile",
                optimization_loops=0)
    index.configuration["memo"] = False
    queries = unit_rows(2, 1200, 128)
    want = index.search(queries).indices.clone()
    some = vectors.data_ptr()           # a plan reads no memory
    small = BeamParams(vectors=some, n=20_000, dim=128, graph=some, graph_w=16, pvc=4, queries=some, rows=1200, seed_ids=some,
                       seed_dist=some, seed_ld=32, seed_cols=32, sq_len=32, vq_len=32, seen_cap=160, out_ids=some, out_dist=some,
                       out_ld=32, out_cols=32, n_iters=45, readahead=5, self_base=-1, changed_flags=some, group_full=some, status=some)
    (size, per_block, blocks) = (ctypes.c_int(), ctypes.c_int(), ctypes.c_int())
    stop = threading.Event()
    refused = []

    def plan():
        while not stop.is_set():
            if lib().vl_beam_search_plan(ctypes.byref(small), ctypes.byref(size), ctypes.byref(per_block), ctypes.byref(blocks)):
                refused.append(lib().vl_last_error())

    planner = threading.Thread(target=plan)
    planner.start()
    try:
        for _ in range(60):
            assert torch.equal(index.search(queries).indices, want)
    finally:
        stop.set()
        planner.join()
    assert not refused and blocks.value > 0


def test_the_seed_table_outlives_its_place_in_the_cache(built_lib):
    """A table that leaves the cache while another stream has yet to read it: its memory is not given to anyone before."""
    from vectorlink_gpu import utils
    utils._sorted_primes.cache_clear()
    want = utils.seed_offsets(700, DEV).clone()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(400_000_000)
        table = utils.seed_offsets(700, DEV)
        at = table.data_ptr()
        read = table + 0
    del table
    utils._sorted_primes.cache_clear()
    others = [torch.full((700,), -1, dtype=torch.int32, device=DEV) for _ in range(3000)]
    early = not side.query()                 # all of them were made while the other stream had still to read
    torch.cuda.synchronize()
    assert torch.equal(read, want)
    assert not early or all(o.data_ptr() != at for o in others)


def test_the_status_word_is_zero_before_another_stream_sets_a_bit(built_lib):
    from vectorlink_gpu import _lib
    from vectorlink_gpu.kernels import calculate_distances
    vectors = unit_rows(1, 10, 64)
    bad = torch.full((10, 1), 99, dtype=torch.int32, device=DEV)      # no such row: skipped and reported
    calculate_distances(vectors, bad)
    assert _lib.read_status(DEV) == 1
    torch.cuda.synchronize()
    _lib._status.clear()
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda._sleep(200_000_000)
        _lib.status_word(DEV)
    with torch.cuda.stream(torch.cuda.Stream()):
        calculate_distances(vectors, bad)
    torch.cuda.synchronize()
    assert _lib.read_status(DEV) == 1
