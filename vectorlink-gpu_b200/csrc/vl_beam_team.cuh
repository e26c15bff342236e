// The fused beam search with the warps of a CTA sharing one query row.
//
// An iteration of a row is: neighbour ids and memo probes, the gather of the candidates the memo does not
// know, the choice of those that can enter a queue - each split over all warps - and then the two
// queue steps, side by side where there are warps for it (the search queue's on warp 0, the visit queue's
// on warp 1).
#pragma once
#include "vl_beam.cuh"

namespace {

constexpr int kMaxTeam = 16;                                   // most warps per row
// CTAs per SM that launches of many rows aim for: teams of one warp (96 registers) or two (64)
constexpr int many_per_sm(int team) { return team == 1 ? 20 : 16; }
constexpr unsigned long long kWaitLimitNs = 2000000000ull;     // 2 s per wait, unless the caller asks for another limit

struct TeamSmem {      // carve-up of the CTA's shared memory, in bytes
    int memo, query, cand, sq_a, sq_b, vq_a, vq_b, hash, todo, list_s, list_v, ctl, total;
    int hash_slots, hash_shift, memo_buckets, memo_shift;
};

// memo_entries: entries of the row's distance memo, 0 = none; on_chip: they are in shared memory; lists: space for the
// lists of entrants (a single warp makes them one after the other in the place of `todo`)
__host__ inline TeamSmem team_layout(int m, int sq_len, int vq_len, int seen_cap, int query_bytes, int memo_entries, bool on_chip,
                                     bool lists)
{
    TeamSmem s;
    int off = 0;
    s.memo_buckets = memo_entries / 2;
    s.memo_shift = 32;
    for (int b = s.memo_buckets; b > 1; b >>= 1) --s.memo_shift;
    s.memo = off; off += on_chip ? 8 * memo_entries : 0;       // first: 16-byte aligned buckets
    s.query = off; off += query_bytes;
    s.cand = off; off += 8 * m;
    s.sq_a = off; off += 8 * sq_len;
    s.sq_b = off; off += 8 * sq_len;
    s.vq_a = off; off += 8 * vq_len;
    s.vq_b = off; off += 8 * vq_len;
    int slots = 32, shift = 27;
    while (slots < seen_cap + seen_cap / 2 + 1) { slots <<= 1; --shift; }
    s.hash_slots = slots;
    s.hash_shift = shift;
    s.hash = off; off += 4 * slots;
    s.ctl = off; off += 4 * 16;
    s.todo = off; off += 2 * m;
    s.list_s = lists ? off : s.todo; off += lists ? 2 * m : 0;
    s.list_v = lists ? off : s.todo; off += lists ? 2 * m : 0;
    s.total = (off + 15) & ~15;
    return s;
}

// words of the control block: list lengths, real keys of the visit and the search queue, the end of the
// batch, which buffer holds each queue, the cycle counters (the clock at the last phase of warp 0 and of the visit
// queue's warp, then a sum per phase), and between two rows the next row
enum { kTodo = 0, kListS, kListV, kQueued, kHeld, kStop, kSqBuf, kVqBuf, kClock, kClockV, kPop, kProbe, kGather, kSearchQ, kVisitQ, kWords,
       kRowLo = kTodo, kRowHi = kListS };
static_assert(kWords <= 16, "control block");

__device__ __forceinline__ unsigned long long team_now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// appends `c` of the lanes flagged `take` to list[*count ..]; the order within the list is free
__device__ __forceinline__ void team_append(unsigned short* list, int* count, bool take, int c, int lane)
{
    const unsigned mask = __ballot_sync(0xffffffffu, take);
    if (!mask) return;
    int at = 0;
    if (lane == 0) at = atomicAdd(count, __popc(mask));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (take) list[at + __popc(mask & ((1u << lane) - 1u))] = (unsigned short)c;
}

__device__ __forceinline__ bool team_excluded(const int32_t* excl, int e, int32_t id)
{
#pragma unroll 1
    for (int x = 0; x < e; ++x) {     // kernels.py:478-488
        const int32_t ex = excl[x];
        if (ex == VL_MAXINT) return false;
        if (ex == id) return true;
    }
    return false;
}

// One step of a sorted queue of at most `len` distinct keys: the first `skip` keys of `cur` leave, the keys of
// the lanes flagged `want` enter unless they are present, and the `len` smallest go to `nxt`, sentinels
// behind them.  `n`: real keys of `cur` behind the skipped ones.  Returns the real keys of `nxt`.
// A key's place is its lower bound in `cur` plus its rank among the entering keys; a kept key moves up
// by the entering keys placed before it.  Most offered keys are present already, so the usual call
// has a handful of entering keys: a branchless search by all lanes at once, one broadcast per entering
// key and four kept keys per lane in registers make up its latency, which is what bounds the search (the
// queue steps are a serial chain).  All 32 lanes call this; both buffers are this warp's alone.
__device__ __noinline__ int queue_step(const vl_key_t* cur, vl_key_t* nxt, int len, int skip, int n, vl_key_t key, bool want, int lane)
{
    const vl_key_t* list = cur + skip;
    int lo = 0;                                   // list keys below key
    if (n > 0) {
        for (int s = 1 << (31 - __clz(n)); s > 0; s >>= 1) {
            const int m = lo + s;
            const vl_key_t e = list[(m <= n ? m : n) - 1];
            if (m <= n && e < key) lo = m;
        }
        if (lo < n && list[lo] == key) want = false;
    }
    unsigned mask = __ballot_sync(0xffffffffu, want);
    int rank = 0;
    bool repeat = false;
    for (unsigned m = mask; m; m &= m - 1) {
        const int src = __ffs(m) - 1;
        const vl_key_t o = __shfl_sync(0xffffffffu, key, src);
        rank += o < key;
        repeat |= o == key && src < lane;
    }
    const unsigned again = __ballot_sync(0xffffffffu, want && repeat);
    if (again) {                                  // the same candidate twice in one iteration: keep the first
        mask &= ~again;
        want = want && !repeat;
        rank = 0;
        for (unsigned m = mask; m; m &= m - 1) rank += __shfl_sync(0xffffffffu, key, __ffs(m) - 1) < key;
    }
    for (int jb = 0; jb < n; jb += 128) {
        vl_key_t e[4];
        int at[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            at[u] = jb + 32 * u + lane;
            e[u] = at[u] < n ? list[at[u]] : 0ull;
        }
        int up[4] = {0, 0, 0, 0};
        for (unsigned m = mask; m; m &= m - 1) {
            const int pos = __shfl_sync(0xffffffffu, lo, __ffs(m) - 1);
#pragma unroll
            for (int u = 0; u < 4; ++u) up[u] += pos <= at[u];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (at[u] < n && at[u] + up[u] < len) nxt[at[u] + up[u]] = e[u];
    }
    if (want && lo + rank < len) nxt[lo + rank] = key;
    const int total = n + __popc(mask);
    for (int j = total + lane; j < len; j += 32) nxt[j] = vl_sentinel_key();
    __syncwarp();
    return total < len ? total : len;
}

// Distance of the loaded row against the query in shared memory (zero-padded to LPR * JP chunks).
template <int LPR, int JP, int METRIC, bool ALIGNED>
__device__ __forceinline__ float team_row_distance(float4 (&x)[JP], const float4* q4, const float* row, const float* qfull,
                                                   int dim, int lg, bool live)
{
#pragma unroll
    for (int j = 0; j < JP; ++j) x[j] = vl_term4<METRIC>(x[j], q4[LPR * j]);
    if (dim > 1024) {  // kernels.py:43-47: fold element 1024k+t onto t, k rising
        const int nchunks = (dim + 3) >> 2;
#pragma unroll 1
        for (int k = 1; 256 * k < nchunks; ++k) {
#pragma unroll
            for (int j = 0; j < JP; ++j) {
                const int c = 256 * k + lg + LPR * j;
                if (live && c < nchunks && lg + LPR * j < 256)
                    x[j] = vl_add4(x[j], vl_term4<METRIC>(vl_load_chunk<ALIGNED>(row, c, dim), vl_load_chunk<ALIGNED>(qfull, c, dim)));
            }
        }
    }
    return vl_finish<METRIC>(vl_tree_reduce<LPR, JP>(x));
}

// Distances of the candidates listed in todo[0, n): G rows per warp and step, U steps in flight.
template <int LPR, int JP, int JU, int METRIC, bool ALIGNED, int TEAM>
__device__ __forceinline__ void team_gather(const vl_beam_params& p, uint2* cand, const unsigned short* todo, int n,
                                            const float4* q4, const float* q, int warp, int nwarps, int lane, uint64_t pol,
                                            vl_key_t* memo, int memo_buckets, int memo_shift, int way)
{
    constexpr int G = 32 / LPR;
    constexpr int JX = JU > 0 ? JU : JP;
    constexpr int U = TEAM == 1 ? (JX <= 4 ? 2 : 1) : TEAM == 2 ? 1 : (JU > 0 ? (JX <= 4 ? 4 : 2) : 1);
    const int g = lane / LPR, lg = lane % LPR;
#pragma unroll 1
    for (int t0 = warp * G; t0 < n; t0 += nwarps * U * G) {
        bool live[U];
        int mi[U];
        const float* rp[U];
        float dd[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int t = t0 + u * nwarps * G + g;
            live[u] = t < n;
            mi[u] = live[u] ? todo[t] : 0;
            const int32_t id = live[u] ? (int32_t)cand[mi[u]].x : 0;
            rp[u] = p.vectors + (int64_t)id * p.dim;
        }
        if constexpr (JU > 0 && TEAM <= 2) {
            // pull the next round of candidate rows into L1 while this one is reduced
            constexpr int LINES = (4 * LPR * JU * 4) / 128;          // 128-byte lines per row
            const int tn = t0 + nwarps * U * G;
#pragma unroll
            for (int l0 = 0; l0 < U * G * LINES; l0 += 32) {
                const int l = l0 + lane;
                const int t = tn + (l / LINES / G) * nwarps * G + (l / LINES) % G;
                if (l < U * G * LINES && t < n) {
                    const int32_t nid = (int32_t)cand[todo[t]].x;
                    asm volatile("prefetch.global.L1 [%0];" : : "l"(p.vectors + (int64_t)nid * p.dim + (l % LINES) * 32));
                }
            }
        }
        if constexpr (JU > 0) {
            float4 x[U][JU];
#pragma unroll
            for (int u = 0; u < U; ++u) vl_load_exact_hint<LPR, JU>(rp[u], lg, x[u], pol);
#pragma unroll
            for (int u = 0; u < U; ++u) dd[u] = vl_exact_distance_q<LPR, JP, JU, METRIC>(x[u], q4 + lg);
        } else {
            float4 x[U][JP];
#pragma unroll
            for (int u = 0; u < U; ++u) vl_load_row<LPR, JP, ALIGNED>(rp[u], p.dim, lg, live[u], x[u]);
#pragma unroll
            for (int u = 0; u < U; ++u) dd[u] = team_row_distance<LPR, JP, METRIC, ALIGNED>(x[u], q4 + lg, rp[u], q, p.dim, lg, live[u]);
        }
        if (lg == 0) {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (live[u]) {
                    const uint32_t ord = vl_ord(dd[u]);
                    cand[mi[u]].y = ord;
                    if (memo) memo_put(memo, memo_buckets, memo_shift, ((vl_key_t)ord << 32) | cand[mi[u]].x, way);   // remember it
                }
        }
    }
}

// TEAM <= 2: launches of many rows, many_per_sm(TEAM) CTAs per SM, the memo in global memory (L2).
// TEAM == kMaxTeam: launches of few rows, 2 to 16 warps per CTA (blockDim), the memo in shared memory.
// JU > 0: exact-fit rows (dim == 4*LPR*JU, see vl_load_exact); JU == 0: any dimension, with 128-bit
// loads when ALIGNED (dim % 4 == 0 and 16-byte aligned rows) and four scalar loads per chunk otherwise.
// TIMED: with the cycle counters of `stats` (vl_beam_timed.cu).  A test of the launch's flags at every phase instead costs
// launches without counters too: clusters of 30,000 x 96 9.16 / 9.44 ms, rounds 2 and 3 of 150,000 x 128 76, 78 / 82, 84.
template <int LPR, int JP, int JU, int METRIC, bool ALIGNED, int TEAM, bool TIMED = false>
__global__ void __launch_bounds__(TEAM * 32, TEAM <= 2 ? many_per_sm(TEAM) : 1)
beam_team_kernel(const vl_beam_params p, const TeamSmem lay, const int64_t* __restrict__ row_order, unsigned int* arrivals)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, threads = TEAM <= 2 ? TEAM * 32 : blockDim.x, nwarps = threads >> 5;
    vl_key_t* memo = TEAM <= 2 ? (p.memo ? p.memo + (size_t)blockIdx.x * (size_t)p.memo_entries : nullptr)
                               : reinterpret_cast<vl_key_t*>(smem + lay.memo);
    float4* q4 = reinterpret_cast<float4*>(smem + lay.query);
    uint2* cand = reinterpret_cast<uint2*>(smem + lay.cand);
    vl_key_t* candk = reinterpret_cast<vl_key_t*>(smem + lay.cand);
    int32_t* hash = reinterpret_cast<int32_t*>(smem + lay.hash);
    unsigned short* todo = reinterpret_cast<unsigned short*>(smem + lay.todo);
    unsigned short* list_s = reinterpret_cast<unsigned short*>(smem + lay.list_s);
    unsigned short* list_v = reinterpret_cast<unsigned short*>(smem + lay.list_v);
    int* ctl_count = reinterpret_cast<int*>(smem + lay.ctl);
    volatile int* ctl = ctl_count;

    const int wb = p.graph_w, pvc = p.pvc, m_total = pvc * wb;
    const int sq_len = p.sq_len, vq_len = p.vq_len, e_cap = p.seen_cap;
    const int k_none = (e_cap + pvc - 1) / pvc + 1;   // first iteration at which `seen` is full
    const int n_run = p.n_iters < k_none ? p.n_iters : k_none;
    const vl_key_t kSent = vl_sentinel_key();
    const uint32_t kPoppedOrd = 0xffffffffu;          // "popped" mark of a memo entry, above every real ordered distance
    const float inv_wb = 1.0f / (float)wb;
    // TIMED: lane 0 of a warp adds the cycles since its last call to a phase (`sum`; kTodo = none, start only).
    auto phase = [&](int since, int sum) {
        if constexpr (TIMED) {
            if (lane == 0) {
                unsigned int now;
                asm volatile("mov.u32 %0, %%clock;" : "=r"(now) : : "memory");
                if (sum != kTodo) ctl[sum] = (int)((unsigned int)ctl[sum] + now - (unsigned int)ctl[since]);
                ctl[since] = (int)now;
            }
        }
    };
    // With a memo a candidate row is read about once per query row: unless rows are taken neighbourhood by
    // neighbourhood, stream it through L2 and keep the graph rows and the memo there instead.
    const uint64_t pol_stream = (TEAM <= 2 && p.memo && !row_order) ? vl_policy_evict_first() : vl_policy_evict_normal();
    const uint64_t pol_keep = (TEAM <= 2 && p.memo) ? vl_policy_evict_last() : vl_policy_evict_normal();

    // Row schedule: the first row of a CTA is fixed; after that either a fixed stride or, when the caller
    // provides a zeroed counter, the next row nobody has taken yet (rows take unequal time).  `place`
    // counts rows in the order they are taken: by row number, or through `row_order`.
    int64_t place = blockIdx.x;
#pragma unroll 1
    while (place < p.rows) {
        const int64_t row = row_order ? row_order[place] : place;
        const float* q = p.queries + row * (int64_t)p.dim;
        vl_key_t* sq = reinterpret_cast<vl_key_t*>(smem + lay.sq_a);
        vl_key_t* vq = reinterpret_cast<vl_key_t*>(smem + lay.vq_a);

        // ---- prologue: Queue.insert of the seeds into an empty queue (queue.py:37-61) ----
        for (int c = tid; c < LPR * JP; c += threads)
            q4[c] = 4 * c < p.dim ? vl_load_chunk<ALIGNED>(q, c, p.dim) : make_float4(0.f, 0.f, 0.f, 0.f);
        for (int i = tid; i < sq_len; i += threads) sq[i] = kSent;
        for (int i = tid; i < lay.hash_slots; i += threads) hash[i] = kHashEmpty;
        if (memo)
            for (int i = tid; i < lay.memo_buckets; i += threads)
                reinterpret_cast<ulonglong2*>(memo)[i] = make_ulonglong2(~0ull, ~0ull);
        if (tid < kWords) ctl[tid] = 0;
        __syncthreads();
        // The ids that iteration `k` pops are visited from then on (utils.py:61-82): they can never enter the
        // visit queue again, and the search queue only looks at newly gathered ids, so their memo entries
        // only have to say "popped".  Both ways of the bucket are overwritten without a read: losing the
        // other one costs a gather if that id comes back.
        auto mark_popped = [&](const vl_key_t* queue, int k) {
            const int first = (k - 1) * pvc;
            const int ncopy = first < e_cap ? ((e_cap - first) < pvc ? (e_cap - first) : pvc) : 0;
            if (lane < ncopy) {
                const int32_t node = vl_key_id(queue[lane]);
                if (node >= 0 && (int64_t)node < p.n) {
                    hash_insert(hash, lay.hash_slots, lay.hash_shift, node, p.status);
                    if (memo) {
                        const vl_key_t mark = ((vl_key_t)kPoppedOrd << 32) | (uint32_t)node;
                        reinterpret_cast<ulonglong2*>(memo)[memo_bucket((uint32_t)node, lay.memo_shift, lay.memo_buckets)] =
                            make_ulonglong2(mark, mark);
                    }
                }
            }
        };
        if (warp == 0) {
            vl_key_t* sq_n = reinterpret_cast<vl_key_t*>(smem + lay.sq_b);
            int held = 0;
#pragma unroll 1
            for (int c0 = 0; c0 < p.seed_cols; c0 += 32) {
                const int c = c0 + lane;
                vl_key_t key = kSent;
                if (c < p.seed_cols)
                    key = vl_entry_key(__ldg(p.seed_dist + row * p.seed_ld + c), __ldg(p.seed_ids + row * p.seed_ld + c));
                if (memo && key != kSent) memo_put(memo, lay.memo_buckets, lay.memo_shift, key, 0);   // a seed's distance is known
                const bool want = key < sq[sq_len - 1];
                if (__any_sync(0xffffffffu, want)) {
                    held = queue_step(sq, sq_n, sq_len, 0, held, key, want, lane);
                    vl_key_t* t = sq; sq = sq_n; sq_n = t;
                }
            }
            // visit_queue.initialize_from_queue (queue.py:30-35)
            const int head = sq_len < vq_len ? sq_len : vq_len;
#pragma unroll 1
            for (int i = lane; i < vq_len; i += 32) vq[i] = i < head ? sq[i] : kSent;
            __syncwarp();
            mark_popped(vq, 1);
            if (lane == 0) {
                ctl[kQueued] = held < head ? held : head;
                ctl[kHeld] = held;
                ctl[kSqBuf] = sq == reinterpret_cast<vl_key_t*>(smem + lay.sq_a) ? lay.sq_a : lay.sq_b;
                ctl[kVqBuf] = lay.vq_a;
            }
        }
        __syncthreads();

        const int32_t self_id = p.self_base >= 0 ? (int32_t)(p.self_base + row) : VL_MAXINT;
        const int32_t* excl = p.exclude_w > 0 ? p.exclude + row * (int64_t)p.exclude_w : nullptr;
        const int64_t group = p.group_rows > 0 ? (p.group_row0 + row) / p.group_rows : 0;
        bool always_full = true, dumped = false, waits = true;
        unsigned int st_todo = 0, st_m = 0, st_v = 0, st_a = 0, st_b = 0;
        int k = 1;

#pragma unroll 1
        for (; k <= n_run; ++k) {
            if (warp == 0) phase(kClock, kTodo);
            const int first = (k - 1) * pvc;
            const bool seen_live = first < e_cap;    // utils.py:62-69
            const bool raw = p.dump_last && k == p.n_iters;   // needs every real distance
            sq = reinterpret_cast<vl_key_t*>(smem + ctl[kSqBuf]);
            vq = reinterpret_cast<vl_key_t*>(smem + ctl[kVqBuf]);
            // ---- pop_n_ids (queue.py:87-95): the heads are read in place, warp 1's queue step drops them ----
            const int queued = ctl[kQueued];          // real keys in the visit queue before the pop
            const int n_old = queued > pvc ? queued - pvc : 0;
            int32_t popped = VL_MAXINT;               // lane v < pvc: the v-th popped id
            if (lane < pvc) {
                popped = vl_key_id(vq[lane]);
                if (popped != VL_MAXINT && (popped < 0 || (int64_t)popped >= p.n)) {
                    if (warp == 0) atomicOr(p.status, VL_STATUS_BAD_ID);
                    popped = VL_MAXINT;
                }
            }
            const int ncopy = seen_live ? ((e_cap - first) < pvc ? (e_cap - first) : pvc) : 0;
            if (__any_sync(0xffffffffu, lane < ncopy && popped == VL_MAXINT)) always_full = false;
            if (warp == 0) phase(kClock, kPop);
            // ---- neighbour ids (kernels.py:244), then which of them need a gather: live ids the memo does not know.
            // PB chunks per warp and round: the graph-row loads, then the memo loads, of a round are in flight together.
            constexpr int PB = TEAM <= 2 ? 6 : 4;
#pragma unroll 1
            for (int cb = warp * 32; cb < m_total; cb += threads * PB) {
                int32_t idr[PB];
#pragma unroll
                for (int u = 0; u < PB; ++u) {
                    const int c = cb + u * threads + lane;
                    const int v = __float2int_rz(((float)c + 0.5f) * inv_wb);
                    const int32_t node = __shfl_sync(0xffffffffu, popped, v & 31);
                    idr[u] = (c < m_total && node != VL_MAXINT) ? vl_ldg_hint(p.graph + (int64_t)node * wb + (c - v * wb), pol_keep) : VL_MAXINT;
                }
                ulonglong2 bk[PB];
#pragma unroll
                for (int u = 0; u < PB; ++u) {
                    if (idr[u] != VL_MAXINT && (idr[u] < 0 || (int64_t)idr[u] >= p.n)) {
                        atomicOr(p.status, VL_STATUS_BAD_ID);
                        idr[u] = VL_MAXINT;
                    }
                    bk[u] = make_ulonglong2(~0ull, ~0ull);
                    if (memo && idr[u] != VL_MAXINT) {
                        const ulonglong2* at = reinterpret_cast<const ulonglong2*>(memo) + memo_bucket((uint32_t)idr[u], lay.memo_shift, lay.memo_buckets);
                        if constexpr (TEAM <= 2) bk[u] = vl_ld_hint(at, pol_keep);
                        else bk[u] = *at;
                    }
                }
#pragma unroll
                for (int u = 0; u < PB; ++u) {
                    if (cb + u * threads >= m_total) break;      // the same for the whole warp
                    const int c = cb + u * threads + lane;
                    const uint32_t id = (uint32_t)idr[u];
                    bool need = (idr[u] != VL_MAXINT);
                    uint32_t ord = (uint32_t)(kSent >> 32);
                    if (need) {
                        if ((uint32_t)bk[u].x == id) { ord = (uint32_t)(bk[u].x >> 32); need = false; }
                        else if ((uint32_t)bk[u].y == id) { ord = (uint32_t)(bk[u].y >> 32); need = false; }
                        if (raw && ord == kPoppedOrd) need = true;
                    }
                    if (c < m_total) cand[c] = make_uint2(id, ord);
                    team_append(todo, ctl_count + kTodo, need, c, lane);
                }
            }
            __syncthreads();
            if (warp == 0) phase(kClock, kProbe);
            // ---- gathered distances (kernels.py:248-257) ----
            const int n_todo = ctl[kTodo];
            st_todo += n_todo;
            team_gather<LPR, JP, JU, METRIC, ALIGNED, TEAM>(p, cand, todo, n_todo, q4, q, warp, nwarps, lane, pol_stream, memo,
                                                            lay.memo_buckets, lay.memo_shift, k & 1);
            __syncthreads();
            if (warp == 0) phase(kClock, kGather);
            if (raw) { dumped = true; break; }
            // ---- which candidates can enter a queue: every warp looks at its share ----
            // Search queue: only candidates gathered now (a candidate the memo knew was offered when it was first
            // gathered, and the cut-off only falls).  Visit queue: every unvisited candidate below its largest kept
            // key (class A); the popped entries left free slots, and if class A does not fill them the smallest
            // unvisited candidates above it do (class B).  Same queue as offering every candidate.
            const vl_key_t cut = sq[sq_len - 1];
            const bool usual = seen_live && n_old > 0 && vq_len - n_old <= 8;
            const vl_key_t t0key = n_old > 0 ? vq[n_old - 1 + pvc] : kSent;
            int n_entrants = 0;                       // of the search queue, in list_s (one warp per row)
#pragma unroll 1
            for (int t0 = warp * 32; t0 < n_todo; t0 += threads) {
                const int t = t0 + lane;
                const int c = t < n_todo ? todo[t] : 0;
                const vl_key_t key = t < n_todo ? candk[c] : kSent;
                bool want = key < cut;
                if (want) {
                    const int32_t id = vl_key_id(key);
                    if (id == self_id || (excl && team_excluded(excl, p.exclude_w, id))) want = false;
                }
                if constexpr (TEAM == 1) {            // list_s is todo: never ahead of the reads, which this ballot waits for
                    const unsigned mask = __ballot_sync(0xffffffffu, want);
                    if (want) list_s[n_entrants + __popc(mask & ((1u << lane) - 1u))] = (unsigned short)c;
                    n_entrants += __popc(mask);
                } else {
                    team_append(list_s, ctl_count + kListS, want, c, lane);
                }
            }
            if (TEAM > 1 && usual) {
#pragma unroll 1
                for (int c0 = warp * 32; c0 < m_total; c0 += threads) {
                    const int c = c0 + lane;
                    const bool in_a = c < m_total && candk[c] < t0key;
                    team_append(list_v, ctl_count + kListV, in_a, c, lane);
                }
            }
            __syncthreads();
            if (warp == 0) {
                // ---- search_queue.insert(..., exclude) (ann.py:75-80) ----
                bool changed = false;
                const int n_in = TEAM == 1 ? n_entrants : ctl[kListS];
                int held = ctl[kHeld];
                if (n_in) {
                    vl_key_t* sq_n = reinterpret_cast<vl_key_t*>(smem + (lay.sq_a + lay.sq_b - ctl[kSqBuf]));
                    vl_key_t now = cut;
#pragma unroll 1
                    for (int t0 = 0; t0 < n_in; t0 += 32) {
                        const int t = t0 + lane;
                        const vl_key_t key = t < n_in ? candk[list_s[t]] : kSent;
                        const bool want = key < now;
                        if (!__any_sync(0xffffffffu, want)) continue;
                        // a new key is below the last one: the queue grows, or its last key leaves
                        const vl_key_t tail = sq[sq_len - 1];
                        const int before = held;
                        held = queue_step(sq, sq_n, sq_len, 0, held, key, want, lane);
                        vl_key_t* u = sq; sq = sq_n; sq_n = u;
                        now = sq[sq_len - 1];
                        changed |= held != before || now != tail;
                        st_m += 1;
                    }
                }
                __syncwarp();
                phase(kClock, kSearchQ);
                if (lane == 0) {
                    ctl[kTodo] = 0;
                    ctl[kListS] = 0;
                    ctl[kHeld] = held;
                    ctl[kSqBuf] = sq == reinterpret_cast<vl_key_t*>(smem + lay.sq_a) ? lay.sq_a : lay.sq_b;
                    const int chk = k / p.readahead - 1;
                    if ((k % p.readahead) == 0 && chk < p.n_checks) {
                        unsigned int* flag = p.changed_flags + group * p.n_checks + chk;
                        if (changed) atomicOr(flag, 1u);
                        if (TEAM > 2 && arrivals) {
                            __threadfence();
                            atomicAdd(arrivals + chk, 1u);
                            if (!changed && waits) {
                                const unsigned long long t0 = team_now_ns(), limit = p.wait_us > 0 ? p.wait_us * 1000ull : kWaitLimitNs;
                                for (;;) {
                                    // all rows have reported, and none of them a change (a row's flag precedes its arrival)
                                    if (*(volatile unsigned int*)(arrivals + chk) >= (unsigned int)p.rows) {
                                        __threadfence();
                                        ctl[kStop] = *(volatile unsigned int*)flag == 0 ? 1 : 0;
                                        break;
                                    }
                                    if (*(volatile unsigned int*)flag != 0) break;
                                    if (team_now_ns() - t0 > limit) {
                                        atomicOr(p.status, VL_STATUS_TIMEOUT);
                                        atomicOr(flag, 1u);
                                        waits = false;
                                        break;
                                    }
                                    __nanosleep(64);
                                }
                            }
                        }
                    }
                }
            }
            if (warp == (TEAM == 1 ? 0 : 1)) {
                // ---- the popped heads leave, visit_queue.insert(..., exclude=seen) ----
                phase(kClockV, kTodo);
                if (TEAM == 1 && usual) {
#pragma unroll 1
                    for (int c0 = 0; c0 < m_total; c0 += 32)
                        team_append(list_v, ctl_count + kListV, c0 + lane < m_total && candk[c0 + lane] < t0key, c0 + lane, lane);
                    __syncwarp();
                }
                vl_key_t* vq_n = reinterpret_cast<vl_key_t*>(smem + (lay.vq_a + lay.vq_b - ctl[kVqBuf]));
                const int n_a = usual ? ctl[kListV] : (seen_live ? m_total : 0);   // an (almost) empty queue is offered every candidate
                st_a += usual ? n_a : 0;
                int n_real = n_old, skip = pvc;
                int t0 = 0;
#pragma unroll 1
                do {
                    const int t = t0 + lane;
                    vl_key_t key = kSent;
                    if (t < n_a) key = candk[usual ? list_v[t] : t];
                    bool want = key < kSent && (skip || n_real < vq_len || key < vq[vq_len - 1]);
                    if (want && hash_contains(hash, lay.hash_slots, lay.hash_shift, vl_key_id(key))) want = false;
                    if (skip || __any_sync(0xffffffffu, want)) {
                        n_real = queue_step(vq, vq_n, vq_len, skip, n_real, key, want, lane);
                        { vl_key_t* u = vq; vq = vq_n; vq_n = u; }
                        skip = 0;
                        st_v += 1;
                    }
                    t0 += 32;
                } while (t0 < n_a);
                if (usual) {
                    vl_key_t last = t0key;
#pragma unroll 1
                    while (n_real < vq_len) {
                        st_b += 1;
                        vl_key_t best = ~0ull;
#pragma unroll 1
                        for (int c = lane; c < m_total; c += 32) {
                            const vl_key_t kk = candk[c];
                            if (kk > last && kk < kSent && kk < best) best = kk;
                        }
                        const uint32_t hi = __reduce_min_sync(0xffffffffu, (uint32_t)(best >> 32));
                        if (hi == 0xffffffffu) break;
                        const uint32_t id = __reduce_min_sync(0xffffffffu, (uint32_t)(best >> 32) == hi ? (uint32_t)best : 0xffffffffu);
                        best = ((vl_key_t)hi << 32) | id;
                        last = best;
                        if (hash_contains(hash, lay.hash_slots, lay.hash_shift, vl_key_id(best))) continue;
                        if (lane == 0) vq[n_real] = best;
                        ++n_real;
                        st_v += 1;
                    }
                }
                __syncwarp();
                if (lane == 0) {
                    ctl[kListV] = 0;
                    ctl[kQueued] = n_real;
                    ctl[kVqBuf] = vq == reinterpret_cast<vl_key_t*>(smem + lay.vq_a) ? lay.vq_a : lay.vq_b;
                }
                mark_popped(vq, k + 1);
                phase(kClockV, kVisitQ);
            }
            __syncthreads();
            if (TEAM > 2 && ctl[kStop] != 0) {
                // The batch ends here: this iteration's insert is left to the caller's full-row sort, which
                // wants every candidate's distance; those of visited ids are taken again.
#pragma unroll 1
                for (int c0 = warp * 32; c0 < m_total; c0 += threads) {
                    const int c = c0 + lane;
                    team_append(todo, ctl_count + kTodo, c < m_total && cand[c].y == kPoppedOrd, c, lane);
                }
                __syncthreads();
                team_gather<LPR, JP, JU, METRIC, ALIGNED, TEAM>(p, cand, todo, ctl[kTodo], q4, q, warp, nwarps, lane, pol_stream,
                                                                memo, lay.memo_buckets, lay.memo_shift, 0);
                __syncthreads();
                dumped = true;
                if (tid == 0 && row == 0) arrivals[p.n_checks] = (unsigned int)k;
                break;
            }
        }

        // ---- results: the head, then sentinels, or the raw candidates of the last iteration ----
        sq = reinterpret_cast<vl_key_t*>(smem + ctl[kSqBuf]);
#pragma unroll 1
        for (int i = tid; i < p.out_cols; i += threads) {
            vl_key_t key = kSent;
            if (i < sq_len) key = sq[i];
            else if (dumped && i < sq_len + m_total) {
                key = candk[i - sq_len];
                const int32_t id = vl_key_id(key);
                if (id == self_id || (excl && team_excluded(excl, p.exclude_w, id))) key = kSent;
            }
            p.out_ids[row * p.out_ld + i] = vl_key_id(key);
            p.out_dist[row * p.out_ld + i] = vl_key_dist(key);
        }
        if (always_full && tid == 0) atomicOr(p.group_full + group, 1u);
        if (p.stats && lane == 0) {
            if (warp == 0) {
                atomicAdd(p.stats + 1, (unsigned long long)st_todo);
                atomicAdd(p.stats + 2, (unsigned long long)st_m);
                atomicAdd(p.stats + 6, 1ull);
                atomicAdd(p.stats + 7, (unsigned long long)(k <= n_run ? k : n_run));
                if constexpr (TIMED) {
                    atomicAdd(p.stats + 8, (unsigned long long)(unsigned int)ctl[kPop]);
                    atomicAdd(p.stats + 9, (unsigned long long)(unsigned int)ctl[kProbe]);
                    atomicAdd(p.stats + 10, (unsigned long long)(unsigned int)ctl[kGather]);
                    atomicAdd(p.stats + 12, (unsigned long long)(unsigned int)ctl[kSearchQ]);
                    atomicAdd(p.stats + 13, (unsigned long long)(unsigned int)ctl[kVisitQ]);
                }
            }
            if (warp == (TEAM == 1 ? 0 : 1)) {
                atomicAdd(p.stats + 3, (unsigned long long)st_v);
                atomicAdd(p.stats + 4, (unsigned long long)st_a);
                atomicAdd(p.stats + 5, (unsigned long long)st_b);
            }
        }
        if (p.row_ticket) {
            if (tid == 0) {
                const unsigned long long t = gridDim.x + atomicAdd(p.row_ticket, 1ull);
                ctl[kRowLo] = (int)(unsigned int)t;
                ctl[kRowHi] = (int)(unsigned int)(t >> 32);
            }
            __syncthreads();
            place = (int64_t)(((unsigned long long)(unsigned int)ctl[kRowHi] << 32) | (unsigned int)ctl[kRowLo]);
        } else {
            place += gridDim.x;
        }
        __syncthreads();
    }
}

}  // namespace
