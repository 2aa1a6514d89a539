// Frontier loops of one thread-block cluster: BFS levels and SSSP rounds of
// small frontiers, with no host round trip and no queue in global memory.
//
// A road-like graph runs thousands of levels of about a thousand vertices,
// so a level's time is its chain of dependent accesses.  The loops here keep
// that chain short:
//   - each CTA queues what its threads discover in its own shared memory
//     (one shared atomic per warp step), and every CTA takes an equal share
//     of every queue for the next level, reading it over the cluster;
//   - a queue entry is a piece of at most kClPiece edges of a vertex's list,
//     (vertex, first edge, edges): the offsets were read when the vertex was
//     queued, and a hub's list is spread over the whole cluster;
//   - the edges of a piece are visited kClBatch at a time, one atomicMin each
//     that both tests and claims (no read before it);
//   - the counts of a level go to every CTA as asynchronous stores that
//     complete an mbarrier there, the only synchronisation between levels.
// All exit decisions are taken by every thread from the same counts, so the
// cluster leaves together.
//
// The wait for a level's counts ends after a time limit (cl_wait): the CTA
// then drops what it has queued and leaves, and the run returns CGB_ETIMEOUT.
// That covers counts which come late or not at all.  The cluster's hardware
// barrier at either end of a loop has no limit of its own: it is reached by
// every CTA, because nothing between the two waits for longer than that.
//
// Vertices without out-edges are claimed but not queued.  Vertices beyond a
// CTA's queue spill to the global queue; the loop then returns
// to the host after that level, as it does when the frontier outgrows the
// bounds it is given, with the frontier in the global queue.
#include <cooperative_groups.h>

#include "persist.cuh"

namespace cgb {

namespace {

constexpr int kClThreads = 512;
constexpr int kClWarps = kClThreads / 32;
constexpr unsigned long long kClWaitNs = 1000000000ull;  // a level's counts take longer: the loop gives up
constexpr uint32_t kClSpins = 1u << 28;  // and after so many polls, whatever the clock says
constexpr uint32_t kClPollNs = 10000, kClEarly = 64;
constexpr uint32_t kClMaxCtas = 16;
constexpr uint32_t kClQueue = 8192;  // entries per CTA and buffer
constexpr uint32_t kClPiece = 8;     // edges per entry
constexpr uint32_t kClFirst = 0x80;  // marks a vertex's first entry,
constexpr uint32_t kClSingle = 0x40; // and its only one
constexpr int kClBatch = 4;
static_assert(kClQueue * kClPiece == kClusterList, "the longest list that fits a queue");

// What a CTA tells the others about the level it has built.  `word` packs
// the entries (at most kClQueue, so that the cluster's sum stays below 2^20)
// and the spill flag, so that one reduction adds both.
constexpr uint32_t kEntryMask = (1u << 20) - 1, kSpill = 1u << 20;

struct __align__(16) ClCounts {
    uint32_t word;     // entries, spill
    uint32_t medges;   // out-edges of the next frontier
    uint32_t min_far;  // SSSP split: smallest distance left in the far bitmap,
    uint32_t far;      // and the vertices left; SSSP round: far bits set (a vertex may count twice)
};

struct ClShared {
    uint64_t list[2][kClQueue];  // first edge, edges << 32 (and kClFirst)
    uint32_t v[2][kClQueue];
    ClCounts from[2][kClMaxCtas];
    uint64_t arrived[2];  // mbarriers: the counts of a level have come from every CTA
    uint32_t entries, medges, far, min_far;  // of the level being built
    uint32_t gave_up;
};

__device__ __forceinline__ void cl_reset(ClShared& s)
{
    s.entries = s.medges = s.far = 0;
    s.min_far = kValueMax;
}

// Queues the selected vertices (list at [start, start + deg)) in buffer buf
// of this CTA and adds their out-edges to `edges` (per thread; cl_next_level
// collects it); warp-collective.  Vertices without edges are skipped; a
// vertex for which the queue has no room spills to the global queue if
// take(v) holds.
template <int N, class Take>
__device__ __forceinline__ void cl_push(ClShared& s, uint32_t buf, const bool (&pred)[N], const uint32_t (&v)[N],
                                        const uint32_t (&start)[N], const uint32_t (&deg)[N], uint32_t* spill_q,
                                        uint32_t cap, ClusterState* st, uint32_t& edges, const Take& take)
{
    const uint32_t lane = lane_id();
    bool big = false;
#pragma unroll
    for (int i = 0; i < N; i++) {
        big |= pred[i] && deg[i] > kClPiece;
        edges += pred[i] ? deg[i] : 0;
    }
    auto spill = [&](bool pred, uint32_t vv) {  // warp-collective
        if (!__any_sync(0xffffffffu, pred)) return;
        warp_append(pred && take(vv), vv, spill_q, &st->qlen, cap, &st->status);
    };
    if (!__any_sync(0xffffffffu, big)) {
        // one entry per vertex
        uint32_t m[N], total = 0;
#pragma unroll
        for (int i = 0; i < N; i++) {
            m[i] = __ballot_sync(0xffffffffu, pred[i] && deg[i]);
            total += __popc(m[i]);
        }
        if (!total) return;
        uint32_t pos = 0;
        if (lane == 0) pos = atomicAdd(&s.entries, total);
        pos = __shfl_sync(0xffffffffu, pos, 0);
#pragma unroll
        for (int i = 0; i < N; i++) {
            const uint32_t at = pos + __popc(m[i] & lanemask_lt());
            const bool mine = (m[i] >> lane) & 1u;
            if (mine && at < kClQueue) {
                s.list[buf][at] = start[i] | (uint64_t)(deg[i] | kClFirst | kClSingle) << 32;
                s.v[buf][at] = v[i];
            }
            pos += __popc(m[i]);
            if (pos > kClQueue) spill(mine && at >= kClQueue, v[i]);
        }
        return;
    }
    uint32_t n[N], cnt = 0;
#pragma unroll
    for (int i = 0; i < N; i++) {
        n[i] = pred[i] ? (deg[i] + kClPiece - 1) / kClPiece : 0;
        cnt += n[i];
    }
    const uint32_t incl = warp_incl_scan(cnt);
    uint32_t pos = 0;
    if (lane == 31) pos = atomicAdd(&s.entries, incl);
    pos = __shfl_sync(0xffffffffu, pos, 31) + incl - cnt;
#pragma unroll
    for (int i = 0; i < N; i++) {
        // a vertex whose entries do not all fit spills; what it took stays empty
        auto put = [&](uint32_t at, uint32_t k, uint32_t vv, uint32_t ss, uint32_t dd, bool fits) {
            if (at >= kClQueue) return;
            const uint32_t len = fits ? min(kClPiece, dd - k * kClPiece) | (k == 0 ? kClFirst : 0) |
                                        (dd <= kClPiece ? kClSingle : 0)
                                      : 0;
            s.list[buf][at] = (ss + k * kClPiece) | (uint64_t)len << 32;
            s.v[buf][at] = vv;
        };
        const bool fits = pos + n[i] <= kClQueue;
        spill(n[i] && !fits, v[i]);
        if (n[i] <= 4)
            for (uint32_t k = 0; k < n[i]; k++) put(pos + k, k, v[i], start[i], deg[i], fits);
        for (uint32_t todo = __ballot_sync(0xffffffffu, n[i] > 4); todo; todo &= todo - 1) {
            const uint32_t l = __ffs(todo) - 1;
            const uint32_t bn = __shfl_sync(0xffffffffu, n[i], l), bp = __shfl_sync(0xffffffffu, pos, l);
            const uint32_t bv = __shfl_sync(0xffffffffu, v[i], l), bs = __shfl_sync(0xffffffffu, start[i], l);
            const uint32_t bd = __shfl_sync(0xffffffffu, deg[i], l);
            const uint32_t room = bp < kClQueue ? min(bn, kClQueue - bp) : 0;
            for (uint32_t k = lane; k < room; k += 32) put(bp + k, k, bv, bs, bd, bp + bn <= kClQueue);
        }
        pos += n[i];
    }
}

// Keeps the stages of a batch apart: everything before it is issued (and
// here x[] waited for) before anything after it.  Left to itself the compiler
// ran the batch's slots one after the other, each with its own chain
// (1200 x 1250 grid BFS: 9.0 instead of 6.9 ms).
template <int N>
__device__ __forceinline__ void stage(uint32_t (&x)[N])
{
#pragma unroll
    for (int i = 0; i < N; i++) asm volatile("" : "+r"(x[i])::"memory");
}

// One poll of phase `parity` of an mbarrier of this CTA.  It may suspend the
// thread until the phase completes, for a time that the device chooses or
// (late) kClPollNs at most.
template <bool kLate>
__device__ __forceinline__ bool cl_poll(uint32_t mbar, uint32_t parity)
{
    uint32_t done;
    if (kLate)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(mbar), "r"(parity), "r"(kClPollNs)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
    return done != 0;
}

// The rest of a wait that has polled a while: at most wait_ns by the clock
// and kClSpins polls.
__device__ __forceinline__ bool cl_wait_late(uint32_t mbar, uint32_t parity, unsigned long long wait_ns)
{
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (uint32_t spin = 0; spin < kClSpins; spin++) {
        if (cl_poll<true>(mbar, parity)) return true;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 > wait_ns) return false;
    }
    return false;
}

// Waits for phase `parity` of an mbarrier of this CTA; false after kClEarly
// polls and wait_ns.  The clock is not looked at, and no time is given to a
// poll, while the early polls run: 1200 x 1250 grid BFS 6.88 ms without a
// limit by the clock, 6.94 as it is, 6.97 with a time given to every poll,
// 7.1 with a look at the clock every 64 polls.
__device__ __forceinline__ bool cl_wait(uint32_t mbar, uint32_t parity, unsigned long long wait_ns)
{
    bool done = false;
    for (uint32_t spin = 0; !done && spin < kClEarly; spin++) done = cl_poll<false>(mbar, parity);
    return done || cl_wait_late(mbar, parity, wait_ns);
}

// Ends level `level`: sends this CTA's counts to every CTA (buffer level &
// 1) and waits for theirs.  The counts travel as asynchronous stores that
// complete the receiver's mbarrier, so a level costs one trip over the
// cluster (the hardware barrier after remote stores took twice as long).
// The fence orders the queue entries before the counts.  Buffers alternate,
// and a CTA sends the counts of a level only after it has received all of
// the level before, so no slot, queue or mbarrier phase is overtaken.
// Returns false when the wait gave up (the same CTA-wide): the counts in
// from[] are then not this level's.  send = false (the self-check) keeps this
// CTA's counts back.
__device__ __forceinline__ bool cl_next_level(cooperative_groups::cluster_group& cluster, ClShared& s, uint32_t level,
                                              uint32_t edges, ClusterState* st, unsigned long long wait_ns,
                                              bool send = true)
{
    const uint32_t buf = level & 1, ctas = cluster.num_blocks();
    if (__any_sync(0xffffffffu, edges != 0)) {
        edges = __reduce_add_sync(0xffffffffu, edges);
        if (lane_id() == 0) atomicAdd(&s.medges, edges);
    }
    __syncthreads();
    const uint32_t mbar = (uint32_t)__cvta_generic_to_shared(&s.arrived[buf]);
    if (threadIdx.x < 32) {
        const uint32_t n = s.entries;
        const ClCounts c{min(n, kClQueue) | (n > kClQueue ? kSpill : 0), s.medges, s.min_far, s.far};
        __syncwarp();
        if (threadIdx.x == 0) {
            cl_reset(s);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar),
                         "r"(ctas * (uint32_t)sizeof(ClCounts))
                         : "memory");
        }
        if (threadIdx.x < ctas && send) {
            asm volatile("fence.acq_rel.cluster;" ::: "memory");
            uint32_t to, to_bar;
            asm("mapa.shared::cluster.u32 %0, %1, %2;"
                : "=r"(to)
                : "r"((uint32_t)__cvta_generic_to_shared(&s.from[buf][cluster.block_rank()])), "r"(threadIdx.x));
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to_bar) : "r"(mbar), "r"(threadIdx.x));
            asm volatile(
                "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to),
                "r"(c.word), "r"(c.medges), "r"(c.min_far), "r"(c.far), "r"(to_bar)
                : "memory");
        }
    }
    if (!cl_wait(mbar, (level >> 1) & 1, wait_ns)) {
        s.gave_up = 1;
        atomicOr(&st->status, 2u);
    }
    __syncthreads();  // the counts were reset, and all threads agree on gave_up
    return !s.gave_up;
}

// Ends the loop at level `level`: every CTA passes the cluster's barrier, so
// none leaves while another may read its queue.  One that gave up may still
// have that level's counts on their way to it: all CTAs have sent what they
// send, and it waits for them once more before its shared memory goes.
__device__ __forceinline__ void cl_leave(cooperative_groups::cluster_group& cluster, ClShared& s, uint32_t level,
                                         unsigned long long wait_ns)
{
    __threadfence();
    cluster.sync();
    if (s.gave_up)
        cl_wait((uint32_t)__cvta_generic_to_shared(&s.arrived[level & 1]), (level >> 1) & 1, wait_ns);
}

__device__ __forceinline__ void cl_setup(cooperative_groups::cluster_group& cluster, ClShared& s, ClusterState* st)
{
    if (threadIdx.x == 0) {
        cl_reset(s);
        s.gave_up = 0;
        for (int i = 0; i < 2; i++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(&s.arrived[i]))
                         : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (cluster.block_rank() == 0) *st = ClusterState{};
    }
    __threadfence();
    cluster.sync();
}

// The frontier given in q[0, nf) as entries of buffer 0; returns this
// thread's out-edges.
__device__ __forceinline__ uint32_t cl_load(cooperative_groups::cluster_group& cluster, ClShared& s,
                                            const uint32_t* __restrict__ off, const uint32_t* q, uint32_t nf,
                                            uint32_t* spill_q, uint32_t cap, ClusterState* st)
{
    const uint32_t ctas = cluster.num_blocks();
    uint32_t edges = 0;
    for (uint32_t b = 0; b < nf; b += kClThreads * ctas) {
        const uint32_t i = b + cluster.block_rank() + ctas * threadIdx.x;
        const bool pred[1] = {i < nf};
        const uint32_t v[1] = {pred[0] ? q[i] : 0};
        const uint32_t s0[1] = {pred[0] ? off[v[0]] : 0};
        const uint32_t d[1] = {pred[0] ? off[v[0] + 1] - s0[0] : 0};
        cl_push<1>(s, 0, pred, v, s0, d, spill_q, cap, st, edges, [](uint32_t) { return true; });
    }
    return edges;
}

// Visits every entry of buffer buf: visit(entry, start, len, flags) is
// warp-collective (len 0 on idle lanes), entry a pointer to the vertex, flags
// kClFirst and kClSingle (0 on idle lanes).  A
// CTA takes the entries j = rank mod ctas of every queue, neighbouring lanes
// from neighbouring CTAs' queues, so that all CTAs have equal shares and a
// small frontier fills few warps.
template <class Visit>
__device__ __forceinline__ void cl_for_entries(cooperative_groups::cluster_group& cluster, ClShared& s, uint32_t buf,
                                               const Visit& visit)
{
    const uint32_t ctas = cluster.num_blocks();  // a power of two
    const uint32_t from = threadIdx.x & (ctas - 1);
    const uint32_t n = s.from[buf][from].word & kEntryMask;
    const ClShared* r = cluster.map_shared_rank(&s, from);
    for (uint32_t j = cluster.block_rank() + threadIdx.x / ctas * ctas;; j += kClThreads) {
        if (!__any_sync(0xffffffffu, j < n)) break;
        const uint64_t list = j < n ? r->list[buf][j] : 0;
        const uint32_t len = (uint32_t)(list >> 32);
        visit(&r->v[buf][j], (uint32_t)list, len & (kClSingle - 1), len & (kClFirst | kClSingle));
    }
}

// Writes the frontier (this CTA's entries of buffer buf) to the global
// queue: the vertices for which take(v) holds.
template <class Take>
__device__ __forceinline__ void cl_flush(ClShared& s, uint32_t buf, uint32_t rank, const uint32_t* __restrict__ off,
                                         uint32_t* q, uint32_t cap, ClusterState* st, const Take& take)
{
    const uint32_t n = s.from[buf][rank].word & kEntryMask;
    uint32_t mx = 0;
    for (uint32_t b = 0; b < n; b += kClThreads) {
        const uint32_t j = b + threadIdx.x;
        bool first = j < n && (s.list[buf][j] >> 32 & kClFirst);
        const uint32_t v = first ? s.v[buf][j] : 0u;
        if (first) first = take(v);
        if (first) mx = max(mx, off[v + 1] - off[v]);
        warp_append(first, v, q, &st->qlen, cap, &st->status);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane_id() == 0 && mx) atomicMax(&st->max_deg, mx);
}

}  // namespace

// BFS levels from q_in[0, nf), the vertices of level start_level.  Stops
// before a level whose frontier exceeds nf_exit queue entries or scout_exit
// out-edges, after a spill or max_levels levels.
__global__ void __launch_bounds__(kClThreads, 1)
    k_bfs_cluster(const uint32_t* __restrict__ off, const uint32_t* __restrict__ dst, uint32_t* level,
                  uint32_t* visited, const uint32_t* q_in, uint32_t* q_out, uint32_t cap, uint32_t nz,
                  uint32_t start_level, uint32_t nf, uint32_t nf_exit, uint32_t scout_exit, uint32_t max_levels,
                  unsigned long long wait_ns, ClusterState* st, ClusterState* host)
{
    extern __shared__ __align__(16) unsigned char smem[];
    ClShared& s = *reinterpret_cast<ClShared*>(smem);
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const uint32_t ctas = cluster.num_blocks(), rank = cluster.block_rank();
    const bool leader = rank == 0 && threadIdx.x == 0;
    cl_setup(cluster, s, st);
    bool ok = cl_next_level(cluster, s, 0, cl_load(cluster, s, off, q_in, nf, q_out, cap, st), st, wait_ns);
    uint32_t it = 0, found = 0, word, scout;
    // a vertex that leaves for the global queue gets its visited bit now
    auto mark = [&](uint32_t v) {
        atomicOr(visited + (v >> 5), 1u << (v & 31u));
        return true;
    };
    unsigned long long scouts = 0;
    for (;; it++) {
        const uint32_t buf = it & 1;
        const ClCounts c = lane_id() < ctas ? s.from[buf][lane_id()] : ClCounts{};
        word = __reduce_add_sync(0xffffffffu, c.word);
        scout = __reduce_add_sync(0xffffffffu, c.medges);
        if (!ok || (word & kEntryMask) == 0 || (word & ~kEntryMask) || (word & kEntryMask) > nf_exit || scout > scout_exit ||
            it >= max_levels)
            break;
        scouts += scout;
        const uint32_t next_level = start_level + it + 1;
        uint32_t edges = 0;
        cl_for_entries(cluster, s, buf, [&](const uint32_t* entry, uint32_t start, uint32_t len, uint32_t) {
            // the visited bit of a queued vertex, off the level's chain
            if (len) {
                const uint32_t v = *entry;
                atomicOr(visited + (v >> 5), 1u << (v & 31u));
            }
            for (uint32_t b = 0; __any_sync(0xffffffffu, b < len); b += kClBatch) {
                uint32_t d[kClBatch], old[kClBatch], lo[kClBatch], dg[kClBatch];
                bool enq[kClBatch];
#pragma unroll
                for (int i = 0; i < kClBatch; i++) d[i] = b + i < len ? dst[start + b + i] : 0u;
                stage(d);
#pragma unroll
                for (int i = 0; i < kClBatch; i++) {
                    // claim, and read the list bounds meanwhile, whether or not the claim wins
                    const bool in = b + i < len;
                    old[i] = in ? atomicMin(level + d[i], next_level) : 0u;
                    lo[i] = in ? off[d[i]] : 0u;
                    dg[i] = in ? off[d[i] + 1] : 0u;
                }
                stage(lo);
                stage(dg);
                stage(old);
#pragma unroll
                for (int i = 0; i < kClBatch; i++) {
                    const bool win = old[i] == kValueMax;  // levels are below it
                    found += win ? 1u : 0u;
                    dg[i] -= lo[i];
                    enq[i] = win && d[i] < nz;
                    // not queued: its visited bit is set here
                    if (win && !(enq[i] && dg[i])) atomicOr(visited + (d[i] >> 5), 1u << (d[i] & 31u));
                }
                cl_push<kClBatch>(s, buf ^ 1, enq, d, lo, dg, q_out, cap, st, edges, mark);
            }
        });
        ok = cl_next_level(cluster, s, it + 1, edges, st, wait_ns);
    }
    found = __reduce_add_sync(0xffffffffu, found);
    if (lane_id() == 0 && found) atomicAdd(&st->found, found);
    if (ok && it > 0) cl_flush(s, it & 1, rank, off, q_out, cap, st, mark);
    cl_leave(cluster, s, it, wait_ns);
    if (leader) {
        ClusterState h{};
        h.qlen = __ldcg(&st->qlen);
        h.status = __ldcg(&st->status);
        // (kept where vertices spill, the longest list cost SSSP rounds 5 to 12 %)
        h.max_deg = word & ~kEntryMask ? 0xFFFFFFFFu : __ldcg(&st->max_deg);
        h.found = __ldcg(&st->found);
        h.levels = it;
        h.scout = scout;
        h.scouts = scouts;
        *host = h;
    }
}

// SSSP rounds and bucket splits (see sssp_device_tail) from the near queue
// q_in[0, nf) at threshold thr.  stamp (zero on entry) holds the round that
// last expanded a vertex: one that several edges improve in a round is queued
// as often, and its later entries are skipped (checking when it is queued
// would lengthen the round's chain; only lists of several pieces pay that).
// Rounds only grow and kLeft is above them all, so marks are set by
// atomicMax: an entry expanded later in the round leaves the mark of a vertex
// that has gone to the global queue.
// far_len_out receives the far bitmap's population on exit.
template <bool kHasW>
__global__ void __launch_bounds__(kClThreads, 1)
    k_sssp_cluster(const uint32_t* __restrict__ off, const uint32_t* __restrict__ dst, const uint32_t* __restrict__ w,
                   uint32_t* dist, uint32_t* stamp, uint32_t* far_bm, uint32_t words, const uint32_t* q_in,
                   uint32_t* q_out, uint32_t cap, uint32_t nz, uint32_t nf, unsigned long long thr, uint32_t nfar,
                   unsigned long long bucket_lo, uint32_t delta, uint32_t nf_exit, uint32_t scout_exit,
                   uint32_t far_exit, uint32_t max_rounds, uint32_t* far_len_out, unsigned long long wait_ns,
                   ClusterState* st, ClusterState* host)
{
    extern __shared__ __align__(16) unsigned char smem[];
    ClShared& s = *reinterpret_cast<ClShared*>(smem);
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const uint32_t ctas = cluster.num_blocks(), rank = cluster.block_rank(), lane = lane_id();
    const bool leader = rank == 0 && threadIdx.x == 0;
    cl_setup(cluster, s, st);
    bool ok = cl_next_level(cluster, s, 0, cl_load(cluster, s, off, q_in, nf, q_out, cap, st), st, wait_ns);
    uint32_t it = 0, word, scout, added = 0;
    // a vertex goes to the global queue once (its short list may be queued twice)
    const uint32_t kLeft = 0xFFFFFFFFu;
    auto take = [&](uint32_t v) { return atomicExch(stamp + v, kLeft) != kLeft; };
    uint32_t far = nfar;  // at least the far bitmap's population
    bool after_split = false;
    for (;; it++) {
        const uint32_t buf = it & 1;
        ClCounts c{0, 0, kValueMax, 0};
        if (lane < ctas) c = s.from[buf][lane];
        word = __reduce_add_sync(0xffffffffu, c.word);
        scout = __reduce_add_sync(0xffffffffu, c.medges);
        const uint32_t far_level = __reduce_add_sync(0xffffffffu, c.far);
        far = after_split ? far_level : far + min(far_level, 0xFFFFFFFFu - far);
        const uint32_t entries = word & kEntryMask;
        // a large far set is split by the whole machine
        if (!ok || (entries == 0 && (far == 0 || far > far_exit))) break;
        if ((word & ~kEntryMask) || entries > nf_exit || scout > scout_exit || it >= max_rounds) break;
        uint32_t edges = 0;
        if (entries) {
            const uint32_t bound = (uint32_t)min(thr, (unsigned long long)kValueMax);
            uint32_t far_set = 0;
            cl_for_entries(cluster, s, buf, [&](const uint32_t* entry, uint32_t start, uint32_t len, uint32_t flags) {
                const uint32_t v = len ? *entry : 0u;
                const uint32_t du = len ? __ldcg(dist + v) : 0u;
                // a vertex queued twice: the second entry is skipped
                const bool again = (flags & kClSingle) && atomicMax(stamp + v, it + 1) == it + 1;
                added += (flags & kClFirst) && !again ? 1u : 0u;  // a vertex counts with its first entry
                for (uint32_t b = 0; __any_sync(0xffffffffu, b < len); b += kClBatch) {
                    uint32_t d[kClBatch], nd[kClBatch], old[kClBatch], lo[kClBatch], dg[kClBatch];
                    bool near[kClBatch], to_far[kClBatch];
#pragma unroll
                    for (int i = 0; i < kClBatch; i++) {
                        const bool in = b + i < len;
                        d[i] = in ? dst[start + b + i] : 0u;
                        const uint64_t c = (uint64_t)du + (kHasW ? (in ? w[start + b + i] : 0u) : 1u);
                        nd[i] = in && !again && c < kValueMax ? (uint32_t)c : kValueMax;  // never lowers a distance
                    }
                    stage(d);
                    stage(nd);
#pragma unroll
                    for (int i = 0; i < kClBatch; i++) {
                        // relax, and read the list bounds meanwhile, whether or not it improves
                        const bool in = nd[i] < kValueMax;
                        old[i] = in ? atomicMin(dist + d[i], nd[i]) : 0u;
                        lo[i] = in ? off[d[i]] : 0u;
                        dg[i] = in ? off[d[i] + 1] : 0u;
                    }
                    stage(lo);
                    stage(dg);
                    stage(old);
#pragma unroll
                    for (int i = 0; i < kClBatch; i++) {
                        const bool better = nd[i] < old[i] && d[i] < nz;
                        near[i] = better && nd[i] < bound;
                        to_far[i] = better && !near[i];
                        dg[i] -= lo[i];
                        // the entries of a longer list do not know of one another: it is queued once
                        if (near[i] && dg[i] > kClPiece) {
                            const uint32_t was = atomicMax(stamp + d[i], it + 2);
                            near[i] = was != it + 2 && was != kLeft;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < kClBatch; i++) {
                        if (to_far[i]) atomicOr(far_bm + (d[i] >> 5), 1u << (d[i] & 31u));
                        far_set += to_far[i] ? 1u : 0u;
                    }
                    cl_push<kClBatch>(s, buf ^ 1, near, d, lo, dg, q_out, cap, st, edges, take);
                }
            });
            far_set = __reduce_add_sync(0xffffffffu, far_set);
            if (lane == 0 && far_set) atomicAdd(&s.far, far_set);
            after_split = false;
        } else {
            // next bucket [thr, hi); after a split that found nothing, jump
            // to the bucket of the smallest far distance
            unsigned long long hi = thr + delta;
            const uint32_t min_far = __reduce_min_sync(0xffffffffu, c.min_far);
            if (after_split && min_far != kValueMax)
                hi = max(hi, ((unsigned long long)min_far / delta + 1) * delta);
            bucket_lo = thr;
            thr = hi;
            const uint32_t lo32 = (uint32_t)min(bucket_lo, (unsigned long long)kValueMax);
            const uint32_t hi32 = (uint32_t)min(hi, (unsigned long long)kValueMax);
            uint32_t mn = kValueMax, kept = 0;
            // a warp takes 32 words with one coalesced load and visits the
            // non-zero ones kClBatch at a time, lane b of word j reading the
            // distance of vertex 32 j + b; it owns its words
            for (uint32_t w0 = (rank * kClWarps + (threadIdx.x >> 5)) * 32; w0 < words; w0 += ctas * kClThreads) {
                const uint32_t bits = w0 + lane < words ? __ldcg(far_bm + w0 + lane) : 0u;
                uint32_t todo = __ballot_sync(0xffffffffu, bits != 0);
                while (todo) {
                    uint32_t wi[kClBatch], wb[kClBatch], v[kClBatch], dv[kClBatch], lo[kClBatch], dg[kClBatch];
                    bool near[kClBatch];
#pragma unroll
                    for (int k = 0; k < kClBatch; k++) {
                        const uint32_t j = todo ? __ffs(todo) - 1 : 0u;
                        wb[k] = __shfl_sync(0xffffffffu, bits, j);
                        if (!todo) wb[k] = 0;
                        todo &= todo ? todo - 1 : 0u;
                        wi[k] = w0 + j;
                        v[k] = wi[k] * 32 + lane;
                        dv[k] = (wb[k] >> lane) & 1u ? __ldcg(dist + v[k]) : 0u;
                    }
                    stage(dv);
#pragma unroll
                    for (int k = 0; k < kClBatch; k++) {
                        const bool in = (wb[k] >> lane) & 1u, keep = in && dv[k] >= hi32;
                        near[k] = in && !keep && dv[k] >= lo32;
                        if (keep) mn = min(mn, dv[k]);
                        const uint32_t km = __ballot_sync(0xffffffffu, keep);
                        if (lane == 0 && wb[k]) {
                            if (km != wb[k]) far_bm[wi[k]] = km;
                            kept += __popc(km);
                        }
                        lo[k] = near[k] ? off[v[k]] : 0u;
                        dg[k] = near[k] ? off[v[k] + 1] : 0u;
                    }
                    stage(lo);
                    stage(dg);
#pragma unroll
                    for (int k = 0; k < kClBatch; k++) dg[k] -= lo[k];
                    cl_push<kClBatch>(s, buf ^ 1, near, v, lo, dg, q_out, cap, st, edges, take);
                }
            }
            mn = __reduce_min_sync(0xffffffffu, mn);
            if (lane == 0) {
                if (mn != kValueMax) atomicMin(&s.min_far, mn);
                if (kept) atomicAdd(&s.far, kept);
            }
            after_split = true;
        }
        ok = cl_next_level(cluster, s, it + 1, edges, st, wait_ns);
    }
    if (ok && it > 0) cl_flush(s, it & 1, rank, off, q_out, cap, st, take);
    added = __reduce_add_sync(0xffffffffu, added);
    if (lane == 0 && added) atomicAdd(&st->found, added);
    if (ok && far) {
        uint32_t pop = 0;
        for (uint32_t i = rank * kClThreads + threadIdx.x; i < words; i += ctas * kClThreads)
            pop += __popc(__ldcg(far_bm + i));
        pop = __reduce_add_sync(0xffffffffu, pop);
        if (lane == 0 && pop) atomicAdd(&st->far_left, pop);
    }
    cl_leave(cluster, s, it, wait_ns);
    if (leader) {
        ClusterState h{};
        h.qlen = __ldcg(&st->qlen);
        h.status = __ldcg(&st->status);
        h.far_left = __ldcg(&st->far_left);
        // (kept where vertices spill, the longest list cost SSSP rounds 5 to 12 %)
        h.max_deg = word & ~kEntryMask ? 0xFFFFFFFFu : __ldcg(&st->max_deg);
        h.found = __ldcg(&st->found);
        h.levels = it;
        h.scout = scout;
        h.thr = thr;
        h.bucket_lo = bucket_lo;
        *far_len_out = h.far_left;
        *host = h;
    }
}

// Self-check of the time limit: level 0 completes; at level 1 CTA 0 sends
// nothing, so every CTA's wait runs out, and all meet at the last barrier.
__global__ void __launch_bounds__(kClThreads, 1)
    k_cluster_timeout(unsigned long long wait_ns, ClusterState* st, ClusterState* host)
{
    extern __shared__ __align__(16) unsigned char smem[];
    ClShared& s = *reinterpret_cast<ClShared*>(smem);
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    cl_setup(cluster, s, st);
    uint32_t it = 0;
    bool ok = cl_next_level(cluster, s, 0, 0, st, wait_ns);
    if (ok) ok = cl_next_level(cluster, s, ++it, 0, st, wait_ns, cluster.block_rank() != 0);
    cl_leave(cluster, s, it, wait_ns);
    if (cluster.block_rank() == 0 && threadIdx.x == 0) {
        ClusterState h{};
        h.status = __ldcg(&st->status);
        h.levels = it;
        *host = h;
    }
}

// CTAs of the cluster: 16 when the device schedules such a cluster (a
// non-portable size), else 8, else 0 (no cluster loops).
template <class K>
static uint32_t cluster_ctas(K kern)
{
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ClShared)) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    for (int c : {16, 8}) {
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim = {(unsigned)c, 1, 1};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(c);
        cfg.blockDim = dim3(kClThreads);
        cfg.dynamicSmemBytes = sizeof(ClShared);
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0) return (uint32_t)c;
        cudaGetLastError();
    }
    return 0;
}

// The cluster size of the current device (the smallest over the kernels),
// decided once per device; the kernels' attributes are set on the way.
uint32_t cluster_loop_ctas()
{
    constexpr int kMaxDevices = 64;
    static std::atomic<int> cache[kMaxDevices];  // CTAs + 1
    int dev = 0;
    CGB_CUDA_TRY(cudaGetDevice(&dev));
    CGB_REQUIRE(dev >= 0 && dev < kMaxDevices, CGB_EUNSUPPORTED, "device ordinal out of range");
    int c = cache[dev].load(std::memory_order_acquire);
    if (!c) {
        c = 1 + (int)std::min({cluster_ctas(k_bfs_cluster), cluster_ctas(k_sssp_cluster<true>),
                               cluster_ctas(k_sssp_cluster<false>), cluster_ctas(k_cluster_timeout)});
        cache[dev].store(c, std::memory_order_release);
    }
    return (uint32_t)(c - 1);
}

// Launches a cluster loop on stream st and returns what it reports (through
// pinned host memory; synchronises the stream).
template <class... P, class... A>
static ClusterState launch_cluster(cudaStream_t st, void (*kern)(P...), A... args)
{
    PinnedArray<ClusterState> h(1);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {cluster_loop_ctas(), 1, 1};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(attr[0].val.clusterDim.x);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = sizeof(ClShared);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CGB_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, args..., h.data()));
    CGB_CUDA_TRY(cudaStreamSynchronize(st));
    return h[0];
}

// The same for a graph's run.
template <class... P, class... A>
static ClusterState run_cluster(cgb_graph* g, void (*kern)(P...), A... args)
{
    if (!g->cluster) g->cluster = pool_alloc(sizeof(ClusterState), g->stream);
    ++g->stats.launches;
    const ClusterState h = launch_cluster(g->stream, kern, args..., kClWaitNs, (ClusterState*)g->cluster);
    CGB_REQUIRE(!(h.status & 2u), CGB_ETIMEOUT, "cluster loop: a level's counts did not come in time");
    CGB_REQUIRE(!h.status, CGB_EOVERFLOW, "cluster loop: queue overflow");
    return h;
}

cgb_status cluster_timeout_check(uint32_t limit_us)
{
    CGB_REQUIRE(cluster_loop_ctas() > 0, CGB_EUNSUPPORTED, "the device schedules no cluster of 8 CTAs");
    ClusterState* st = nullptr;
    CGB_CUDA_TRY(cudaMalloc((void**)&st, sizeof(ClusterState)));
    cudaStream_t stream = nullptr;
    ClusterState h{};
    try {
        CGB_CUDA_TRY(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
        h = launch_cluster(stream, k_cluster_timeout, limit_us * 1000ull, st);
    } catch (...) {
        if (stream) cudaStreamDestroy(stream);
        cudaFree(st);
        throw;
    }
    cudaStreamDestroy(stream);
    cudaFree(st);
    CGB_REQUIRE(h.levels == 1, CGB_ECUDA, "cluster self-check: the first level did not complete");
    return (h.status & 2u) ? CGB_ETIMEOUT : CGB_OK;
}

PersistResult bfs_cluster(cgb_graph* g, uint32_t cur, uint32_t nf, uint32_t level, uint32_t nf_exit,
                          uint32_t scout_exit, uint32_t max_levels)
{
    const ClusterState h =
        run_cluster(g, k_bfs_cluster, (const uint32_t*)g->off, (const uint32_t*)g->dst, g->value, g->visited,
                    (const uint32_t*)g->q[cur], g->q[cur ^ 1], g->V, g->nz, level, nf, nf_exit, scout_exit,
                    max_levels);
    PersistResult r;
    r.levels = h.levels;
    r.cur = h.levels ? cur ^ 1 : cur;
    r.nf = h.levels ? h.qlen : nf;
    r.scout = h.scout;
    r.max_deg = std::min(h.max_deg, g->max_degree);
    r.found = h.found;
    r.scouts = h.scouts;
    return r;
}

SsspTail sssp_cluster(cgb_graph* g, uint32_t cur, uint32_t nf, uint64_t thr, uint32_t nfar, uint64_t bucket_lo,
                      uint32_t* far_bm, uint32_t delta, uint32_t nf_exit, uint32_t scout_exit, uint32_t far_exit,
                      uint32_t max_rounds)
{
    CGB_CUDA_TRY(cudaMemsetAsync(g->stamp, 0, (size_t)g->V * 4, g->stream));
    const ClusterState h =
        run_cluster(g, g->w ? k_sssp_cluster<true> : k_sssp_cluster<false>, (const uint32_t*)g->off,
                    (const uint32_t*)g->dst, (const uint32_t*)g->w, g->value, g->stamp, far_bm, g->words(),
                    (const uint32_t*)g->q[cur], g->q[cur ^ 1], g->V, g->nz, nf, (unsigned long long)thr, nfar,
                    (unsigned long long)bucket_lo, delta, nf_exit, scout_exit, far_exit, max_rounds,
                    &g->ctr->far_len[0]);
    SsspTail t;
    t.r.levels = h.levels;
    t.r.cur = h.levels ? cur ^ 1 : cur;
    t.r.nf = h.levels ? h.qlen : nf;
    t.r.scout = h.scout;
    t.r.max_deg = std::min(h.max_deg, g->max_degree);
    t.r.added = h.found;
    t.thr = h.thr;
    t.nfar = h.far_left;
    t.bucket_lo = h.bucket_lo;
    return t;
}

}  // namespace cgb
