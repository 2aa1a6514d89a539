// Delta-stepping SSSP (near queue, far bitmap) with atomicMin relaxation.
//
// Result semantics follow the reference's SSSP: dist[root] = 0, relaxation
// dist[d] = min(dist[d], dist[u] + w) applied only when it lowers the value
// (my_project/CGgraph/device_algorithm.cuh:293-329, host_algorithm.hpp:277-300),
// unreachable vertices keep 999999999; a candidate >= 999999999 never lowers
// a value, exactly as in the reference's uint32 comparison.  The reference
// re-relaxes Bellman-Ford style from a worklist; any order of monotone
// atomicMin relaxations reaches the same fixpoint, so the result is
// bit-identical.
//
// Schedule: vertices whose tentative distance is below the current threshold
// T form the near queue, which is expanded round after round with the
// degree-binned push of push.cuh; a vertex improved to a distance >= T sets
// its bit in the far bitmap (V/32 words, L2-resident).  When the near queue
// empties, the bitmap is split at [T, T + delta): those vertices become the
// near queue, vertices below T are dropped (any improvement below T was
// pushed to the near queue and has been expanded), the rest stay.  A near
// bitmap, cleared before each round, keeps each vertex at most once in a
// round's queue.
#include "engine.cuh"
#include "persist.cuh"
#include "policy.cuh"
#include "push.cuh"

namespace cgb {

__shared__ uint32_t s_sssp_newfar;  // per-CTA count of vertices newly set in the far bitmap
__shared__ unsigned long long s_sssp_medges;  // per-CTA out-degree sum of the next near queue
__shared__ uint32_t s_sssp_touched;  // per-CTA count of vertices reached for the first time
__shared__ uint32_t s_sssp_maxdeg;   // per-CTA longest list of the next near queue

// Push round: each improvement is an atomicMin whose returned value tells the
// one thread that lowered a distance; it claims the vertex in the near
// bitmap (next near queue, distance below thr) or the far bitmap.  Edges are
// visited kBatch slots per lane at a time (push.cuh): the slots' edge,
// distance and bitmap loads are each issued together.
template <bool kHasW>
struct SsspOp {
    const uint32_t* __restrict__ off;
    const uint32_t* __restrict__ dst;
    const uint32_t* __restrict__ w;
    uint32_t* dist;
    uint32_t* near_bm;  // dedup of this round's near queue (cleared before the round)
    uint32_t thr;
    uint32_t nz;
    uint32_t* near_out;
    uint32_t* near_len;
    uint32_t cap;
    uint32_t* far_bm;
    DevCounters* ctr;
    uint32_t t_newfar = 0, t_touched = 0, t_edges = 0, t_maxdeg = 0;  // this thread's counts
    static constexpr bool kStaged = true;
    static constexpr int kBatch = 4;

    __device__ __forceinline__ bool load(uint32_t v, uint32_t& s, uint32_t& d, uint32_t& m) const
    {
        s = off[v];
        d = off[v + 1] - s;
        m = dist[v];
        return m < kValueMax;
    }
    template <int N>
    __device__ __forceinline__ void edges(const bool (&valid)[N], const uint32_t (&e)[N],
                                          const uint32_t (&du)[N])
    {
        uint32_t d[N], nd[N], cur[N], old[N], word[N], bit[N];
        bool ok[N], near_c[N], far_c[N], first[N], to_near[N], new_far[N];
#pragma unroll
        for (int i = 0; i < N; i++) {
            // the edge arrays stream through once: evict first, so L2 keeps dist[] and the bitmaps
            d[i] = valid[i] ? __ldcs(dst + e[i]) : 0u;
            const uint64_t cand = (uint64_t)du[i] + (kHasW ? (valid[i] ? (uint64_t)__ldcs(w + e[i]) : 0ull) : 1ull);
            ok[i] = valid[i] && cand < kValueMax;
            nd[i] = ok[i] ? (uint32_t)cand : 0u;
        }
#pragma unroll
        for (int i = 0; i < N; i++) cur[i] = ok[i] ? __ldcg(dist + d[i]) : 0u;  // L2 only: a gather rarely hits L1
#pragma unroll
        for (int i = 0; i < N; i++) {
            ok[i] = ok[i] && nd[i] < cur[i];
            old[i] = ok[i] ? atomicMin(dist + d[i], nd[i]) : 0u;
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            first[i] = ok[i] && old[i] == kValueMax;
            const bool q = ok[i] && nd[i] < old[i] && d[i] < nz;
            near_c[i] = q && nd[i] < thr;
            far_c[i] = q && !near_c[i];
            bit[i] = 1u << (d[i] & 31u);
            word[i] = q ? (near_c[i] ? near_bm : far_bm)[d[i] >> 5] : ~0u;
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            bool fresh = false;
            if (!(word[i] & bit[i])) fresh = !(atomicOr((near_c[i] ? near_bm : far_bm) + (d[i] >> 5), bit[i]) & bit[i]);
            to_near[i] = fresh && near_c[i];
            new_far[i] = fresh && far_c[i];
        }
        stage_append_n<N>(to_near, d, near_out, near_len, cap, &ctr->overflow);
        // out-edges of the next near queue: the next round's push / pull choice
        uint32_t lo[N], hi[N];
#pragma unroll
        for (int i = 0; i < N; i++) {
            lo[i] = to_near[i] ? off[d[i]] : 0u;
            hi[i] = to_near[i] ? off[d[i] + 1] : 0u;
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            t_newfar += new_far[i] ? 1u : 0u;
            t_touched += first[i] ? 1u : 0u;
            t_edges += hi[i] - lo[i];
            t_maxdeg = max(t_maxdeg, hi[i] - lo[i]);
        }
    }
    __device__ __forceinline__ void edge(bool valid, uint32_t e, uint32_t du)
    {
        const bool v[1] = {valid};
        const uint32_t ee[1] = {e}, m[1] = {du};
        edges<1>(v, ee, m);
    }
    __device__ __forceinline__ void block_begin() const
    {
        stage_begin();
        if (threadIdx.x == 0) {
            s_sssp_newfar = 0;
            s_sssp_medges = 0;
            s_sssp_touched = 0;
            s_sssp_maxdeg = 0;
        }
    }
    __device__ __forceinline__ void block_end() const
    {
        const uint32_t nf = __reduce_add_sync(0xffffffffu, t_newfar), nt = __reduce_add_sync(0xffffffffu, t_touched);
        const uint32_t dg = __reduce_add_sync(0xffffffffu, t_edges);  // at most E < 2^32
        const uint32_t mx = __reduce_max_sync(0xffffffffu, t_maxdeg);
        if (lane_id() == 0) {
            if (nf) atomicAdd(&s_sssp_newfar, nf);
            if (nt) atomicAdd(&s_sssp_touched, nt);
            if (dg) atomicAdd(&s_sssp_medges, (unsigned long long)dg);
            if (mx) atomicMax(&s_sssp_maxdeg, mx);
        }
        stage_end(near_out, near_len, cap, &ctr->overflow);  // a CTA barrier is inside
        if (threadIdx.x == 0 && s_sssp_newfar) atomicAdd(&ctr->far_len[0], s_sssp_newfar);
        if (threadIdx.x == 0 && s_sssp_medges) atomicAdd(&ctr->medges, s_sssp_medges);
        if (threadIdx.x == 0 && s_sssp_touched) atomicAdd(&ctr->touched, s_sssp_touched);
        if (threadIdx.x == 0 && s_sssp_maxdeg) atomicMax(&ctr->max_deg, s_sssp_maxdeg);
    }
};

// Dense-frontier relaxation: the near set's out-edges lower dist[] with
// fire-and-forget atomicMin (the result is unused, so it issues as a
// reduction) and enqueue nothing; k_sssp_dense_scan then finds the improved
// vertices by comparing dist[] with its snapshot from before the round.
// (Marking improved vertices in a bitmap instead costs more than the scan:
// the bitmap's words are shared by 32 vertices, and their reductions queue
// behind each other.)  Edges are visited kBatch slots per lane at a time.
template <bool kHasW>
struct SsspDenseOp {
    const uint32_t* __restrict__ off;
    const uint32_t* __restrict__ dst;
    const uint32_t* __restrict__ w;
    uint32_t* dist;
    static constexpr int kBatch = 4;

    __device__ __forceinline__ bool load(uint32_t v, uint32_t& s, uint32_t& d, uint32_t& m) const
    {
        s = off[v];
        d = off[v + 1] - s;
        m = dist[v];
        return m < kValueMax;
    }
    template <int N>
    __device__ __forceinline__ void edges(const bool (&valid)[N], const uint32_t (&e)[N],
                                          const uint32_t (&du)[N]) const
    {
        uint32_t d[N], nd[N], cur[N];
        bool ok[N];
#pragma unroll
        for (int i = 0; i < N; i++) {
            d[i] = valid[i] ? __ldcs(dst + e[i]) : 0u;
            const uint64_t cand = (uint64_t)du[i] + (kHasW ? (valid[i] ? (uint64_t)__ldcs(w + e[i]) : 0ull) : 1ull);
            ok[i] = valid[i] && cand < kValueMax;
            nd[i] = ok[i] ? (uint32_t)cand : 0u;
        }
#pragma unroll
        for (int i = 0; i < N; i++) cur[i] = ok[i] ? __ldcg(dist + d[i]) : 0u;  // L2 only: a gather rarely hits L1
#pragma unroll
        for (int i = 0; i < N; i++)
            if (ok[i] && nd[i] < cur[i]) atomicMin(dist + d[i], nd[i]);
    }
    __device__ __forceinline__ void edge(bool valid, uint32_t e, uint32_t du) const
    {
        const bool v[1] = {valid};
        const uint32_t ee[1] = {e}, m[1] = {du};
        edges<1>(v, ee, m);
    }
    __device__ __forceinline__ void block_begin() const {}
    __device__ __forceinline__ void block_end() const {}
};

// After a dense round: every vertex whose distance dropped below its snapshot
// joins the next near queue (below thr) or the far bitmap; first touches
// (the snapshot was infinite) are counted.  A lane takes four consecutive
// vertices with one 16-byte load of each array, so a warp covers 128
// vertices = 4 bitmap words per step; the 8 lanes of a word OR their far
// bits together, and the first of them writes the word (no atomics: only
// this warp touches it).  Next-queue vertices are staged (push.cuh), so warps
// do not wait for one another.  The next queue's out-edges and the new far
// bits are counted, and the snapshot is brought up to date where it changed,
// so that a dense round that follows needs no copy.
__global__ void __launch_bounds__(kBlock) k_sssp_dense_scan(uint32_t V, const uint32_t* __restrict__ dist,
                                                            uint32_t* __restrict__ snap, uint32_t thr,
                                                            uint32_t nz, const uint32_t* __restrict__ off,
                                                            uint32_t* far_bm, uint32_t* near_out, uint32_t* near_len,
                                                            uint32_t cap, DevCounters* ctr)
{
    const uint32_t lane = lane_id();
    unsigned long long deg_sum = 0;
    uint32_t new_far = 0, touched = 0, max_deg = 0;
    stage_begin();
    if (threadIdx.x == 0) {
        s_sssp_newfar = 0;
        s_sssp_medges = 0;
        s_sssp_touched = 0;
        s_sssp_maxdeg = 0;
    }
    __syncthreads();
    for (uint64_t b0 = (uint64_t)blockIdx.x * kBlock * 4; b0 < V; b0 += (uint64_t)gridDim.x * kBlock * 4) {
        const uint32_t v0 = (uint32_t)b0 + 4 * threadIdx.x;
        uint32_t dv[4], sv[4], v[4];
        const bool whole = (uint64_t)v0 + 3 < V;
        if (whole) {
            const uint4 a = *reinterpret_cast<const uint4*>(dist + v0);
            const uint4 b = *reinterpret_cast<const uint4*>(snap + v0);
            dv[0] = a.x, dv[1] = a.y, dv[2] = a.z, dv[3] = a.w;
            sv[0] = b.x, sv[1] = b.y, sv[2] = b.z, sv[3] = b.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++) {
                dv[k] = v0 + k < V ? dist[v0 + k] : kValueMax;
                sv[k] = v0 + k < V ? snap[v0 + k] : kValueMax;
            }
        }
        if (dv[0] != sv[0] || dv[1] != sv[1] || dv[2] != sv[2] || dv[3] != sv[3]) {
            if (whole) {
                *reinterpret_cast<uint4*>(snap + v0) = make_uint4(dv[0], dv[1], dv[2], dv[3]);
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (v0 + k < V) snap[v0 + k] = dv[k];
            }
        }
        bool to_near[4];
        uint32_t far4 = 0, lo[4], hi[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = v0 + k;
            touched += (sv[k] == kValueMax && dv[k] < kValueMax) ? 1u : 0u;
            const bool imp = v[k] < nz && dv[k] < sv[k];
            to_near[k] = imp && dv[k] < thr;
            if (imp && !to_near[k]) far4 |= 1u << k;
            lo[k] = to_near[k] ? off[v[k]] : 0u;
            hi[k] = to_near[k] ? off[v[k] + 1] : 0u;
        }
        // lanes 8j .. 8j+7 hold the 32 vertices of bitmap word b0/32 + j
        uint32_t fm = far4 << (4 * (lane & 7u));
        fm |= __shfl_xor_sync(0xffffffffu, fm, 1);
        fm |= __shfl_xor_sync(0xffffffffu, fm, 2);
        fm |= __shfl_xor_sync(0xffffffffu, fm, 4);
        if ((lane & 7u) == 0 && fm) {
            const uint32_t wi = v0 >> 5;
            const uint32_t old = far_bm[wi];
            if (fm & ~old) {
                far_bm[wi] = old | fm;
                new_far += __popc(fm & ~old);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            deg_sum += hi[k] - lo[k];
            max_deg = max(max_deg, hi[k] - lo[k]);
        }
        stage_append_n<4>(to_near, v, near_out, near_len, cap, &ctr->overflow);
    }
    // one set of counter atomics per CTA
    deg_sum = warp_sum(deg_sum);
    touched = __reduce_add_sync(0xffffffffu, touched);
    new_far = __reduce_add_sync(0xffffffffu, new_far);
    max_deg = __reduce_max_sync(0xffffffffu, max_deg);
    if (lane == 0) {
        if (deg_sum) atomicAdd(&s_sssp_medges, deg_sum);
        if (new_far) atomicAdd(&s_sssp_newfar, new_far);
        if (touched) atomicAdd(&s_sssp_touched, touched);
        if (max_deg) atomicMax(&s_sssp_maxdeg, max_deg);
    }
    __syncthreads();
    stage_end(near_out, near_len, cap, &ctr->overflow);
    if (threadIdx.x == 0) {
        if (s_sssp_medges) atomicAdd(&ctr->medges, s_sssp_medges);
        if (s_sssp_newfar) atomicAdd(&ctr->far_len[0], s_sssp_newfar);
        if (s_sssp_touched) atomicAdd(&ctr->touched, s_sssp_touched);
        if (s_sssp_maxdeg) atomicMax(&ctr->max_deg, s_sssp_maxdeg);
    }
}

// Counters of the next round (and, for a push round, the near-dedup bitmap)
// reset by one launch instead of one memset each: rounds are short, and a
// run has dozens of them.
__global__ void k_sssp_round_reset(DevCounters* ctr, int out, uint32_t* bm, uint32_t words)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctr->qlen[out] = 0;
        ctr->chunk_len = 0;
        ctr->medges = 0;
        ctr->max_deg = 0;
    }
    if (bm)
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += gridDim.x * blockDim.x) bm[i] = 0;
}

// The same before a bucket split: next queue, far count, smallest far distance.
__global__ void k_sssp_split_reset(DevCounters* ctr, int out)
{
    ctr->qlen[out] = 0;
    ctr->far_len[0] = 0;
    ctr->min_far = 0xFFFFFFFFu;
    ctr->medges = 0;
    ctr->max_deg = 0;
}

__global__ void k_sssp_init(uint32_t V, uint32_t* dist, uint32_t* far_bm, uint32_t words, uint32_t root, uint32_t* q0)
{
    const uint32_t stride = gridDim.x * blockDim.x, i0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t i = i0; i < V; i += stride) dist[i] = i == root ? 0 : kValueMax;
    for (uint32_t i = i0; i < words; i += stride) far_bm[i] = 0;
    if (i0 == 0) q0[0] = root;
}

// Splits the far bitmap at [lo, hi) (see file comment).  A warp takes 32
// consecutive words with one coalesced load and visits the non-zero ones
// four at a time, lane b of word j reading the distance of vertex 32 * j + b
// (coalesced, four words in flight); the warp owns its words, so it writes
// back what stays without atomics.  far_len[0] receives the number of
// vertices left in the bitmap and min_far the smallest distance among them.
__global__ void __launch_bounds__(kBlock) k_sssp_split(uint32_t words, uint32_t* far_bm, const uint32_t* dist,
                                                       uint32_t lo, uint32_t hi, uint32_t* near_out,
                                                       uint32_t* near_len, uint32_t cap, DevCounters* ctr,
                                                       const uint32_t* __restrict__ off)
{
    constexpr int N = 4;
    const uint32_t lane = lane_id();
    const uint32_t gw = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    uint32_t mn = kValueMax, left = 0, max_deg = 0;
    unsigned long long dg = 0;
    for (uint32_t w0 = gw * 32; w0 < words; w0 += nwarps * 32) {
        const uint32_t mine = w0 + lane < words ? far_bm[w0 + lane] : 0u;
        uint32_t todo = __ballot_sync(0xffffffffu, mine != 0);
        while (todo) {
            uint32_t wi[N], bits[N], v[N], dv[N];
            bool in[N];
#pragma unroll
            for (int k = 0; k < N; k++) {
                const uint32_t j = todo ? __ffs(todo) - 1 : 32u;
                todo &= todo ? todo - 1 : 0u;
                bits[k] = j < 32 ? __shfl_sync(0xffffffffu, mine, j & 31u) : 0u;
                wi[k] = w0 + (j & 31u);
                v[k] = wi[k] * 32 + lane;
                in[k] = (bits[k] >> lane) & 1u;
            }
#pragma unroll
            for (int k = 0; k < N; k++) dv[k] = in[k] ? dist[v[k]] : 0u;
            bool to_near[N];
            uint32_t a[N], b[N];
#pragma unroll
            for (int k = 0; k < N; k++) {
                const bool leave = in[k] && dv[k] < hi;
                to_near[k] = leave && dv[k] >= lo;
                const bool keep = in[k] && !leave;
                if (keep) mn = min(mn, dv[k]);
                const uint32_t km = __ballot_sync(0xffffffffu, keep);
                if (lane == 0 && bits[k]) {
                    if (km != bits[k]) far_bm[wi[k]] = km;
                    left += __popc(km);
                }
                a[k] = to_near[k] ? off[v[k]] : 0u;
                b[k] = to_near[k] ? off[v[k] + 1] : 0u;
            }
#pragma unroll
            for (int k = 0; k < N; k++) {
                dg += b[k] - a[k];
                max_deg = max(max_deg, b[k] - a[k]);
            }
            warp_append_n<N>(to_near, v, near_out, near_len, cap, &ctr->overflow);
        }
    }
    mn = __reduce_min_sync(0xffffffffu, mn);
    dg = warp_sum(dg);
    max_deg = warp_max(max_deg);
    if (lane == 0) {
        if (mn != kValueMax) atomicMin(&ctr->min_far, mn);
        if (left) atomicAdd(&ctr->far_len[0], left);
        if (dg) atomicAdd(&ctr->medges, dg);
        if (max_deg) atomicMax(&ctr->max_deg, max_deg);
    }
}

// Near rounds smaller than this (and with fewer than E / 1024 out-edges)
// are neither sampled for the learned scheduler nor preceded by its
// inference: their variant hardly changes the run's time.
constexpr uint64_t kCollectMinRound = 4096;

template <bool kHasW>
static void sssp_loop(cgb_graph* g, uint32_t root, uint32_t delta, const cgb_options& o)
{
    const bool timing = g->flags & CGB_FLAG_KERNEL_TIMING;
    const bool tracing = g->flags & CGB_FLAG_TRACE;
    const uint32_t V = g->V;
    const uint32_t words = g->words();
    uint32_t* far_bm = g->front_bm;  // the BFS bitmaps are free during SSSP
    uint32_t* near_bm = g->visited;
    const uint64_t max_iters = o.max_iterations ? o.max_iterations : ~0ull;
    Policy* pol = (o.schedule == CGB_SCHED_LEARNED) ? policy_for(g) : nullptr;
    PolicySamples* collect = g->collect;
    const uint32_t base_delta = delta;

    CGB_CUDA_TRY(cudaEventRecord(g->ev_start, g->stream));
    if (timing) ktimer_begin(g, CGB_K_INIT);
    ++g->stats.launches;
    k_sssp_init<<<grid_for(V, kBlock, num_sms() * 4), kBlock, 0, g->stream>>>(V, g->value, far_bm, words, root,
                                                                           g->q[0]);
    if (timing) ktimer_end(g);

    int cur = 0;
    uint64_t nnear = root < g->nz ? 1 : 0;
    uint64_t nfar = 0;
    uint64_t thr = delta;
    uint64_t bucket_lo = 0;      // the current bucket is [bucket_lo, thr): every near vertex is in it
    uint64_t near_edges = 0;     // out-edges of the near queue (0 = unknown: push)
    uint32_t near_maxdeg = ~0u;  // longest list of the near queue (unknown for the root: its round runs here)
    double touch_rate = 0.0;     // vertices reached for the first time per edge, last push or dense round
    uint64_t touched_seen = 0;   // ctr->touched after that round
    // pull rounds need the in-edges (and their weights in CSC order)
    const bool pull_ok = o.schedule != CGB_SCHED_FIXED && g->tune.sssp_pull_alpha > 0;
    uint64_t iters = 0;
    uint64_t expanded = 0;

    // Device-resident rounds (persist.cuh).  The cluster loop takes near
    // queues of at most cluster_enter vertices and kClusterEnterEdges
    // out-edges on any graph (a hub's list is spread over the cluster).  The
    // grid loop takes up to persist_enter vertices on graphs whose lists are
    // all shorter than persist_deg edges; on others (power-law graphs) its
    // one-warp-per-list expansion walks medium lists slowly, and frontiers
    // outgrow its bounds bucket after bucket (RMAT-24: 6.9 against 5.2 ms a
    // run).  Both run near rounds and bucket splits until the run ends or a
    // frontier outgrows their bounds (then the rounds below take over again),
    // and keep the current delta for the buckets they split.  Under the
    // learned schedule the network picks that delta at the first bucket
    // boundary: until then the cluster loop returns there, and the grid loop
    // waits.
    const bool tail_allowed = !tracing && o.schedule != CGB_SCHED_FIXED && g->tune.persist_enter > 0;
    const bool grid_fits = tail_allowed && g->max_degree < g->tune.persist_deg;
    const bool cluster_fits = tail_allowed && g->tune.cluster_enter > 0 && cluster_loop_ctas() > 0;
    bool tail_delta_chosen = pol == nullptr;
    bool snapshot_ok = false;  // stamp[] holds the distances (dense rounds)
    enum { kNoTail, kClusterTail, kGridTail };
    auto tail_kind = [&]() {
        if (cluster_fits && nnear <= std::min(g->tune.cluster_enter, g->tune.persist_enter) &&
            near_edges <= kClusterEnterEdges && (nnear > 0 || nfar <= kClusterFar))
            return kClusterTail;
        if (grid_fits && tail_delta_chosen && nnear <= g->tune.persist_enter && near_maxdeg < g->tune.persist_deg) return kGridTail;
        return kNoTail;
    };
    // Runs the loop that takes the near queue (or, when it is empty, the next
    // split); false if none does or it ran no round.
    auto device_tail = [&]() -> bool {
        const int kind = tail_kind();
        if (kind == kNoTail) return false;
        snapshot_ok = false;
        const uint32_t max_rounds = (uint32_t)std::min<uint64_t>(max_iters - iters, 1u << 30);
        if (timing) ktimer_begin(g, CGB_K_PUSH);
        const SsspTail t =
            kind == kClusterTail
                ? sssp_cluster(g, cur, (uint32_t)nnear, thr, (uint32_t)nfar, bucket_lo, far_bm, delta,
                               std::min(g->tune.persist_enter, 2 * g->tune.cluster_enter), kClusterExitEdges,
                               tail_delta_chosen ? kClusterFar : 0, std::min(max_rounds, g->cluster_rounds))
                : sssp_device_tail(g, cur, (uint32_t)nnear, near_maxdeg, thr, (uint32_t)nfar, bucket_lo, far_bm, delta,
                                   g->tune.persist_enter, g->tune.persist_deg, max_rounds);
        if (timing) ktimer_end(g);
        iters += t.r.levels;
        expanded += t.r.added;
        nnear = t.r.nf;
        if (t.r.levels > 0) near_maxdeg = t.r.max_deg;
        nfar = t.nfar;
        thr = t.thr;
        bucket_lo = t.bucket_lo;
        near_edges = t.r.scout;  // 0 (unknown) from the grid loop: push next
        cur = (int)t.r.cur;
        return t.r.levels > 0;
    };
    // Queues one near round of the given RoundVariant, next near queue to q[out].
    auto run_round = [&](int variant, int out) {
        const bool pull = variant == kRoundPull, dense = variant == kRoundDense;
        if (pull) {
            ensure_csc(g);
            ensure_csc_weights(g);
        }
        ++g->stats.launches;
        k_sssp_round_reset<<<(!pull && !dense) ? num_sms() * 2 : 1, kBlock, 0, g->stream>>>(
            g->ctr, out, (!pull && !dense) ? near_bm : nullptr, words);
        if (timing) ktimer_begin(g, pull ? CGB_K_PULL : CGB_K_PUSH);
        if (pull) {
            sssp_pull_round(g, g->q[cur], (uint32_t)nnear, (uint32_t)std::min<uint64_t>(bucket_lo, kValueMax),
                            (uint32_t)std::min<uint64_t>(thr, kValueMax), g->q[out], &g->ctr->qlen[out], far_bm,
                            g->aux_bm);
        } else if (dense) {
            // the scan of a dense round leaves the snapshot up to date for the next one
            if (!snapshot_ok)
                CGB_CUDA_TRY(cudaMemcpyAsync(g->stamp, g->value, (size_t)V * 4, cudaMemcpyDeviceToDevice, g->stream));
            SsspDenseOp<kHasW> op{g->off, g->dst, g->w, g->value};
            launch_push(g, g->q[cur], (uint32_t)nnear, op, false);
            ++g->stats.launches;
            k_sssp_dense_scan<<<grid_for(div_up(V, 4), kBlock, num_sms() * 8), kBlock, stage_bytes(kBlock),
                                g->stream>>>(
                V, g->value, g->stamp, (uint32_t)std::min<uint64_t>(thr, kValueMax), g->nz, g->off, far_bm,
                g->q[out], &g->ctr->qlen[out], V, g->ctr);
        } else {
            SsspOp<kHasW> op{g->off, g->dst, g->w, g->value, near_bm,
                             (uint32_t)std::min<uint64_t>(thr, kValueMax), g->nz, g->q[out], &g->ctr->qlen[out],
                             V, far_bm, g->ctr};
            launch_push(g, g->q[cur], (uint32_t)nnear, op, false,
                        variant == kRoundPushChunked ? kExpandChunked : kExpandBinned);
        }
        if (timing) ktimer_end(g);
        snapshot_ok = dense && !collect;  // (the trials of a sample restore the distances)
    };
    int last_variant = kRoundPush;
    bool have_round_out = false;  // the policy's outputs for the next round were read back
    // set while a bucket phase runs as one of the delta trials of a sample:
    // its rounds are not sampled themselves (the trial's timing events must
    // span the whole phase)
    bool in_delta_trial = false;
    auto round_state = [&]() {
        FeatIn in{};
        in.alg = CGB_SSSP;
        in.iteration = (uint32_t)iters;
        in.prev_dir = last_variant;
        in.symmetric = g->symmetric == 1;
        in.V = V;
        in.E = g->E;
        in.nf = (double)nnear;
        in.mf = (double)near_edges;
        in.max_deg = near_maxdeg == ~0u ? 0.0 : (double)near_maxdeg;
        in.unvisited_v = (double)V - (double)g->h_ctr->touched;
        in.unvisited_e = (double)near_edges * touch_rate;  // improvements the round is expected to make
        in.delta = delta;
        in.base_delta = base_delta;
        in.far_count = (double)nfar;
        in.settled = (double)std::min<uint64_t>(expanded, V);
        return in;
    };
    // Near rounds at threshold thr until the near queue is empty.
    auto near_rounds = [&]() {
        while (nnear > 0) {
            CGB_REQUIRE(iters < max_iters, CGB_ETIMEOUT, "SSSP iteration budget exhausted");
            if (!collect && device_tail()) {
                have_round_out = false;
                continue;
            }
            const int out = cur ^ 1;
            // heuristic: pull when the near set's out-edges times alpha exceed the graph's
            // edges; else a dense frontier when they are many for what the round will change.
            // A push round pays an atomic with a returned value and a queue append per
            // improvement, a dense round a reduction per edge plus one pass over V.  While the
            // search reaches new territory nearly every edge improves its target, so the
            // out-edges are weighted by the previous round's first touches per edge, floored at
            // 1/8 for the rounds that mostly lower known distances.  A push round chunks every
            // list of 32 edges or more when its queue is small.
            const bool h_pull = pull_ok && (double)near_edges * g->tune.sssp_pull_alpha > (double)g->E;
            const bool h_dense = !h_pull && o.schedule != CGB_SCHED_FIXED && g->tune.sssp_dense_alpha > 0 &&
                                 (double)near_edges * g->tune.sssp_dense_alpha * std::max(touch_rate, 0.125) >
                                     (double)V;
            const int heur = h_pull ? kRoundPull
                             : h_dense ? kRoundDense
                                       : (nnear <= kSmallFrontier ? kRoundPushChunked : kRoundPush);
            int variant = heur;
            if (collect && !in_delta_trial && (nnear >= kCollectMinRound || near_edges >= g->E / 1024)) {
                // counterfactual: the four round variants from the same state, timed
                ensure_csc(g);
                ensure_csc_weights(g);
                const size_t vbytes = (size_t)V * 4, wbytes = (size_t)words * 4, qbytes = nnear * 4;
                CGB_CUDA_TRY(cudaMemcpyAsync(collect->save_value, g->value, vbytes, cudaMemcpyDeviceToDevice,
                                             g->stream));
                CGB_CUDA_TRY(cudaMemcpyAsync(collect->save_bm0, far_bm, wbytes, cudaMemcpyDeviceToDevice, g->stream));
                CGB_CUDA_TRY(cudaMemcpyAsync(collect->save_q, g->q[cur], qbytes, cudaMemcpyDeviceToDevice,
                                             g->stream));
                CGB_CUDA_TRY(cudaMemcpyAsync(collect->save_ctr, g->ctr, sizeof(DevCounters),
                                             cudaMemcpyDeviceToDevice, g->stream));
                float ms[kPolicyOutputs] = {};
                bool have[kPolicyOutputs] = {};
                int best = heur;
                // every trial starts right after a restore, the first one too (the
                // snapshot copy alone leaves dist[] colder in L2 for the first)
                CGB_CUDA_TRY(cudaMemcpyAsync(g->value, collect->save_value, vbytes, cudaMemcpyDeviceToDevice,
                                             g->stream));
                CGB_CUDA_TRY(cudaMemcpyAsync(far_bm, collect->save_bm0, wbytes, cudaMemcpyDeviceToDevice, g->stream));
                for (int v = 0; v < kNumRoundChoices; v++) {
                    CGB_CUDA_TRY(cudaEventRecord(g->ev_iter[0], g->stream));
                    run_round(v, out);
                    CGB_CUDA_TRY(cudaEventRecord(g->ev_iter[1], g->stream));
                    CGB_CUDA_TRY(cudaEventSynchronize(g->ev_iter[1]));
                    CGB_CUDA_TRY(cudaEventElapsedTime(&ms[kOutRound0 + v], g->ev_iter[0], g->ev_iter[1]));
                    have[kOutRound0 + v] = true;
                    if (ms[kOutRound0 + v] < ms[kOutRound0 + best]) best = v;
                    CGB_CUDA_TRY(cudaMemcpyAsync(g->value, collect->save_value, vbytes, cudaMemcpyDeviceToDevice,
                                                 g->stream));
                    CGB_CUDA_TRY(cudaMemcpyAsync(far_bm, collect->save_bm0, wbytes, cudaMemcpyDeviceToDevice,
                                                 g->stream));
                    CGB_CUDA_TRY(cudaMemcpyAsync(g->q[cur], collect->save_q, qbytes, cudaMemcpyDeviceToDevice,
                                                 g->stream));
                    CGB_CUDA_TRY(cudaMemcpyAsync(g->ctr, collect->save_ctr, sizeof(DevCounters),
                                                 cudaMemcpyDeviceToDevice, g->stream));
                }
                policy_log_sample(g, round_state(), ms, have);
                variant = best;
            } else if (pol && have_round_out) {
                const int c = policy_pick_round(g->h_ctr->policy_out, heur);
                if (c >= 0) variant = c;
            }
            if (tracing) CGB_CUDA_TRY(cudaEventRecord(g->ev_iter[0], g->stream));
            const FeatIn before = round_state();
            run_round(variant, out);
            if (variant == kRoundPull) g->stats.pulls_bu++;
            else g->stats.pushes_td++;
            if (tracing) CGB_CUDA_TRY(cudaEventRecord(g->ev_iter[1], g->stream));
            // inference for the next round, fused before the counter read-back; skipped
            // after small rounds, whose successors' variant hardly matters
            const bool infer =
                kPolicyRounds && pol && !collect && (nnear >= kCollectMinRound || near_edges >= g->E / 1024);
            if (infer) policy_enqueue(pol, g, before, 2, false, out);
            have_round_out = infer;
            last_variant = variant;
            sync_counters(g);
            CGB_REQUIRE(!g->h_ctr->overflow, CGB_EOVERFLOW, "SSSP queue overflow");
            if (tracing) {
                float ms = 0.f;
                CGB_CUDA_TRY(cudaEventElapsedTime(&ms, g->ev_iter[0], g->ev_iter[1]));
                cgb_iter_trace t{};
                t.iteration = (uint32_t)iters;
                t.algorithm = CGB_SSSP;
                t.frontier_vertices = nnear;
                t.unvisited_vertices = g->h_ctr->far_len[0];
                t.variant = variant == kRoundPull ? CGB_VAR_PULL : variant == kRoundDense ? CGB_VAR_DENSE : CGB_VAR_TWC;
                t.frontier_edges = near_edges;
                t.delta = delta;
                t.ms = ms;
                g->trace.push_back(t);
            }
            expanded += nnear;
            if (variant != kRoundPull && near_edges > 0) {
                touch_rate = (double)(g->h_ctr->touched - touched_seen) / (double)near_edges;
                touched_seen = g->h_ctr->touched;
            }
            nnear = g->h_ctr->qlen[out];
            nfar = g->h_ctr->far_len[0];
            near_edges = g->h_ctr->medges;
            near_maxdeg = g->h_ctr->max_deg;
            cur = out;
            iters++;
        }
    };
    // Next bucket [thr, thr + d): split the far bitmap (jumping over empty
    // buckets) until the near queue is non-empty or the bitmap is empty.
    auto advance = [&](uint32_t d) {
        uint64_t lo = thr;
        thr += d;
        for (;;) {
            CGB_REQUIRE(iters < max_iters, CGB_ETIMEOUT, "SSSP iteration budget exhausted");
            const int out = cur ^ 1;
            ++g->stats.launches;
            k_sssp_split_reset<<<1, 1, 0, g->stream>>>(g->ctr, out);
            if (timing) ktimer_begin(g, CGB_K_FRONTIER);
            ++g->stats.launches;
            k_sssp_split<<<grid_for(words, kBlock, num_sms() * 4), kBlock, 0, g->stream>>>(
                words, far_bm, g->value, (uint32_t)std::min<uint64_t>(lo, kValueMax),
                (uint32_t)std::min<uint64_t>(thr, kValueMax), g->q[out], &g->ctr->qlen[out], V, g->ctr, g->off);
            if (timing) ktimer_end(g);
            sync_counters(g);
            CGB_REQUIRE(!g->h_ctr->overflow, CGB_EOVERFLOW, "SSSP queue overflow");
            nnear = g->h_ctr->qlen[out];
            nfar = g->h_ctr->far_len[0];
            near_edges = g->h_ctr->medges;
            near_maxdeg = g->h_ctr->max_deg;
            cur = out;
            iters++;
            bucket_lo = lo;
            if (nnear > 0 || nfar == 0) break;
            // every vertex left is at or above thr: jump to the bucket of the smallest
            const uint64_t mn = g->h_ctr->min_far;
            lo = thr;
            thr = (mn / d + 1) * (uint64_t)d;
        }
    };
    auto state_now = [&]() {
        FeatIn in{};
        in.alg = CGB_SSSP;
        in.iteration = (uint32_t)iters;
        in.symmetric = g->symmetric == 1;
        in.V = V;
        in.E = g->E;
        in.nf = (double)nnear;
        in.unvisited_v = (double)V - (double)std::min<uint64_t>(expanded, V);
        in.delta = delta;
        in.base_delta = base_delta;
        in.far_count = (double)nfar;
        in.settled = (double)std::min<uint64_t>(expanded, V);
        return in;
    };

    // The learned (or collected) delta is chosen once, at the first bucket
    // boundary, for the rest of the run: a counterfactual trial runs the whole
    // remainder of the run with each candidate, so the sample's costs include
    // everything a narrower or wider bucket changes later (a trial of one
    // bucket phase saw only that phase).
    bool delta_decided = false;
    near_rounds();
    while (nfar > 0) {
        uint32_t d = delta;
        if (collect && !delta_decided) {
            const size_t vbytes = (size_t)V * 4, wbytes = (size_t)words * 4;
            CGB_CUDA_TRY(cudaMemcpyAsync(collect->save_value, g->value, vbytes, cudaMemcpyDeviceToDevice, g->stream));
            CGB_CUDA_TRY(cudaMemcpyAsync(collect->save_bm0, far_bm, wbytes, cudaMemcpyDeviceToDevice, g->stream));
            const uint64_t s_thr = thr, s_iters = iters, s_exp = expanded, s_far = nfar, s_lo = bucket_lo;
            const int s_cur = cur;
            float ms[kPolicyOutputs] = {};
            bool have[kPolicyOutputs] = {};
            int best = kDeltaUnit;
            in_delta_trial = true;
            CGB_CUDA_TRY(cudaMemcpyAsync(g->value, collect->save_value, vbytes, cudaMemcpyDeviceToDevice, g->stream));
            CGB_CUDA_TRY(cudaMemcpyAsync(far_bm, collect->save_bm0, wbytes, cudaMemcpyDeviceToDevice, g->stream));
            for (int k = 0; k < kNumDeltaChoices; k++) {
                const uint32_t dk = std::max<uint32_t>(1u, (uint32_t)(base_delta * delta_scale(k)));
                CGB_CUDA_TRY(cudaEventRecord(g->ev_iter[0], g->stream));
                // the rest of the run as a run with this delta would go, the
                // device-resident tail included (it changes what a round costs)
                delta = dk;
                do {
                    near_maxdeg = 0;
                    near_edges = 0;
                    if (device_tail()) {
                        near_rounds();
                        continue;
                    }
                    advance(dk);
                    near_rounds();
                } while (nfar > 0);
                CGB_CUDA_TRY(cudaEventRecord(g->ev_iter[1], g->stream));
                CGB_CUDA_TRY(cudaEventSynchronize(g->ev_iter[1]));
                float t = 0.f;
                CGB_CUDA_TRY(cudaEventElapsedTime(&t, g->ev_iter[0], g->ev_iter[1]));
                ms[kOutDelta0 + k] = t;  // the rest of the run
                have[kOutDelta0 + k] = true;
                if (ms[kOutDelta0 + k] < ms[kOutDelta0 + best]) best = k;
                CGB_CUDA_TRY(cudaMemcpyAsync(g->value, collect->save_value, vbytes, cudaMemcpyDeviceToDevice,
                                             g->stream));
                CGB_CUDA_TRY(cudaMemcpyAsync(far_bm, collect->save_bm0, wbytes, cudaMemcpyDeviceToDevice, g->stream));
                thr = s_thr;
                iters = s_iters;
                expanded = s_exp;
                nfar = s_far;
                bucket_lo = s_lo;
                nnear = 0;
                cur = s_cur;
                delta = base_delta;
            }
            in_delta_trial = false;
            policy_log_sample(g, state_now(), ms, have);
            d = std::max<uint32_t>(1u, (uint32_t)(base_delta * delta_scale(best)));
            delta_decided = true;
        } else if (pol && !delta_decided) {
            policy_enqueue(pol, g, state_now(), 0, false, 0);
            sync_counters(g);
            const int k = policy_pick_delta(g->h_ctr->policy_out);
            if (k >= 0) d = std::max<uint32_t>(1u, (uint32_t)(base_delta * delta_scale(k)));
            delta_decided = true;
        }
        delta = d;
        tail_delta_chosen = true;
        if (!collect) {
            // the next bucket's split, and what follows, on the device
            near_maxdeg = 0;
            near_edges = 0;
            if (device_tail()) {
                near_rounds();
                continue;
            }
        }
        advance(d);
        near_rounds();
    }
    CGB_CUDA_TRY(cudaEventRecord(g->ev_stop, g->stream));
    g->stats.iterations = iters;
    g->stats.sssp_delta = delta;
}

// c x (mean weight / mean out-degree), in [1, 1e8].  A single-root run
// takes c = 128: fixed-delta sweeps over RMAT-20/22/24 (edge factors 4 and
// 16), 1000^2 and 4800 x 5000 grids and a Chung-Lu graph put the best delta
// at 64-2048 x the unit, and 128 was within 6 % of the best on all but
// Chung-Lu (22 %), where 64 was best.  Graph batches keep c = 8 and
// multi-root passes 64.
uint32_t sssp_delta_for(const cgb_graph* g, double c)
{
    if (g->E == 0 || g->V == 0) return 1;
    const double mean_w = g->w ? (double)g->sum_w / (double)g->E : 1.0;
    const double mean_deg = (double)g->E / (double)g->V;
    double d = c * mean_w / std::max(1.0, mean_deg);
    if (d < 1.0) d = 1.0;
    if (d > 1e8) d = 1e8;
    return (uint32_t)d;
}

// Graphs without hubs (no list of kMeshDeg edges) of kMeshLarge vertices or
// more whose edge lengths differ take c = 64: on meshes their near sets grow
// with the bucket and the graph's width, and the cluster loop's 16 SMs are
// full from a few thousand vertices on.  Where all lengths are equal a bucket
// is a few whole levels, a wider one saves splits and relaxes no edge twice:
// they keep 128, on meshes and random graphs alike.  (Equal lengths show in
// the sum alone: a mean that is a whole number.  Lengths that differ and have
// such a mean just keep 128.)  c = 128 / 64, ms:
//                          lengths 1 .. 1000    all equal
//   700 x 901 grid             5.61 /  5.16     3.67 / 3.81
//   1000^2                     8.54 /  7.88     5.49 / 5.72
//   3000^2                     80.9 /  45.0     25.2 / 27.9
//   4800 x 5000                 154 /   145     57.1 / 66.4
//   100 x 20000                91.2 /  96.3     60.3 / 62.5
//   200^3                      17.8 /  17.1     9.99 / 11.2
//   random, 2^19 x 16          3.02 /  3.17     0.63 / 0.80
//   random, 2^23 x 4           5.38 /  5.45     1.96 / 2.00
//   random, 2^23 x 8           8.52 /  8.54     2.16 / 3.12
constexpr uint32_t kMeshDeg = 64, kMeshLarge = 1u << 19;

uint32_t sssp_default_delta(const cgb_graph* g)
{
    const bool lengths_differ = g->w && g->E && g->sum_w % g->E != 0;
    return sssp_delta_for(g, g->max_degree < kMeshDeg && g->V >= kMeshLarge && lengths_differ ? 64.0 : 128.0);
}

void run_sssp(cgb_graph* g, uint32_t root, const cgb_options& o)
{
    ensure_frontier(g);
    if (g->w && g->sum_w == 0) compute_weight_sum(g);
    const uint32_t delta = o.sssp_delta ? o.sssp_delta : sssp_default_delta(g);
    if (g->w) sssp_loop<true>(g, root, delta, o);
    else sssp_loop<false>(g, root, delta, o);
}

}  // namespace cgb
