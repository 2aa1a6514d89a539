// Direction-optimising BFS.
//
// Result semantics follow the reference's BFS: level[root] = 0, a vertex's
// level is its parent's + 1, unreachable vertices keep 999999999
// (my_project/CGgraph/GraphDevice.cuh:224-235, device_algorithm.cuh:85-119).
// The reference pushes with atomicMin until no value changes; this engine
// runs level-synchronously, which reaches the same fixpoint:
//   top-down  -- push from a vertex queue with the degree-binned expansion of
//                push.cuh; a visited bitmap (V/32 words, L2-resident) filters
//                before one atomicOr claims a vertex, so each vertex is
//                written and enqueued exactly once;
//   bottom-up -- every unvisited vertex scans its in-edges (the CSC) until it
//                finds a parent in the frontier bitmap; one warp owns 32
//                consecutive vertices = one bitmap word, so visited and next-
//                frontier words are written without atomics.
// The direction switch is Beamer's (alpha = 15, beta = 18) unless the
// schedule says otherwise.
#include "engine.cuh"
#include "persist.cuh"
#include "policy.cuh"
#include "push.cuh"

namespace cgb {

// Per-CTA accumulators of the top-down op (flushed once per CTA).
__shared__ unsigned long long s_td_medges;
__shared__ uint32_t s_td_maxdeg;
__shared__ uint32_t s_bu_found;  // bottom-up

struct BfsTdOp {
    const uint32_t* __restrict__ off;
    const uint32_t* __restrict__ dst;
    uint32_t* level;
    uint32_t* visited;
    uint32_t next_level;
    uint32_t nz;
    uint32_t* qout;
    uint32_t* qlen;
    uint32_t cap;
    DevCounters* ctr;
    uint32_t t_edges = 0, t_maxdeg = 0;  // of the vertices this thread claimed
    static constexpr bool kStaged = true;
    static constexpr int kBatch = 4;  // edge slots per lane visited together (push.cuh)

    __device__ __forceinline__ bool load(uint32_t v, uint32_t& s, uint32_t& d, uint32_t& m) const
    {
        s = off[v];
        d = off[v + 1] - s;
        m = 0;
        return true;
    }
    template <int N>
    __device__ __forceinline__ void edges(const bool (&valid)[N], const uint32_t (&e)[N], const uint32_t (&)[N])
    {
        uint32_t d[N], word[N], bit[N], lo[N], hi[N];
        bool win[N], enq[N];
#pragma unroll
        for (int i = 0; i < N; i++) d[i] = valid[i] ? __ldcs(dst + e[i]) : 0u;  // streamed once: evict first
#pragma unroll
        for (int i = 0; i < N; i++) {
            bit[i] = 1u << (d[i] & 31u);
            word[i] = valid[i] ? visited[d[i] >> 5] : ~0u;
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            win[i] = false;
            if (!(word[i] & bit[i])) win[i] = !(atomicOr(visited + (d[i] >> 5), bit[i]) & bit[i]);
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            if (win[i]) level[d[i]] = next_level;
            enq[i] = win[i] && d[i] < nz;
            lo[i] = enq[i] ? off[d[i]] : 0u;
            hi[i] = enq[i] ? off[d[i] + 1] : 0u;
        }
        stage_append_n<N>(enq, d, qout, qlen, cap, &ctr->overflow);
#pragma unroll
        for (int i = 0; i < N; i++) {
            t_edges += hi[i] - lo[i];
            t_maxdeg = max(t_maxdeg, hi[i] - lo[i]);
        }
    }
    __device__ __forceinline__ void edge(bool valid, uint32_t e, uint32_t m)
    {
        const bool v[1] = {valid};
        const uint32_t ee[1] = {e}, mm[1] = {m};
        edges<1>(v, ee, mm);
    }
    __device__ __forceinline__ void block_begin() const
    {
        stage_begin();
        if (threadIdx.x == 0) {
            s_td_medges = 0;
            s_td_maxdeg = 0;
        }
    }
    __device__ __forceinline__ void block_end() const
    {
        const uint32_t sum = __reduce_add_sync(0xffffffffu, t_edges);  // at most E < 2^32
        const uint32_t mx = __reduce_max_sync(0xffffffffu, t_maxdeg);
        if (lane_id() == 0 && sum) {
            atomicAdd(&s_td_medges, (unsigned long long)sum);
            atomicMax(&s_td_maxdeg, mx);
        }
        stage_end(qout, qlen, cap, &ctr->overflow);  // a CTA barrier is inside
        if (threadIdx.x == 0 && s_td_medges) {
            atomicAdd(&ctr->medges, s_td_medges);
            atomicMax(&ctr->max_deg, s_td_maxdeg);
        }
    }
};

__global__ void k_bfs_init(uint32_t V, uint32_t* level, uint32_t* visited, uint32_t words, uint32_t root, uint32_t* q0)
{
    const uint32_t stride = gridDim.x * blockDim.x, i0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t i = i0; i < V; i += stride) level[i] = i == root ? 0 : kValueMax;
    for (uint32_t i = i0; i < words; i += stride) visited[i] = i == root >> 5 ? 1u << (root & 31u) : 0;
    if (i0 == 0) q0[0] = root;
}

// Queue -> frontier bitmap (bitmap cleared beforehand).
__global__ void k_q2bm(const uint32_t* __restrict__ q, uint32_t n, uint32_t* bm)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t v = q[i];
        atomicOr(bm + (v >> 5), 1u << (v & 31u));
    }
}

// Few staged items a warp: what the stage takes of an SM's memory L1 lacks,
// from which lanes read the lists that they walk.  Every level pulled, 2^20
// vertices of 30 edges: 256 items 2.40 ms, 128 1.91, 64 1.75, 32 1.76 (with
// a CTA's finds appended together, without a stage, 1.78); RMAT-20 12.7,
// 12.1, 11.3, 11.3 (10.5).
constexpr uint32_t kBuStage = 64;

// One bottom-up level.  Reads front (current frontier bitmap), writes
// next (all words, so it needs no clearing) and the next queue.  A warp takes
// one bitmap word per step, and warps share nothing between steps (finds are
// staged, push.cuh): what bounds the level is each warp's chain of dependent
// loads, so no warp waits for another's.  Each lane scans its vertex's
// in-list four entries at a time: four source loads, then their four
// frontier words, are in flight together, and the scan stops after the group
// that holds a parent.
__global__ void __launch_bounds__(kBlock) k_bfs_bu(uint32_t V, const uint32_t* __restrict__ in_off,
                                                   const uint32_t* __restrict__ in_src,
                                                   const uint32_t* __restrict__ off, uint32_t* level,
                                                   uint32_t* visited, const uint32_t* __restrict__ front,
                                                   uint32_t* next, uint32_t next_level, uint32_t nz, uint32_t* qout,
                                                   uint32_t* qlen, uint32_t cap, DevCounters* ctr)
{
    const uint32_t words = (V + 31) / 32, lane = lane_id();
    const uint32_t warps = gridDim.x * (kBlock / 32);
    uint32_t medges = 0, found_cnt = 0, mx = 0;
    stage_begin();
    if (threadIdx.x == 0) {
        s_td_medges = 0;
        s_td_maxdeg = 0;
        s_bu_found = 0;
    }
    __syncthreads();
    for (uint32_t wi = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); wi < words; wi += warps) {
        const uint32_t v = wi * 32 + lane;
        const uint32_t vis = visited[wi];
        uint32_t fm = 0;
        if (vis != 0xFFFFFFFFu) {
            bool found = false;
            if (v < V && !((vis >> lane) & 1u)) {
                const uint32_t e1 = in_off[v + 1];
                for (uint32_t e = in_off[v]; e < e1 && !found; e += 4) {
                    uint32_t u[4], f[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) u[k] = e + k < e1 ? in_src[e + k] : in_src[e];
#pragma unroll
                    for (int k = 0; k < 4; k++) f[k] = front[u[k] >> 5] >> (u[k] & 31u);
#pragma unroll
                    for (int k = 0; k < 4; k++) found |= (f[k] & 1u) != 0;
                }
            }
            fm = __ballot_sync(0xffffffffu, found);
            if (fm) {
                if (found) level[v] = next_level;
                const bool enq[1] = {found && v < nz};
                const uint32_t deg = enq[0] ? off[v + 1] - off[v] : 0;
                medges += deg;
                found_cnt += enq[0];
                mx = max(mx, deg);
                const uint32_t it[1] = {v};
                stage_append_n<1, kBuStage>(enq, it, qout, qlen, cap, &ctr->overflow);
            }
        }
        if (lane == 0) {
            next[wi] = fm;
            if (fm) visited[wi] = vis | fm;
        }
    }
    // one set of counter atomics per CTA: per warp, they were 38 us of a level
    const uint32_t warp_edges = __reduce_add_sync(0xffffffffu, medges);  // at most E < 2^32
    found_cnt = __reduce_add_sync(0xffffffffu, found_cnt);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0 && found_cnt) {
        atomicAdd(&s_td_medges, (unsigned long long)warp_edges);
        atomicAdd(&s_bu_found, found_cnt);
        atomicMax(&s_td_maxdeg, mx);
    }
    __syncthreads();
    stage_end<kBuStage>(qout, qlen, cap, &ctr->overflow);
    if (threadIdx.x == 0 && s_bu_found) {
        atomicAdd(&ctr->medges, s_td_medges);
        atomicAdd(&ctr->found, s_bu_found);
        atomicMax(&ctr->max_deg, s_td_maxdeg);
    }
}

__global__ void k_level_reset(DevCounters* ctr, int out)
{
    ctr->qlen[out] = 0;
    ctr->chunk_len = 0;
    ctr->medges = 0;
    ctr->found = 0;
    ctr->max_deg = 0;
}

// qlen[out], chunk_len, medges, found, max_deg: one launch, not five memsets
static void reset_level_counters(cgb_graph* g, int out)
{
    ++g->stats.launches;
    k_level_reset<<<1, 1, 0, g->stream>>>(g->ctr, out);
}

// A graph of at most this many edges runs in the cluster from start to end,
// all levels pushed: no host round trips, but 16 of the SMs and no pulls.
// Bounds of 2^18 / 2^19 / 2^20 edges, mean of 5 roots, us:
//   Chung-Lu, 280 k edges                         200 / 107 / 107
//   random, 2^13 vertices of 60, 490 k edges      105 / 119 / 119
//   random, 2^18 vertices of 2, 524 k             448 / 260 / 257
//   Chung-Lu, 546 k                               225 / 229 / 158
//   random, 2^10 vertices of 554, 568 k            81 /  82 / 120
//   random, 2^11 vertices of 444, 908 k            85 /  87 / 156
//   RMAT-16, 955 k                                149 / 147 / 191
//   random, 2^16 vertices of 15, 983 k            184 / 176 / 203
//   random, 2^18 vertices of 4, 1049 k            290 / 302 / 284
// A list beyond kClusterList ends the loop, and the run would come back to it
// for nothing: such a graph takes the rule for small frontiers.
constexpr uint32_t kClusterWholeEdges = 1u << 19;

void run_bfs(cgb_graph* g, uint32_t root, const cgb_options& o)
{
    ensure_frontier(g);
    const bool want_pull = !(o.schedule == CGB_SCHED_FIXED && o.variant != CGB_VAR_PULL && o.variant != CGB_VAR_AUTO);
    const bool force_pull = (o.schedule == CGB_SCHED_FIXED && o.variant == CGB_VAR_PULL);
    if (want_pull) ensure_csc(g);
    const double alpha = o.bfs_alpha > 0 ? o.bfs_alpha : 15.0;
    const double beta = o.bfs_beta > 0 ? o.bfs_beta : 18.0;
    const uint32_t V = g->V;
    const uint32_t words = g->words();
    const bool timing = g->flags & CGB_FLAG_KERNEL_TIMING;
    const bool tracing = g->flags & CGB_FLAG_TRACE;
    PolicySamples* collect = want_pull && !force_pull ? g->collect : nullptr;
    Policy* pol = (o.schedule == CGB_SCHED_LEARNED && want_pull && !force_pull) ? policy_for(g) : nullptr;

    // device-resident levels for small frontiers (not while collecting
    // samples, which time each level's variants on the host)
    const bool persist_ok = !tracing && !collect && o.schedule != CGB_SCHED_FIXED;
    const bool cluster_ok =
        persist_ok && g->tune.persist_enter > 0 && g->tune.cluster_enter > 0 && cluster_loop_ctas() > 0;
    // the root's out-degree, which the cluster loop finds out for itself
    uint64_t scout = 0;
    if (!cluster_ok) {
        PinnedArray<uint32_t> host_root_deg(2);  // pinned: see pinned_acquire
        CGB_CUDA_TRY(cudaMemcpyAsync(host_root_deg.data(), g->off + root, 2 * sizeof(uint32_t),
                                     cudaMemcpyDeviceToHost, g->stream));
        CGB_CUDA_TRY(cudaStreamSynchronize(g->stream));
        scout = host_root_deg[1] - host_root_deg[0];
    }
    CGB_CUDA_TRY(cudaEventRecord(g->ev_start, g->stream));
    if (timing) ktimer_begin(g, CGB_K_INIT);
    ++g->stats.launches;
    k_bfs_init<<<grid_for(V, kBlock, num_sms() * 4), kBlock, 0, g->stream>>>(V, g->value, g->visited, words, root,
                                                                          g->q[0]);
    if (timing) ktimer_end(g);

    uint32_t cur = 0;  // queue holding the current frontier
    uint64_t nf = (root < g->nz) ? 1 : 0;
    uint64_t prev_nf = 0;
    int64_t edges_to_check = (int64_t)g->E;
    uint32_t maxdeg = (uint32_t)scout;
    uint64_t visited_cnt = 1;
    uint32_t level = 0;
    bool bottom_up = false;
    bool have_policy_out = false;
    uint64_t awake = 0, old_awake = 0;
    uint32_t* front = g->front_bm;
    uint32_t* next = g->front_bm + words;
    uint64_t iters = 0;
    const uint64_t max_iters = o.max_iterations ? o.max_iterations : (uint64_t)V + 2;

    // Queues one level in the given direction (frontier in q[cur] and, when
    // the last level was pulled, in `front`; next frontier to q[out] / next);
    // a push level with the given expansion variant (PushExpand).
    auto do_level = [&](bool pull, int out, int expand) {
        reset_level_counters(g, out);
        if (pull) {
            if (!bottom_up) {
                // entering bottom-up: frontier queue -> bitmap
                if (timing) ktimer_begin(g, CGB_K_FRONTIER);
                CGB_CUDA_TRY(cudaMemsetAsync(front, 0, words * sizeof(uint32_t), g->stream));
                ++g->stats.launches;
                k_q2bm<<<grid_for(nf, kBlock, num_sms() * 8), kBlock, 0, g->stream>>>(g->q[cur], (uint32_t)nf, front);
                if (timing) ktimer_end(g);
            }
            if (timing) ktimer_begin(g, CGB_K_PULL);
            const uint32_t grid = grid_for((uint64_t)words * 32, kBlock, num_sms() * 16);
            ++g->stats.launches;
            k_bfs_bu<<<grid, kBlock, stage_bytes(kBlock, kBuStage), g->stream>>>(V, g->in_off, g->in_src, g->off, g->value, g->visited, front,
                                                     next, level + 1, g->nz, g->q[out], &g->ctr->qlen[out], V,
                                                     g->ctr);
            if (timing) ktimer_end(g);
        } else {
            if (timing) ktimer_begin(g, CGB_K_PUSH);
            BfsTdOp op{g->off, g->dst, g->value, g->visited, level + 1, g->nz, g->q[out], &g->ctr->qlen[out], V, g->ctr};
            launch_push(g, g->q[cur], (uint32_t)nf, op, false, expand);
            if (timing) ktimer_end(g);
        }
    };
    auto state_now = [&]() {
        FeatIn in{};
        in.alg = CGB_BFS;
        in.iteration = level;
        in.prev_dir = bottom_up ? 1 : 0;
        in.symmetric = g->symmetric == 1;
        in.V = V;
        in.E = g->E;
        in.nf = (double)nf;
        in.mf = (double)scout;
        in.unvisited_v = (double)V - (double)visited_cnt;
        in.unvisited_e = (double)std::max<int64_t>(edges_to_check, 0);
        in.max_deg = maxdeg;
        in.prev_nf = (double)prev_nf;
        return in;
    };

    bool cluster_passed = false;  // the cluster loop ran no level of this frontier
    while (nf > 0) {
        CGB_REQUIRE(iters < max_iters, CGB_ETIMEOUT, "BFS iteration budget exhausted");
        // ----- direction decision
        const bool heur = bottom_up ? (awake >= old_awake) || ((double)awake > (double)V / beta)
                                    : (double)scout > (double)edges_to_check / alpha;
        // small frontiers far from the switch point: run levels on the device;
        // a small graph's whole run, in the cluster
        const bool whole = g->E <= kClusterWholeEdges && g->max_degree <= kClusterList && !bottom_up;
        const bool far_off = !heur && (double)scout * alpha * 4.0 <= (double)edges_to_check;
        const uint64_t scout_exit = (uint64_t)std::max(0.0, (double)edges_to_check / alpha / 4.0);
        const uint32_t max_levels = (uint32_t)std::min<uint64_t>(max_iters - iters, 1u << 20);
        const bool use_cluster = cluster_ok && !cluster_passed &&
                                 nf <= std::min(g->tune.cluster_enter, g->tune.persist_enter) &&
                                 (whole || (far_off && scout <= kClusterEnterEdges));
        const bool use_grid = persist_ok && !use_cluster && far_off && nf <= g->tune.persist_enter &&
                              maxdeg < g->tune.persist_deg && scout > 0;
        if (use_cluster || use_grid) {
            if (timing) ktimer_begin(g, CGB_K_PUSH);
            const PersistResult r =
                use_cluster ? bfs_cluster(g, cur, (uint32_t)nf, level,
                                          whole ? 0xFFFFFFFFu
                                                : std::min(g->tune.persist_enter, 2 * g->tune.cluster_enter),
                                          whole ? 0xFFFFFFFFu
                                                : (uint32_t)std::min<uint64_t>(scout_exit, kClusterExitEdges),
                                          max_levels)
                            : bfs_persistent(g, cur, (uint32_t)nf, scout, maxdeg, level, g->tune.persist_enter,
                                             scout_exit, g->tune.persist_deg, max_levels);
            if (timing) ktimer_end(g);
            scout = r.scout;
            if (r.levels > 0) maxdeg = r.max_deg;
            else if (nf == 1) maxdeg = (uint32_t)scout;
            if (r.levels > 0) {
                visited_cnt += r.found;
                edges_to_check -= (int64_t)r.scouts;
                iters += r.levels;
                level += r.levels;
                g->stats.pushes_td += r.levels;
                prev_nf = nf;
                nf = r.nf;
                cur = r.cur;
                bottom_up = false;
                have_policy_out = false;
                continue;
            }
            if (use_cluster) {
                // the direction is decided again, now that the loop has counted
                // the frontier's out-edges (a root's were not known before)
                cluster_passed = true;
                continue;
            }
        }
        cluster_passed = false;
        const int out = cur ^ 1;
        // the heuristic's expansion of a push level: every list of 32 edges or
        // more chunked for small frontiers, else the degree-binned tiers
        const int heur_expand = nf <= kSmallFrontier ? kExpandChunked : kExpandBinned;
        bool go_pull;
        int expand = heur_expand;
        if (force_pull) go_pull = true;
        else if (!want_pull) go_pull = false;
        else if (collect) {
            // counterfactual: time the three level variants from the same state
            const size_t vbytes = (size_t)V * 4, wbytes = (size_t)words * 4;
            CGB_CUDA_TRY(cudaMemcpyAsync(collect->save_value, g->value, vbytes, cudaMemcpyDeviceToDevice, g->stream));
            CGB_CUDA_TRY(cudaMemcpyAsync(collect->save_bm0, g->visited, wbytes, cudaMemcpyDeviceToDevice, g->stream));
            float ms[kPolicyOutputs] = {};
            bool have[kPolicyOutputs] = {};
            const int outs[3] = {kOutPush, kOutPull, kOutPushChunked};
            // every trial starts right after a restore, the first one too: after
            // the snapshot copy alone the levels array is colder in L2, and the
            // first variant timed slower than it runs (a bias toward the others)
            CGB_CUDA_TRY(cudaMemcpyAsync(g->value, collect->save_value, vbytes, cudaMemcpyDeviceToDevice, g->stream));
            CGB_CUDA_TRY(cudaMemcpyAsync(g->visited, collect->save_bm0, wbytes, cudaMemcpyDeviceToDevice, g->stream));
            for (int d = 0; d < 3; d++) {
                CGB_CUDA_TRY(cudaEventRecord(g->ev_iter[0], g->stream));
                do_level(d == 1, out, d == 2 ? kExpandChunked : kExpandBinned);
                CGB_CUDA_TRY(cudaEventRecord(g->ev_iter[1], g->stream));
                sync_counters(g);
                CGB_CUDA_TRY(cudaEventElapsedTime(&ms[outs[d]], g->ev_iter[0], g->ev_iter[1]));
                have[outs[d]] = true;
                CGB_CUDA_TRY(cudaMemcpyAsync(g->value, collect->save_value, vbytes, cudaMemcpyDeviceToDevice,
                                             g->stream));
                CGB_CUDA_TRY(cudaMemcpyAsync(g->visited, collect->save_bm0, wbytes, cudaMemcpyDeviceToDevice,
                                             g->stream));
            }
            policy_log_sample(g, state_now(), ms, have);
            int best = 0;
            for (int d = 1; d < 3; d++)
                if (ms[outs[d]] < ms[outs[best]]) best = d;
            go_pull = best == 1;
            expand = best == 2 ? kExpandChunked : kExpandBinned;
        } else if (pol && have_policy_out) {
            const int hc = heur ? 1 : (heur_expand == kExpandChunked ? 2 : 0);
            const int choice = policy_pick_bfs_level(g->h_ctr->policy_out, hc);
            go_pull = choice < 0 ? heur : choice == 1;
            if (choice == 0) expand = kExpandBinned;
            if (choice == 2) expand = kExpandChunked;
        } else {
            go_pull = heur;
        }

        float it_ms = 0.f;
        if (tracing) CGB_CUDA_TRY(cudaEventRecord(g->ev_iter[0], g->stream));
        const FeatIn before = state_now();
        do_level(go_pull, out, expand);
        if (go_pull) {
            if (!bottom_up) {
                awake = nf;
                old_awake = 0;
            }
            std::swap(front, next);
            g->stats.pulls_bu++;
        } else {
            g->stats.pushes_td++;
        }
        if (tracing) CGB_CUDA_TRY(cudaEventRecord(g->ev_iter[1], g->stream));
        // inference for the next level, fused before the counter read-back;
        // skipped while both Beamer ratios are far (64x) from their
        // thresholds, where the choice is not in doubt
        const double r_alpha = (double)scout * alpha / (double)std::max<int64_t>(edges_to_check, 1);
        const double r_beta = (double)nf * beta / (double)V;
        const bool near_boundary = (r_alpha > 1.0 / 64 && r_alpha < 64.0) || (r_beta > 1.0 / 64 && r_beta < 64.0);
        const bool infer = kPolicyLevels && pol && near_boundary;
        if (infer) {
            FeatIn in = before;
            in.unvisited_e = (double)std::max<int64_t>(edges_to_check - (int64_t)scout, 0);
            policy_enqueue(pol, g, in, 1, go_pull, out);
        }
        sync_counters(g);
        have_policy_out = infer;
        if (tracing) {
            CGB_CUDA_TRY(cudaEventElapsedTime(&it_ms, g->ev_iter[0], g->ev_iter[1]));
            cgb_iter_trace t{};
            t.iteration = (uint32_t)iters;
            t.algorithm = CGB_BFS;
            t.frontier_vertices = nf;
            t.frontier_edges = scout;
            t.unvisited_vertices = (uint64_t)V - visited_cnt;
            t.unvisited_edges = (uint64_t)std::max<int64_t>(edges_to_check, 0);
            t.max_frontier_degree = maxdeg;
            t.variant = go_pull ? CGB_VAR_PULL : CGB_VAR_TWC;
            t.ms = it_ms;
            g->trace.push_back(t);
        }
        CGB_REQUIRE(!g->h_ctr->overflow, CGB_EOVERFLOW, "BFS frontier queue overflow");
        const uint64_t n_next = g->h_ctr->qlen[out];
        const uint64_t m_next = g->h_ctr->medges;
        if (go_pull) {
            old_awake = awake;
            awake = g->h_ctr->found;
            visited_cnt += g->h_ctr->found;
        } else {
            visited_cnt += n_next;  // upper bound when nz < V; only steers the schedule
        }
        bottom_up = go_pull;
        edges_to_check -= (int64_t)scout;
        scout = m_next;
        maxdeg = g->h_ctr->max_deg;
        prev_nf = nf;
        nf = n_next;
        cur = out;
        level++;
        iters++;
    }
    CGB_CUDA_TRY(cudaEventRecord(g->ev_stop, g->stream));
    g->stats.iterations = iters;
}

}  // namespace cgb
