// Multi-root BFS with bit-packed per-root masks (up to 64 roots per pass).
//
// Every vertex carries three 64-bit masks: seen (roots that reached it),
// frontier (roots for which it is on the current level) and next (roots that
// reach it on the next level).  One traversal of an edge serves every root
// whose bit rides on it (the multi-source BFS of Then et al., VLDB 2014),
// so a batch of 64 roots costs a small multiple of one BFS instead of 64.
//   top-down  -- for each vertex of the active queue and each out-edge (v,u):
//                next[u] |= frontier[v] & ~seen[u] (atomicOr; the first
//                setter queues u), then a finalise pass moves next into
//                seen/frontier and writes the level of every new (root, u);
//   bottom-up -- every vertex not seen by all roots ORs the frontier masks of
//                its in-neighbours restricted to its missing roots, stopping
//                as soon as none is missing; one thread owns the vertex, so
//                its masks are written without atomics.
// Levels go to out[k * V + u] (root-major, 999999999 = unreachable), the
// layout of cgb_run_batch; they equal k separate cgb_run(CGB_BFS) results.
#include "msbfs.cuh"
#include "push.cuh"

namespace cgb {

__global__ void k_ms_init(uint32_t V, unsigned long long* seen, unsigned long long* f0, unsigned long long* next)
{
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        seen[v] = 0;
        f0[v] = 0;
        next[v] = 0;
    }
}

__global__ void k_ms_fill(uint64_t n, uint32_t* a, uint32_t value)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        a[i] = value;
}

// Roots: seen/frontier bits, level 0, and the first active queue (a root
// listed twice still gets one queue entry); one thread per root.
__global__ void k_ms_roots(const uint32_t* roots, uint32_t n, uint32_t V, unsigned long long* seen,
                           unsigned long long* f0, uint32_t* level_out, uint32_t* q, uint32_t* qlen, uint32_t nz,
                           unsigned long long* alive)
{
    const uint32_t k = threadIdx.x;
    if (k >= n) return;
    const uint32_t r = roots[k];
    const unsigned long long bit = 1ull << k;
    if (atomicOr(seen + r, bit) == 0ull && r < nz) q[atomicAdd(qlen, 1u)] = r;
    if (r < nz) {  // only vertices with out-edges are ever read as frontier
        atomicOr(f0 + r, bit);
        atomicOr(alive, bit);
    }
    level_out[(size_t)k * V + r] = 0;
}

// Moves next into seen / the new frontier for the queued vertices, writes
// their levels, and keeps those with new roots (and out-edges) active.
__global__ void __launch_bounds__(kBlock) k_ms_finalize(const uint32_t* __restrict__ q, uint32_t n,
                                                        const uint32_t* n_ptr, unsigned long long* seen, unsigned long long* next,
                                                        unsigned long long* fnext, uint32_t* level_out, uint32_t V,
                                                        uint32_t lvl, uint32_t nz, uint32_t* qact, uint32_t* qact_len,
                                                        uint32_t cap, DevCounters* ctr, const uint32_t* start,
                                                        unsigned long long* alive, const uint32_t* __restrict__ off)
{
    if (n_ptr) n = *n_ptr;
    const uint32_t n_round = (n + 31u) & ~31u;
    unsigned long long live = 0, edges = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_round; i += gridDim.x * blockDim.x) {
        bool act = false;
        uint32_t u = 0;
        if (i < n) {
            u = q[i];
            const unsigned long long x = next[u] & ~seen[u];
            next[u] = 0;
            if (x) {
                seen[u] |= x;
                for (unsigned long long m = x; m; m &= m - 1) {
                    const uint32_t k = __ffsll(m) - 1;
                    level_out[(size_t)k * V + u] = start ? lvl - start[k] : lvl;
                }
                act = u < nz;
                if (act) {
                    fnext[u] = x;
                    live |= x;
                    if (off) edges += off[u + 1] - off[u];
                }
            }
        }
        warp_append(act, u, qact, qact_len, cap, &ctr->overflow);
    }
    if (off) cta_add(edges, &ctr->medges);
    if (alive) {
        live = warp_or(live);
        if (lane_id() == 0 && (live & ~*(volatile unsigned long long*)alive)) atomicOr(alive, live);
    }
}

// The counters of the next level: one launch, not a memset each.
__global__ void k_ms_level_reset(DevCounters* ctr, int nxt)
{
    ctr->qlen[nxt] = 0;
    ctr->alive = 0;
    ctr->found = 0;
    ctr->chunk_len = 0;
    ctr->medges = 0;
}

// Clears the frontier masks of the vertices of a queue.
__global__ void k_ms_clear(const uint32_t* __restrict__ q, uint32_t n, unsigned long long* f)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) f[q[i]] = 0;
}

// Bottom-up levels, binned by in-degree.  A vertex is done when every root
// it still misses (among the roots with a frontier, `full`) has been found
// in its in-neighbours' frontier masks -- rare while the roots sit at
// different depths, so lists are often walked to the end.  Walking a hub's
// list on one thread would make the hub the whole kernel's time, so:
//   k_ms_bu_light  -- the first kMsLight in-edges of every vertex, packed
//                     edge-parallel per warp;
//                     vertices left unfinished go to a warp list (or, with
//                     at least kMsBlockDeg edges left, a hub list, with a
//                     descriptor for each kMsHubChunk edges) with the
//                     roots found so far parked in `acc` (the top-down
//                     scratch mask, zero between levels);
//   k_ms_bu_warp   -- a warp per listed vertex, lanes striding the list;
//   k_ms_bu_chunks -- a warp per hub chunk, merged into acc by atomicOr;
//                     k_ms_bu_settle then finishes the hubs.
// Each vertex has one owner at a time, so its masks and levels are written
// without atomics; new vertices with out-edges join the next queue.
// RMAT-22, 64 roots, the level after the roots' (31 k vertices, 22.8 M
// out-edges; most vertices find few of their roots and walk whole lists):
// walking the hub list in every CTA took 1.27 ms, descriptors take 0.05 ms;
// in the next level (levels written one root's run at a time) the light
// kernel went from 1.09 to 0.51 ms.
constexpr uint32_t kMsLight = 32;
constexpr uint32_t kMsBlockDeg = 4096;
constexpr uint32_t kMsHubChunk = 512;

__device__ __forceinline__ unsigned long long warp_or64(unsigned long long v)
{
    const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)v);
    const uint32_t hi = __reduce_or_sync(0xffffffffu, (uint32_t)(v >> 32));
    return ((unsigned long long)hi << 32) | lo;
}

// Levels of the roots `got` newly found for vertex u, the warp's lanes
// holding consecutive vertices: one root at a time, so that a warp's stores
// are one run of the root's row (a lane writing its own roots one after the
// other touches a sector per root and vertex).
__device__ __forceinline__ void ms_write_levels(uint32_t u, unsigned long long got, uint32_t* level_out, uint32_t V,
                                                uint32_t lvl, const uint32_t* start)
{
    for (unsigned long long m = warp_or64(got); m; m &= m - 1) {
        const uint32_t k = __ffsll(m) - 1;
        if ((got >> k) & 1ull) level_out[(size_t)k * V + u] = start ? lvl - start[k] : lvl;
    }
}

__global__ void __launch_bounds__(kBlock) k_ms_bu_light(MsBuArgs a)
{
    // A warp takes 32 consecutive vertices; a warp scan packs the first
    // kMsLight in-edges of each, kN edges per lane at a time (sources, then
    // masks, in flight together), and the finds are ORed into the owner's
    // shared mask.  Warps share nothing between steps.
    constexpr int kN = 4;
    __shared__ uint32_t s_acc[kBlock / 32][2][32];
    const uint32_t V = a.V, lane = lane_id(), warp = threadIdx.x >> 5;
    unsigned long long live = 0;
    const uint32_t warps = gridDim.x * (kBlock / 32);
    stage_begin();
    __syncthreads();
    for (uint32_t base = (blockIdx.x * (kBlock / 32) + warp) * 32; base < V; base += warps * 32) {
        const uint32_t u = base + lane;
        unsigned long long s = 0, pending = 0;
        uint32_t e0 = 0, deg = 0, cnt = 0;
        if (u < V) {
            s = a.seen[u];
            pending = a.full & ~s;
            if (pending) {
                e0 = a.in_off[u];
                deg = a.in_off[u + 1] - e0;
                cnt = min(deg, kMsLight);
            }
        }
        const uint32_t incl = warp_incl_scan(cnt), total = __shfl_sync(0xffffffffu, incl, 31);
        if (total == 0) continue;
        const uint32_t excl = incl - cnt;
        s_acc[warp][0][lane] = s_acc[warp][1][lane] = 0;
        __syncwarp();
        for (uint32_t b = 0; b < total; b += 32 * kN) {
            uint32_t o[kN], src[kN];
            unsigned long long x[kN];
#pragma unroll
            for (int i = 0; i < kN; i++) {
                const uint32_t p = b + 32 * i + lane;
                o[i] = 0;
#pragma unroll
                for (uint32_t step = 16; step >= 1; step >>= 1) {
                    const uint32_t ex = __shfl_sync(0xffffffffu, excl, o[i] + step);
                    if (ex <= p) o[i] += step;
                }
                const uint32_t e = __shfl_sync(0xffffffffu, e0, o[i]) + p - __shfl_sync(0xffffffffu, excl, o[i]);
                src[i] = p < total ? a.in_src[e] : 0xFFFFFFFFu;
            }
#pragma unroll
            for (int i = 0; i < kN; i++) x[i] = src[i] != 0xFFFFFFFFu ? a.front[src[i]] : 0ull;
#pragma unroll
            for (int i = 0; i < kN; i++) {
                const uint32_t lo = (uint32_t)x[i], hi = (uint32_t)(x[i] >> 32);
                if (lo) atomicOr(&s_acc[warp][0][o[i]], lo);
                if (hi) atomicOr(&s_acc[warp][1][o[i]], hi);
            }
        }
        __syncwarp();
        unsigned long long got =
            pending & (((unsigned long long)s_acc[warp][1][lane] << 32) | s_acc[warp][0][lane]);
        __syncwarp();
        bool act[1] = {false}, to_warp = false, to_hub = false;
        if (got != pending && deg > kMsLight) {
            a.acc[u] = got;  // finish on a warp or in hub chunks
            got = 0;
            to_hub = deg - kMsLight >= kMsBlockDeg;
            to_warp = !to_hub;
        }
        ms_write_levels(u, got, a.level_out, V, a.lvl, a.start);
        if (got) {
            a.seen[u] = s | got;
            if (u < a.nz) {
                a.fnext[u] = got;
                live |= got;
                act[0] = true;
            }
        }
        const uint32_t ua[1] = {u};
        stage_append_n<1>(act, ua, a.qact, a.qact_len, a.cap, &a.ctr->overflow);
        warp_append(to_warp, u, a.heavy_w, a.heavy_len, a.cap, &a.ctr->overflow);
        warp_append(to_hub, u, a.heavy_b, a.heavy_len + 1, a.cap_b, &a.ctr->overflow);
        warp_append_chunks(u, to_hub ? (deg - kMsLight + kMsHubChunk - 1) / kMsHubChunk : 0, a.hub_chunks,
                           a.heavy_len + 2, a.cap_c, &a.ctr->overflow);
    }
    __syncthreads();
    stage_end(a.qact, a.qact_len, a.cap, &a.ctr->overflow);
    if (a.alive) {
        live = warp_or(live);
        if (lane_id() == 0 && (live & ~*(volatile unsigned long long*)a.alive)) atomicOr(a.alive, live);
    }
}

__global__ void __launch_bounds__(kBlock) k_ms_bu_warp(MsBuArgs a)
{
    const uint32_t n = min(a.heavy_len[0], a.cap);
    const uint32_t lane = lane_id();
    unsigned long long live = 0;
    for (uint32_t i = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); i < n; i += gridDim.x * (kBlock / 32)) {
        const uint32_t u = a.heavy_w[i];
        const unsigned long long s = a.seen[u];
        const unsigned long long pending = a.full & ~s;
        unsigned long long got = a.acc[u];
        const uint32_t e1 = a.in_off[u + 1];
        for (uint32_t e = a.in_off[u] + kMsLight; e < e1 && got != pending; e += 128) {
            uint32_t src[4];
#pragma unroll
            for (int j = 0; j < 4; j++) src[j] = e + 32 * j + lane < e1 ? a.in_src[e + 32 * j + lane] : 0xFFFFFFFFu;
            unsigned long long x = 0;
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (src[j] != 0xFFFFFFFFu) x |= a.front[src[j]];
            got |= warp_or64(x & pending);
        }
        bool act = false;
        if (got) {
            // the new roots' levels: lane l writes roots l and l + 32
#pragma unroll
            for (uint32_t k = lane; k < 64; k += 32)
                if ((got >> k) & 1ull) a.level_out[(size_t)k * a.V + u] = a.start ? a.lvl - a.start[k] : a.lvl;
        }
        if (lane == 0) {
            a.acc[u] = 0;
            if (got) {
                a.seen[u] = s | got;
                act = u < a.nz;
                if (act) {
                    a.fnext[u] = got;
                    live |= got;
                }
            }
        }
        warp_append(act, u, a.qact, a.qact_len, a.cap, &a.ctr->overflow);
    }
    if (a.alive) {
        live = warp_or(live);
        if (lane == 0 && (live & ~*(volatile unsigned long long*)a.alive)) atomicOr(a.alive, live);
    }
}

// Hub chunks, one warp each: the chunk's finds are ORed into acc[u]; chunks
// of vertices already complete are skipped.
__global__ void __launch_bounds__(kBlock) k_ms_bu_chunks(MsBuArgs a)
{
    constexpr int kN = 8;
    const uint32_t n = min(a.heavy_len[2], a.cap_c), lane = lane_id();
    const uint32_t warps = gridDim.x * (kBlock / 32);
    for (uint32_t c = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; c < n; c += warps) {
        const uint2 d = a.hub_chunks[c];
        const unsigned long long pending = a.full & ~a.seen[d.x];
        // one read for the warp: other warps are ORing into it
        const unsigned long long have =
            __shfl_sync(0xffffffffu, *(volatile unsigned long long*)(a.acc + d.x), 0);
        if (have == pending) continue;
        const uint32_t b0 = a.in_off[d.x] + kMsLight + d.y * kMsHubChunk;
        const uint32_t e1 = min(a.in_off[d.x + 1], b0 + kMsHubChunk);
        unsigned long long got = 0;
        for (uint32_t e = b0 + lane; e < e1; e += 32 * kN) {
            uint32_t src[kN];
#pragma unroll
            for (int j = 0; j < kN; j++) src[j] = e + 32 * j < e1 ? a.in_src[e + 32 * j] : 0xFFFFFFFFu;
#pragma unroll
            for (int j = 0; j < kN; j++)
                if (src[j] != 0xFFFFFFFFu) got |= a.front[src[j]];
        }
        got = warp_or64(got) & pending;
        if (lane == 0 && (got & ~have)) atomicOr(a.acc + d.x, got);
    }
}

// Records the roots `got` newly found for vertex u (its owner only).
__device__ __forceinline__ bool ms_bu_settle(uint32_t u, unsigned long long s, unsigned long long got,
                                             unsigned long long* seen, unsigned long long* fnext,
                                             uint32_t* level_out, uint32_t V, uint32_t lvl, uint32_t nz,
                                             const uint32_t* start)
{
    seen[u] = s | got;
    for (unsigned long long m = got; m; m &= m - 1) {
        const uint32_t k = __ffsll(m) - 1;
        level_out[(size_t)k * V + u] = start ? lvl - start[k] : lvl;
    }
    if (u < nz) fnext[u] = got;
    return u < nz;
}

// Settles the listed hub vertices from their merged masks.
__global__ void __launch_bounds__(kBlock) k_ms_bu_settle(MsBuArgs a)
{
    const uint32_t n = min(a.heavy_len[1], a.cap_b);
    const uint32_t n_round = (n + 31u) & ~31u;
    unsigned long long live = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_round; i += gridDim.x * blockDim.x) {
        bool act = false;
        uint32_t u = 0;
        if (i < n) {
            u = a.heavy_b[i];
            const unsigned long long s = a.seen[u];
            const unsigned long long got = a.acc[u] & (a.full & ~s);
            a.acc[u] = 0;
            if (got) {
                act = ms_bu_settle(u, s, got, a.seen, a.fnext, a.level_out, a.V, a.lvl, a.nz, a.start);
                if (act) live |= got;
            }
        }
        warp_append(act, u, a.qact, a.qact_len, a.cap, &a.ctr->overflow);
    }
    if (a.alive) {
        live = warp_or(live);
        if (lane_id() == 0 && (live & ~*(volatile unsigned long long*)a.alive)) atomicOr(a.alive, live);
    }
}

void ms_bottom_up(const MsBuArgs& a, cudaStream_t st, uint64_t* launches)
{
    CGB_CUDA_TRY(cudaMemsetAsync(a.heavy_len, 0, 12, st));
    k_ms_bu_light<<<grid_for(a.V, kBlock, num_sms() * 8), kBlock, stage_bytes(kBlock), st>>>(a);
    k_ms_bu_warp<<<num_sms() * 8, kBlock, 0, st>>>(a);
    k_ms_bu_chunks<<<num_sms() * 8, kBlock, 0, st>>>(a);
    k_ms_bu_settle<<<num_sms() * 4, kBlock, 0, st>>>(a);
    if (launches) *launches += 4;
}

__global__ void k_ms_degree_sum(const uint32_t* __restrict__ q, uint32_t n, const uint32_t* n_ptr,
                                const uint32_t* __restrict__ off, DevCounters* ctr)
{
    if (n_ptr) n = *n_ptr;
    unsigned long long s = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t v = q[i];
        s += off[v + 1] - off[v];
    }
    cta_add(s, &ctr->medges);
}

// Out-edges of the reached (root, vertex) pairs, from the seen masks.
__global__ void k_ms_reached(uint32_t V, const unsigned long long* __restrict__ seen, const uint32_t* __restrict__ off,
                             DevCounters* ctr)
{
    unsigned long long edges = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
        edges += (unsigned long long)__popcll(seen[v]) * (off[v + 1] - off[v]);
    cta_add(edges, &ctr->reached_edges);
}

void count_reached_ms(cgb_graph* g)
{
    CGB_CUDA_TRY(cudaMemsetAsync(&g->ctr->reached_edges, 0, 8, g->stream));
    k_ms_reached<<<grid_for(g->V, kBlock, num_sms() * 8), kBlock, 0, g->stream>>>(g->V, g->ms->seen, g->off, g->ctr);
    sync_counters(g);
    g->stats.traversed_edges = g->h_ctr->reached_edges;
}

// Runs one pass of up to 64 roots; level_out (device) receives n * V levels.
void run_msbfs(cgb_graph* g, const uint32_t* d_roots, uint32_t n, uint32_t* level_out, double alpha)
{
    CGB_REQUIRE(n >= 1 && n <= 64, CGB_EINVAL, "multi-root BFS takes 1..64 roots per pass");
    ensure_frontier(g);
    ensure_csc(g);
    const uint32_t V = g->V;
    if (!g->ms) g->ms = ms_buffers_alloc(V, g->E);
    MsBuffers& b = *g->ms;
    // Invariant at the start of a level: front[cur] is non-zero only at the
    // vertices of the active queue q[cur]; front[cur ^ 1] and next are zero.
    const unsigned long long full = n == 64 ? ~0ull : ((1ull << n) - 1);
    const uint32_t gridV = grid_for(V, kBlock, num_sms() * 8);
    ++g->stats.launches;
    k_ms_init<<<gridV, kBlock, 0, g->stream>>>(V, b.seen, b.front[0], b.next);
    CGB_CUDA_TRY(cudaMemsetAsync(b.front[1], 0, (size_t)V * 8, g->stream));
    ++g->stats.launches;
    k_ms_fill<<<num_sms() * 8, kBlock, 0, g->stream>>>((uint64_t)n * V, level_out, kValueMax);
    CGB_CUDA_TRY(cudaMemsetAsync(g->ctr, 0, sizeof(DevCounters), g->stream));
    ++g->stats.launches;
    k_ms_roots<<<1, 64, 0, g->stream>>>(d_roots, n, V, b.seen, b.front[0], level_out, g->q[0], &g->ctr->qlen[0], g->nz,
                                       &g->ctr->alive);
    // Each level is queued whole -- its kernels read the counts of the ones
    // before them on the device, and the next frontier's out-edges (the next
    // direction choice) are counted on the way -- and ends with one read-back.
    k_ms_degree_sum<<<1, kBlock, 0, g->stream>>>(g->q[0], 0, &g->ctr->qlen[0], g->off, g->ctr);
    ++g->stats.launches;
    sync_counters(g);
    uint64_t nact = g->h_ctr->qlen[0];
    // Roots with vertices in the current frontier.  Bottom-up looks only
    // for these: a root whose traversal has ended (a small component) would
    // otherwise keep every vertex scanning its whole in-list.
    unsigned long long live = g->h_ctr->alive & full;
    uint64_t level_edges = g->h_ctr->medges;
    int cur = 0;
    uint32_t lvl = 0;
    while (nact > 0) {
        CGB_REQUIRE(lvl <= V, CGB_ETIMEOUT, "multi-root BFS level bound exceeded");
        // direction: out-edges of the active vertices against the graph's edges
        const bool pull = (double)level_edges * alpha > (double)g->E;
        const bool tracing = (g->flags & CGB_FLAG_TRACE) != 0;
        if (tracing) CGB_CUDA_TRY(cudaEventRecord(g->ev_iter[0], g->stream));
        const int nxt = cur ^ 1;
        unsigned long long* fcur = b.front[cur];
        unsigned long long* fnxt = b.front[nxt];
        ++g->stats.launches;
        k_ms_level_reset<<<1, 1, 0, g->stream>>>(g->ctr, nxt);
        if (pull) {
            MsBuArgs ba{V, g->in_off, g->in_src, fcur, b.seen, fnxt, b.next, live, level_out, lvl + 1, g->nz,
                        g->q[nxt], &g->ctr->qlen[nxt], V, g->ctr, nullptr, &g->ctr->alive, b.heavy_w, b.heavy_b,
                        b.heavy_len, b.cap_b, b.hub_chunks, b.cap_c};
            ms_bottom_up(ba, g->stream, &g->stats.launches);
            ++g->stats.launches;
            k_ms_degree_sum<<<gridV, kBlock, 0, g->stream>>>(g->q[nxt], 0, &g->ctr->qlen[nxt], g->off, g->ctr);
            g->stats.pulls_bu++;
        } else {
            // expansion into next[]: touched vertices are queued once in stamp[]
            MsTdOp op{g->off, g->dst, fcur, b.seen, b.next, g->stamp, &g->ctr->found, V, g->ctr};
            launch_push(g, g->q[cur], (uint32_t)nact, op, false);
            ++g->stats.launches;
            // at most one touched vertex per out-edge
            k_ms_finalize<<<grid_for(std::min<uint64_t>(V, level_edges), kBlock, num_sms() * 8), kBlock, 0,
                            g->stream>>>(g->stamp, 0, &g->ctr->found, b.seen, b.next, fnxt, level_out, V, lvl + 1,
                                         g->nz, g->q[nxt], &g->ctr->qlen[nxt], V, g->ctr, nullptr, &g->ctr->alive,
                                         g->off);
            g->stats.pushes_td++;
        }
        ++g->stats.launches;
        k_ms_clear<<<grid_for(nact, kBlock, num_sms() * 8), kBlock, 0, g->stream>>>(g->q[cur], (uint32_t)nact, fcur);
        sync_counters(g);
        CGB_REQUIRE(!g->h_ctr->overflow, CGB_EOVERFLOW, "multi-root BFS queue overflow");
        if (tracing) {
            CGB_CUDA_TRY(cudaEventRecord(g->ev_iter[1], g->stream));
            CGB_CUDA_TRY(cudaEventSynchronize(g->ev_iter[1]));
            cgb_iter_trace t{};
            t.iteration = lvl;
            t.algorithm = CGB_BFS;
            t.frontier_vertices = nact;
            t.frontier_edges = level_edges;
            t.variant = pull ? CGB_VAR_PULL : CGB_VAR_TWC;
            CGB_CUDA_TRY(cudaEventElapsedTime(&t.ms, g->ev_iter[0], g->ev_iter[1]));
            g->trace.push_back(t);
        }
        nact = g->h_ctr->qlen[nxt];
        live = g->h_ctr->alive;
        level_edges = g->h_ctr->medges;
        cur = nxt;
        lvl++;
    }
    g->stats.iterations = lvl;
}

MsBuffers* ms_buffers_alloc(uint32_t V, uint64_t E)
{
    auto* b = new MsBuffers();
    try {
        b->cap_b = (uint32_t)std::min<uint64_t>(E / kMsBlockDeg + 2, V);
        // every hub's list past kMsLight in chunks: sum of ceil(deg / kMsHubChunk) <= E / kMsHubChunk + hubs
        b->cap_c = (uint32_t)(E / kMsHubChunk + b->cap_b + 1);
        auto arrays = [&](Carve& c) {
            c.take(b->seen, V);
            c.take(b->front[0], V);
            c.take(b->front[1], V);
            c.take(b->next, V);
            c.take(b->heavy_w, V);
            c.take(b->heavy_b, b->cap_b);
            c.take(b->hub_chunks, b->cap_c);
            c.take(b->heavy_len, 3);
        };
        Carve size, place;
        arrays(size);
        CGB_CUDA_TRY(cudaMalloc(&b->block, size.bytes));
        place.base = static_cast<char*>(b->block);
        arrays(place);
        CGB_CUDA_TRY(cudaMemset(b->next, 0, (size_t)V * 8));  // zero between levels (bottom-up parks masks here)
    } catch (...) {
        ms_buffers_free(b);
        throw;
    }
    return b;
}

void ms_buffers_free(MsBuffers* b)
{
    if (!b) return;
    cudaFree(b->block);
    delete b;
}

void free_msbfs(cgb_graph* g)
{
    ms_buffers_free(g->ms);
    g->ms = nullptr;
}

}  // namespace cgb
