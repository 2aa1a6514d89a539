// Degree-binned push expansion over a vertex frontier.
//
// Replaces the reference's per-thread load balancers WarpDonate::schedule
// (my_project/CGgraph/device_warpDonate.cuh:42-388) and CTA::schedule
// (my_project/CGgraph/device_CTA.cuh:28-112), which run one frontier vertex
// per thread and hand large lists to the warp or CTA with __syncthreads
// loops, serialising a hub's whole list on one CTA.  Here each frontier
// vertex is binned by out-degree:
//   deg >= kHugeDeg          deferred to k_push_huge, which splits the list
//                            into kHugeChunk-edge chunks across every CTA;
//   kCtaDeg <= deg < kHuge   the whole CTA walks the list (owner election);
//   32 <= deg < kCtaDeg      one warp walks the list (ballot election);
//   deg < 32                 fine-grained gather: a CTA-wide exclusive scan of
//                            the remaining degrees packs the small lists
//                            into shared memory, one edge per thread.
// Every edge visit is warp-collective (Op::edge is called by all 32 lanes,
// with `valid` false on idle lanes) so that the ops can aggregate their
// queue appends with one ballot and one atomic per warp.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "engine.cuh"

namespace cgb {

// Batched edge visits.  An op that declares `static constexpr int kBatch = N`
// also provides
//   template <int M> __device__ void edges(const bool (&valid)[M],
//                                          const uint32_t (&e)[M],
//                                          const uint32_t (&msg)[M]);
// (warp-collective, like edge; it may keep counts in the op, which is the
// thread's own) which visits M edge slots per lane at once:
// every load of the M slots is issued before any of them is used, so a lane
// keeps M gathers in flight instead of one dependent chain per edge.  The
// expansion loops below hand such ops N slots per lane (32 * N edges per
// warp step); other ops are called edge by edge.
template <class T, class = void>
struct op_batch {
    static constexpr int value = 1;
};
template <class T>
struct op_batch<T, std::void_t<decltype(T::kBatch)>> {
    static constexpr int value = T::kBatch;
};

template <class Op, int N>
__device__ __forceinline__ void visit_n(Op& op, const bool (&valid)[N], const uint32_t (&e)[N],
                                        const uint32_t (&m)[N])
{
    if constexpr (op_batch<Op>::value == 1) {
#pragma unroll
        for (int i = 0; i < N; i++) op.edge(valid[i], e[i], m[i]);
    } else {
        op.template edges<N>(valid, e, m);
    }
}

// Edges [first, end) of one list walked by the calling warp (all lanes call
// it with the same arguments), op_batch<Op> slots per lane at a time.
template <class Op>
__device__ __forceinline__ void warp_range(Op& op, uint32_t first, uint32_t end, uint32_t m)
{
    constexpr int N = op_batch<Op>::value;
    const uint32_t lane = lane_id();
    for (uint32_t k = first; k < end; k += 32 * N) {
        bool valid[N];
        uint32_t e[N], mm[N];
#pragma unroll
        for (int i = 0; i < N; i++) {
            const uint32_t idx = k + 32 * i + lane;
            valid[i] = idx < end;
            e[i] = valid[i] ? idx : 0u;
            mm[i] = m;
        }
        visit_n<Op, N>(op, valid, e, mm);
    }
}

// Warp-aggregated append of up to N items per lane (pred[i] selects item
// i): one atomic per warp.  Every lane of the warp must call it.  Items past
// `cap` are not written and raise *overflow.
template <int N>
__device__ __forceinline__ void warp_append_n(const bool (&pred)[N], const uint32_t (&item)[N], uint32_t* q,
                                              uint32_t* ctr, uint32_t cap, uint32_t* overflow)
{
    uint32_t cnt = 0;
#pragma unroll
    for (int i = 0; i < N; i++) cnt += pred[i] ? 1u : 0u;
    const uint32_t incl = warp_incl_scan(cnt);
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    if (total == 0) return;
    uint32_t base = 0;
    if (lane_id() == 0) base = atomicAdd(ctr, total);
    uint32_t idx = __shfl_sync(0xffffffffu, base, 0) + incl - cnt;
#pragma unroll
    for (int i = 0; i < N; i++) {
        if (pred[i]) {
            if (idx < cap) q[idx] = item[i];
            else atomicOr(overflow, 1u);
            idx++;
        }
    }
}

// Staged append: each warp collects its items in shared memory and writes
// kStage of them at a time with one atomic; what is left at the end goes out
// with one atomic per CTA.  One atomic per warp step on the queue's counter
// queued at its L2 slice (1.5 G same-address atomics a second on a B200): a
// BFS level of 4.3 M edges with 1.4 M finds spent most of its 0.24 ms there.
// stage_begin comes before a CTA barrier, stage_end after one, both called by
// every thread; stage_append_n is warp-collective.  The items are in dynamic
// shared memory, stage_bytes(threads, kItems) of it, kItems per warp.
constexpr uint32_t kStage = 128;
constexpr uint32_t kStageWarps = 512 / 32;  // largest CTA of the push kernels

extern __shared__ uint32_t s_stage[];
__shared__ uint32_t s_staged[kStageWarps];

constexpr uint32_t stage_bytes(uint32_t threads, uint32_t items = kStage) { return threads / 32 * items * 4; }

// An op that stages its finds declares `static constexpr bool kStaged = true`.
template <class T, class = void>
struct op_staged {
    static constexpr bool value = false;
};
template <class T>
struct op_staged<T, std::void_t<decltype(T::kStaged)>> {
    static constexpr bool value = T::kStaged;
};

__device__ __forceinline__ void stage_begin()
{
    if (threadIdx.x < kStageWarps) s_staged[threadIdx.x] = 0;
}

template <uint32_t kItems>
__device__ __forceinline__ void stage_write(uint32_t warp, uint32_t n, uint32_t base, uint32_t* q, uint32_t cap,
                                            uint32_t* overflow)
{
    for (uint32_t i = lane_id(); i < n; i += 32) {
        if (base + i < cap) q[base + i] = s_stage[warp * kItems + i];
        else atomicOr(overflow, 1u);
    }
}

template <int N, uint32_t kItems = kStage>
__device__ __forceinline__ void stage_append_n(const bool (&pred)[N], const uint32_t (&item)[N], uint32_t* q,
                                               uint32_t* ctr, uint32_t cap, uint32_t* overflow)
{
    static_assert(32 * N <= kItems, "one step must fit");
    const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
    uint32_t m[N], total = 0;
#pragma unroll
    for (int i = 0; i < N; i++) {
        m[i] = __ballot_sync(0xffffffffu, pred[i]);
        total += __popc(m[i]);
    }
    if (total == 0) return;
    uint32_t have = s_staged[warp];
    __syncwarp();
    if (have + total > kItems) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(ctr, have);
        stage_write<kItems>(warp, have, __shfl_sync(0xffffffffu, base, 0), q, cap, overflow);
        have = 0;
        __syncwarp();
    }
    if (lane == 0) s_staged[warp] = have + total;
#pragma unroll
    for (int i = 0; i < N; i++) {
        if (pred[i]) s_stage[warp * kItems + have + __popc(m[i] & lanemask_lt())] = item[i];
        have += __popc(m[i]);
    }
    __syncwarp();
}

template <uint32_t kItems = kStage>
__device__ __forceinline__ void stage_end(uint32_t* q, uint32_t* ctr, uint32_t cap, uint32_t* overflow)
{
    __shared__ uint32_t s_base[kStageWarps];
    const uint32_t warp = threadIdx.x >> 5, lane = lane_id(), warps = blockDim.x / 32;
    if (warp == 0) {
        const uint32_t n = lane < warps ? s_staged[lane] : 0;
        const uint32_t incl = warp_incl_scan(n), total = __shfl_sync(0xffffffffu, incl, 31);
        uint32_t base = 0;
        if (lane == 0 && total) base = atomicAdd(ctr, total);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (lane < warps) s_base[lane] = base + incl - n;
    }
    __syncthreads();
    stage_write<kItems>(warp, s_staged[warp], s_base[warp], q, cap, overflow);
}

// Chunk descriptors (v, 0 .. nch - 1) of every lane's vertex, written by the
// warp together with one atomic for all of them; position p belongs to the
// last lane whose first position is <= p (a 5-step shuffle search).
__device__ __forceinline__ void warp_append_chunks(uint32_t v, uint32_t nch, uint2* q, uint32_t* len, uint32_t cap,
                                                   uint32_t* overflow)
{
    if (!__any_sync(0xffffffffu, nch != 0)) return;
    const uint32_t incl = warp_incl_scan(nch), total = __shfl_sync(0xffffffffu, incl, 31);
    const uint32_t excl = incl - nch;
    uint32_t slot = 0;
    if (lane_id() == 0) slot = atomicAdd(len, total);
    slot = __shfl_sync(0xffffffffu, slot, 0);
    for (uint32_t p0 = 0; p0 < total; p0 += 32) {
        const uint32_t p = p0 + lane_id();
        uint32_t o = 0;
#pragma unroll
        for (uint32_t step = 16; step >= 1; step >>= 1) {
            const uint32_t ex = __shfl_sync(0xffffffffu, excl, o + step);
            if (ex <= p) o += step;
        }
        const uint32_t bv = __shfl_sync(0xffffffffu, v, o), ex = __shfl_sync(0xffffffffu, excl, o);
        if (p < total) {
            if (slot + p < cap) q[slot + p] = make_uint2(bv, p - ex);
            else atomicOr(overflow, 1u);
        }
    }
}

// Fine-grained tier: a CTA-wide exclusive scan of the (small) remaining
// degrees packs the lists into shared memory, one edge per thread per round.
// Every thread of the CTA must call it.
template <class Op>
__device__ __forceinline__ void fine_tier(const Op& op, uint32_t start, uint32_t deg, uint32_t msg, uint32_t* s_scan,
                                          uint32_t* s_edge, uint32_t* s_emsg)
{
    const uint32_t tid = threadIdx.x;
    uint32_t total;
    const uint32_t rank = block_excl_scan(deg, total, s_scan);
    uint32_t consumed = 0;
    for (uint32_t done = 0; done < total; done += kBlock) {
        while (consumed < deg && rank + consumed < done + kBlock) {
            s_edge[rank + consumed - done] = start + consumed;
            s_emsg[rank + consumed - done] = msg;
            consumed++;
        }
        __syncthreads();
        const uint32_t n = min((uint32_t)kBlock, total - done);
        const bool valid = tid < n;
        op.edge(valid, valid ? s_edge[tid] : 0u, valid ? s_emsg[tid] : 0u);
        __syncthreads();
    }
}

// Fine-grained tier of one warp (no CTA barriers): a warp-inclusive scan of
// the lanes' remaining degrees (each below 32) packs their lists into rounds
// of 32 edges; in each round every lane takes one edge and finds the lane
// that owns it -- the last lane whose exclusive prefix is <= the edge's
// position -- by a 5-step shuffle search.  Batched ops take op_batch<Op>
// rounds at once.  Called by all 32 lanes.
template <class Op>
__device__ __forceinline__ void fine_tier_warp(Op& op, uint32_t start, uint32_t deg, uint32_t msg)
{
    constexpr int N = op_batch<Op>::value;
    const uint32_t lane = lane_id();
    uint32_t incl = deg;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    const uint32_t excl = incl - deg;
    for (uint32_t base = 0; base < total; base += 32 * N) {
        bool valid[N];
        uint32_t e[N], mm[N];
#pragma unroll
        for (int i = 0; i < N; i++) {
            const uint32_t idx = base + 32 * i + lane;
            uint32_t o = 0;
#pragma unroll
            for (uint32_t step = 16; step >= 1; step >>= 1) {
                const uint32_t ex = __shfl_sync(0xffffffffu, excl, o + step);
                if (ex <= idx) o += step;
            }
            const uint32_t st = __shfl_sync(0xffffffffu, start, o);
            const uint32_t ex = __shfl_sync(0xffffffffu, excl, o);
            mm[i] = __shfl_sync(0xffffffffu, msg, o);
            valid[i] = idx < total;
            e[i] = valid[i] ? st + (idx - ex) : 0u;
        }
        visit_n<Op, N>(op, valid, e, mm);
    }
}

// Op interface:
//   __device__ bool load(uint32_t v, uint32_t& start, uint32_t& deg, uint32_t& msg) const;
//   __device__ void edge(bool valid, uint32_t e, uint32_t msg) const;   // warp-collective
// and, for the engine's kernels (k_push_binned, k_push_chunks), per-CTA hooks
// around all of a CTA's work, each followed / preceded by a CTA barrier:
//   __device__ void block_begin() const;   // e.g. zero shared accumulators
//   __device__ void block_end() const;     // e.g. flush them with one atomic
template <class Op, bool kIdentity>
__global__ void __launch_bounds__(kBlock) k_push_twc(const uint32_t* __restrict__ qin, uint32_t nin, Op op,
                                                     uint32_t* __restrict__ huge_q, uint32_t* huge_len,
                                                     uint32_t huge_cap)
{
    __shared__ uint32_t s_scan[kBlock / 32 + 1];
    __shared__ uint32_t s_owner, s_start, s_deg, s_msg;
    __shared__ uint32_t s_edge[kBlock];
    __shared__ uint32_t s_emsg[kBlock];
    const uint32_t tid = threadIdx.x;

    for (uint32_t base = blockIdx.x * kBlock; base < nin; base += gridDim.x * kBlock) {
        uint32_t i = base + tid;
        uint32_t start = 0, deg = 0, msg = 0;
        if (i < nin) {
            uint32_t v = kIdentity ? i : qin[i];
            if (!op.load(v, start, deg, msg)) deg = 0;
            if (deg >= kHugeDeg) {
                // capacity V: each vertex appears at most once per frontier
                const uint32_t slot = atomicAdd(huge_len, 1u);
                if (slot < huge_cap) huge_q[slot] = v;
                deg = 0;
            }
        }
        // CTA tier
        while (__syncthreads_or(deg >= kCtaDeg)) {
            if (deg >= kCtaDeg) s_owner = tid;
            __syncthreads();
            if (s_owner == tid) {
                s_start = start;
                s_deg = deg;
                s_msg = msg;
                deg = 0;
            }
            __syncthreads();
            const uint32_t st = s_start, dg = s_deg, m = s_msg;
            for (uint32_t k = 0; k < dg; k += kBlock) op.edge(k + tid < dg, st + k + tid, m);
            __syncthreads();
        }
        // warp tier
        uint32_t wmask;
        while ((wmask = __ballot_sync(0xffffffffu, deg >= 32)) != 0) {
            const uint32_t leader = __ffs(wmask) - 1;
            const uint32_t st = __shfl_sync(0xffffffffu, start, leader);
            const uint32_t dg = __shfl_sync(0xffffffffu, deg, leader);
            const uint32_t m = __shfl_sync(0xffffffffu, msg, leader);
            if (lane_id() == leader) deg = 0;
            for (uint32_t k = 0; k < dg; k += 32) op.edge(k + lane_id() < dg, st + k + lane_id(), m);
        }
        fine_tier(op, start, deg, msg, s_scan, s_edge, s_emsg);
    }
}

// Hubs deferred by k_push_twc: the concatenated chunk list of all deferred
// vertices is dealt round-robin to the CTAs of the grid.
template <class Op>
__global__ void __launch_bounds__(kBlock) k_push_huge(const uint32_t* __restrict__ huge_q, const uint32_t* huge_len,
                                                      uint32_t huge_cap, Op op)
{
    const uint32_t n = min(*huge_len, huge_cap);
    uint64_t chunk_base = 0;
    for (uint32_t h = 0; h < n; h++) {
        const uint32_t v = huge_q[h];
        uint32_t start, deg, msg;
        if (!op.load(v, start, deg, msg)) continue;
        const uint32_t nch = (deg + kHugeChunk - 1) / kHugeChunk;
        const uint32_t first = (uint32_t)((blockIdx.x + gridDim.x - (chunk_base % gridDim.x)) % gridDim.x);
        for (uint32_t c = first; c < nch; c += gridDim.x) {
            const uint32_t cs = c * kHugeChunk;
            const uint32_t ce = min(deg, cs + kHugeChunk);
            for (uint32_t k = cs; k < ce; k += kBlock) op.edge(k + threadIdx.x < ce, start + k + threadIdx.x, msg);
        }
        chunk_base += nch;
    }
}

// Binned expansion used by the engine.  Lists of at least big_deg edges are
// cut into chunk-edge pieces whose descriptors (vertex, chunk index) go to a
// chunk queue; k_push_chunks then deals the chunks across the whole grid, so
// a frontier of a few hubs keeps every SM busy however few vertices it has.
// Lists of 32..big_deg-1 edges are walked by one warp, shorter ones by the
// warp's fine-grained tier (fine_tier_warp).  Chunk-queue capacity
// E/chunk + E/big_deg + 64 bounds any frontier in which each vertex appears
// once; the queue is sized for the smallest chunk and big_deg launch_push
// uses (kMinChunk and 32).
template <class Op, bool kIdentity, int kBlk>
__global__ void __launch_bounds__(kBlk) k_push_binned(const uint32_t* __restrict__ qin, uint32_t nin, Op op,
                                                        uint2* __restrict__ chunk_q, uint32_t* chunk_len,
                                                        uint32_t chunk_cap, uint32_t* overflow, uint32_t big_deg,
                                                        uint32_t chunk)
{
    op.block_begin();
    __syncthreads();
    for (uint32_t base = blockIdx.x * kBlk; base < nin; base += gridDim.x * kBlk) {
        const uint32_t i = base + threadIdx.x;
        uint32_t v = 0, start = 0, deg = 0, msg = 0;
        if (i < nin) {
            v = kIdentity ? i : qin[i];
            if (!op.load(v, start, deg, msg)) deg = 0;
        }
        // big lists go to the chunk queue
        const bool is_big = deg >= big_deg;
        warp_append_chunks(v, is_big ? (deg + chunk - 1) / chunk : 0, chunk_q, chunk_len, chunk_cap, overflow);
        if (is_big) deg = 0;
        // warp tier
        uint32_t wmask;
        while ((wmask = __ballot_sync(0xffffffffu, deg >= 32)) != 0) {
            const uint32_t leader = __ffs(wmask) - 1;
            const uint32_t st = __shfl_sync(0xffffffffu, start, leader);
            const uint32_t dg = __shfl_sync(0xffffffffu, deg, leader);
            const uint32_t m = __shfl_sync(0xffffffffu, msg, leader);
            if (lane_id() == leader) deg = 0;
            warp_range(op, st, st + dg, m);
        }
        fine_tier_warp(op, start, deg, msg);
    }
    __syncthreads();
    op.block_end();
}

// One warp per chunk descriptor, grid-stride over the chunk queue: warps
// run ahead of one another, so that a few hundred edges per chunk keep many
// chains of loads in flight.  With no more chunks than CTAs a chunk is cut once
// more, over as many warps as a CTA has (10 levels of a 14 k-vertex Chung-Lu
// graph: 10 us a launch otherwise, 6 cut).  Ops without batched visits take a chunk with the
// whole CTA: one edge per lane at a time, a warp's chunk of 1024 edges is 32
// chains of dependent loads one after the other.  Label propagation, a chunk
// by a warp / by a CTA: RMAT-20 1.37 / 0.97 ms (and 6 rounds instead of 5: the
// long lists' labels arrive late), RMAT-16 0.28 / 0.18.
template <class Op, int kBlk>
__global__ void __launch_bounds__(kBlk) k_push_chunks(const uint2* __restrict__ chunk_q, const uint32_t* chunk_len,
                                                        uint32_t chunk_cap, Op op, uint32_t chunk)
{
    const uint32_t n = min(*chunk_len, chunk_cap);
    constexpr bool kByCta = op_batch<Op>::value == 1;
    const uint32_t parts = kByCta || n > gridDim.x ? 1 : min((uint32_t)kBlk / 32, chunk / 32);
    if (blockIdx.x >= n * parts) return;
    op.block_begin();
    __syncthreads();
    // (warps: CTAs take the first pieces one warp each before any takes a second)
    const uint32_t p0 = kByCta ? blockIdx.x : (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const uint32_t step = kByCta ? gridDim.x : gridDim.x * (kBlk / 32);
    for (uint32_t p = p0; p < n * parts; p += step) {
        const uint2 d = chunk_q[p % n];
        uint32_t start, deg, msg;
        if (!op.load(d.x, start, deg, msg)) continue;
        const uint32_t len = chunk / parts, cs = d.y * chunk + p / n * len, ce = min(deg, cs + len);
        if constexpr (kByCta) {
            for (uint32_t k = cs; k < ce; k += kBlk) {
                const uint32_t i = k + threadIdx.x;
                op.edge(i < ce, i < ce ? start + i : 0u, msg);
            }
        } else if (cs < ce) {
            warp_range(op, start + cs, start + ce, msg);
        }
    }
    __syncthreads();
    op.block_end();
}

// Frontiers of at most this many vertices cut every list of 32 edges or
// more into kMinChunk-edge chunks: with few vertices per warp slot of the
// machine (148 SMs x 64 warps x 32 lanes = 303 k), a warp walking its 32
// vertices' lists one after the other leaves the grid waiting for it.  Bounds
// of 32 k / 131 k / 400 k / 1 M: SSSP RMAT-18 0.49 / 0.47 / 0.43 / 0.43 ms,
// RMAT-20 0.66 / 0.63 / 0.60 / 0.60, Chung-Lu 57 M edges 2.4 / 2.3 / 2.15 /
// 2.2; BFS within 3 %.
constexpr uint32_t kSmallFrontier = 1u << 19;

template <class Op, int kBlk>
inline void launch_push_blk(cgb_graph* g, const uint32_t* qin, uint32_t nin, const Op& op, bool identity,
                            uint32_t ctas, uint32_t big_deg, uint32_t chunk)
{
    const uint32_t grid = grid_for(nin, kBlk, ctas);
    constexpr uint32_t smem = op_staged<Op>::value ? stage_bytes(kBlk) : 0;
    if (identity)
        k_push_binned<Op, true, kBlk><<<grid, kBlk, smem, g->stream>>>(
            qin, nin, op, g->chunk_q, &g->ctr->chunk_len, g->chunk_cap, &g->ctr->overflow, big_deg, chunk);
    else
        k_push_binned<Op, false, kBlk><<<grid, kBlk, smem, g->stream>>>(
            qin, nin, op, g->chunk_q, &g->ctr->chunk_len, g->chunk_cap, &g->ctr->overflow, big_deg, chunk);
    k_push_chunks<Op, kBlk><<<ctas, kBlk, smem, g->stream>>>(g->chunk_q, &g->ctr->chunk_len, g->chunk_cap, op, chunk);
}

// Expansion variants of launch_push: the size rule (chunk every list of 32
// edges or more for frontiers of at most kSmallFrontier vertices, else only
// lists of push_big_deg edges or more), or either tier forced.
enum PushExpand { kExpandAuto = 0, kExpandBinned = 1, kExpandChunked = 2 };

// Launches the binned expansion (plus the chunk kernel) of a queue whose
// length the host knows, with the graph's tuned CTA size (push_block) and
// grid.  The chunk-queue length must be zero beforehand.
template <class Op>
inline void launch_push(cgb_graph* g, const uint32_t* qin, uint32_t nin, const Op& op, bool identity,
                        int expand = kExpandAuto)
{
    if (nin == 0) return;
    const cgb_tuning& t = g->tune;
    const uint32_t ctas = num_sms() * t.push_ctas_per_sm;
    const bool small = expand == kExpandAuto ? nin <= kSmallFrontier : expand == kExpandChunked;
    const uint32_t big_deg = small ? 32u : t.push_big_deg;
    const uint32_t chunk = small ? kMinChunk : t.push_chunk;
    g->stats.launches += 2;
    if (t.push_block == 128) launch_push_blk<Op, 128>(g, qin, nin, op, identity, ctas, big_deg, chunk);
    else if (t.push_block == 512) launch_push_blk<Op, 512>(g, qin, nin, op, identity, ctas, big_deg, chunk);
    else launch_push_blk<Op, 256>(g, qin, nin, op, identity, ctas, big_deg, chunk);
}

}  // namespace cgb
