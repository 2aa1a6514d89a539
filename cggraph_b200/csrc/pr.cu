// Pull-based FP64 PageRank.
//
// The reference's formula (my_project/CGgraph/GraphNuma.cuh:233-244,545-554,
// device_algorithm.cuh:538-545): pr0 = 1/N and per iteration
//     pr'[v] = 0.15/N + 0.85 * sum_{u -> v} pr[u] / outdeg[u],
// with no redistribution of dangling mass.  The reference evaluates it by
// pushing in uint32 (so every value truncates to 0) into the wrong slot; this
// engine evaluates the formula in FP64 by pulling over the in-edge CSC, which
// needs no atomics and gives the same result on every run.
//
// Layout (built once per graph, graph.cu ensure_pr): vertices are relabelled
// by a stable sort on (out-degree bucket floor(log2 outdeg), largest first
// and zero out-degree last; then in-degree, largest first).  Every
// contribution that is ever gathered (the n_src vertices with out-edges) then
// lies in one dense prefix of contrib[] (RMAT-24: 7.4 M of 16.8 M vertices,
// 59 MB, L2-resident), the most gathered ones first, and consecutive rows
// have nearly equal in-degrees.  One last pass maps the result back to the
// caller's vertex ids.
//
// Each iteration reads contrib[u] = pr[u]/outdeg[u] of the previous one and
// writes contrib' (the division is fused into the epilogue); the last
// iteration writes pr instead.  Only the last iteration computes the rows
// without out-edges: nothing reads their contribution.  The edges are stored
// as a sliced ELL, 32 rows per slice (edge j of lane l at slice base + 32j +
// l, padded to the slice's longest row), one warp per slice, one row per
// lane.  Its rows are
//   - the relabelled vertices in order, except the long rows;
//   - the long rows (pr_long_row in-edges or more) cut into segments of
//     nearly equal length, at most pr_seg edges, sorted by their first
//     source.  k_pr_combine adds a row's segments, in an order of their own.
// So no warp holds a long chain of gathers, and since a row lists its
// sources in ascending order (hottest first), the segments running at one
// time gather from one moving range of contributions.  20 iterations, before
// (rows of up to 4095 in-edges on one lane, hub rows in chunks on a second
// stream) and now, on one B200: RMAT-16 2.4 -> 0.23 ms, RMAT-24 16.4 -> 13.6
// ms, Chung-Lu (126 M edges) 13.0 -> 6.3 ms.
// Every summation order is fixed by the graph alone, so results are
// bit-reproducible.
#include "engine.cuh"

namespace cgb {

__global__ void k_pr_init(uint32_t V, uint32_t n_src, const uint32_t* __restrict__ outdeg, double* contrib)
{
    const double p0 = 1.0 / (double)V;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n_src; v += gridDim.x * blockDim.x)
        contrib[v] = p0 / (double)outdeg[v];
}

// What bounds an iteration is the gathers of contrib[]: 8 bytes each, one
// 32-byte sector through the L2-to-SM path, which delivers one sector per
// clock and SM (290 G gathers/s from an L2-resident array, measured with a
// plain gather loop; hits in L1 run at 840 G/s).  A window of the hottest
// contributions in shared memory (16 K doubles) was no faster than leaving
// the space to L1, and a larger one left too few L1 lines for the misses in
// flight.
//
// On skewed graphs (kHint) the gathers of the hottest contributions carry an
// L2 evict-last policy and the rest evict-first, so that 6.5 M doubles (52
// MB, the front of the layout) stay in L2 beside the streamed column indices
// while the long tail passes through.  Graphs without hubs (meshes) keep
// plain loads: their contributions are reused by nearby rows, which
// evict-first cut short (the 4800 x 5000 grid: 6.5 -> 7.5 ms per run with
// the hints).
constexpr uint32_t kPrHot = 6500000;
constexpr uint32_t kPrHintMinDeg = 64;  // largest out-degree from which a graph counts as skewed

__device__ __forceinline__ double ld_f64_l2hint(const double* p, uint64_t policy)
{
    double v;
    asm volatile("ld.global.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(policy));
    return v;
}

struct PrIter {
    uint32_t V;             // padding target: contrib[V] is 0
    uint32_t n_rows;        // rows of this iteration
    uint32_t n_seg;         // segments of long rows
    uint32_t n_seg_slices;  // slices of segments; the slices of rows follow
    const uint64_t* __restrict__ slice_ptr;
    const uint32_t* __restrict__ slice_len;
    const uint32_t* __restrict__ col;
    const uint32_t* __restrict__ seg_id;   // segment of each lane of the segment slices
    const uint32_t* __restrict__ long_bm;  // rows cut into segments
    const uint32_t* __restrict__ outdeg;
    const double* __restrict__ contrib;
    double* part;         // per segment
    double* contrib_out;  // n_rows next contributions, or
    double* pr_out;       // (last iteration) n_rows results
    double base, damp;
};

__device__ __forceinline__ void pr_row_out(const PrIter& a, uint32_t r, double sum)
{
    const double p = a.base + a.damp * sum;
    // not read again this iteration: keep L2 for the gathers
    if (a.pr_out) __stcs(a.pr_out + r, p);
    else __stcs(a.contrib_out + r, p / (double)__ldcs(a.outdeg + r));
}

// One warp per slice: in step j every lane loads its row's j-th source (one
// coalesced 128-byte load per warp) and gathers that contribution; the steps
// go in batches of kU (cgb_tuning.pr_unroll), whose gathers are issued before
// they are summed, in j order, as far as the registers reach: 32 (40 with
// hints) do not hold 16 pending doubles, so at kU = 16 the compiler splits
// the batch, and the three unrolls of a variant differ less than their names.
// Padding slots and the masked steps of the last batch name vertex V, whose
// contribution is 0.
// (The plain kernel is held to 32 registers, 8 CTAs an SM: at 34 registers, 6
// CTAs, the 4800 x 5000 grid took 6.77 instead of 6.34 ms.  The hinted one
// spills there: it has 6.)
template <int kU, bool kHint>
__global__ void __launch_bounds__(kBlock, kHint ? 6 : 8) k_pr_pull(PrIter a)
{
    const uint32_t lane = lane_id();
    const uint32_t nslices = a.n_seg_slices + (a.n_rows + 31) / 32;
    const uint32_t nwarps = gridDim.x * (kBlock / 32);
    uint64_t pol_hot, pol_cold;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol_hot));
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol_cold));
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (uint32_t s = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); s < nslices; s += nwarps) {
        const uint32_t len = a.slice_len[s];
        const uint32_t* c = a.col + a.slice_ptr[s] + lane;
        double acc = 0.0;
        for (uint32_t j = 0; j < len; j += kU) {
            uint32_t u[kU];
#pragma unroll
            for (int t = 0; t < kU; t++) u[t] = j + t < len ? __ldcs(c + 32u * (j + t)) : a.V;  // read once
            double x[kU];
#pragma unroll
            for (int t = 0; t < kU; t++)
                x[t] = kHint ? ld_f64_l2hint(a.contrib + u[t], u[t] < kPrHot ? pol_hot : pol_cold) : a.contrib[u[t]];
#pragma unroll
            for (int t = 0; t < kU; t++) acc += x[t];
        }
        if (s < a.n_seg_slices) {
            const uint32_t i = s * 32 + lane;
            if (i < a.n_seg) a.part[a.seg_id[i]] = acc;
        } else {
            const uint32_t rs = s - a.n_seg_slices, r = rs * 32 + lane;
            if (r < a.n_rows && !((a.long_bm[rs] >> lane) & 1u)) pr_row_out(a, r, acc);
        }
    }
    asm volatile("griddepcontrol.launch_dependents;");
}

// Adds the segments of the long rows: one CTA per hub row (more than
// kPrHubSegs segments, the first n_hubs CTAs), else 8 lanes per row.  (With
// a row per lane, or a warp walking 32 rows one by one, the chains of loads
// took 76 us at RMAT-24 and 33 us at RMAT-16.)
__global__ void __launch_bounds__(kBlock) k_pr_combine(PrIter a, const uint32_t* __restrict__ rows,
                                                       const uint32_t* __restrict__ seg_base, uint32_t n,
                                                       const uint32_t* __restrict__ hubs, uint32_t n_hubs)
{
    const uint32_t lane = lane_id();
    if (blockIdx.x < n_hubs) {
        __shared__ double s_part[kBlock / 32];
        const uint32_t i = hubs[blockIdx.x];
        const uint32_t b = seg_base[i], e = seg_base[i + 1];
        asm volatile("griddepcontrol.wait;" ::: "memory");
        double t = 0.0;
#pragma unroll 4
        for (uint32_t k = b + threadIdx.x; k < e; k += kBlock) t += __ldcg(a.part + k);
        t = warp_sum(t);
        if (lane == 0) s_part[threadIdx.x >> 5] = t;
        __syncthreads();
        if (threadIdx.x < 32) {
            t = warp_sum(lane < kBlock / 32 ? s_part[lane] : 0.0);
            if (lane == 0 && rows[i] < a.n_rows) pr_row_out(a, rows[i], t);
        }
    asm volatile("griddepcontrol.launch_dependents;");
        return;
    }
    const uint32_t i = ((blockIdx.x - n_hubs) * kBlock + threadIdx.x) / 8;
    const uint32_t b = i < n ? seg_base[i] : 0, e = i < n ? seg_base[i + 1] : 0;
    const uint32_t row = i < n ? rows[i] : 0xFFFFFFFFu;
    const bool mine = e - b <= kPrHubSegs;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    double t = 0.0;
    if (mine) {
#pragma unroll 4
        for (uint32_t k = b + (lane & 7u); k < e; k += 8) t += __ldcg(a.part + k);
    }
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    t += __shfl_xor_sync(0xffffffffu, t, 4);
    if (mine && (lane & 7u) == 0 && row < a.n_rows) pr_row_out(a, row, t);
    asm volatile("griddepcontrol.launch_dependents;");
}

// Back to the caller's vertex ids: out[v] = pr[rank[v]].
__global__ void k_pr_unpermute(uint32_t V, const uint32_t* __restrict__ rank, const double* __restrict__ pr,
                               double* out)
{
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) out[v] = pr[rank[v]];
}

void run_pr(cgb_graph* g, uint32_t iters, const cgb_options& o)
{
    (void)o;
    ensure_pr(g);
    ensure_max_degree(g);
    const bool timing = g->flags & CGB_FLAG_KERNEL_TIMING;
    const uint32_t V = g->V;
    const double base = 0.15 / (double)V;
    const double damp = 0.85;
    if (iters == 0) iters = 1;  // graphProcess_device runs at least one iteration
    CGB_CUDA_TRY(cudaEventRecord(g->ev_start, g->stream));
    if (timing) ktimer_begin(g, CGB_K_INIT);
    ++g->stats.launches;
    k_pr_init<<<grid_for(g->n_src, kBlock, num_sms() * 8), kBlock, 0, g->stream>>>(V, g->n_src, g->pr_outdeg,
                                                                                g->contrib[0]);
    if (timing) ktimer_end(g);
    const uint32_t unroll = g->tune.pr_unroll;
    const bool hint = g->max_degree >= kPrHintMinDeg;
    auto pull = unroll == 4 ? (hint ? k_pr_pull<4, true> : k_pr_pull<4, false>)
                : unroll == 16 ? (hint ? k_pr_pull<16, true> : k_pr_pull<16, false>)
                               : (hint ? k_pr_pull<8, true> : k_pr_pull<8, false>);
    PrIter a{};
    a.V = V;
    a.n_seg = g->n_pr_seg;
    a.n_seg_slices = div_up(g->n_pr_seg, 32);
    a.slice_ptr = g->pr_slice_ptr;
    a.slice_len = g->pr_slice_len;
    a.col = g->pr_col;
    a.seg_id = g->pr_seg_id;
    a.long_bm = g->pr_long_bm;
    a.outdeg = g->pr_outdeg;
    a.part = g->pr_part;
    a.base = base;
    a.damp = damp;
    for (uint32_t it = 0; it < iters; it++) {
        const bool last = it + 1 == iters;
        a.n_rows = last ? V : g->n_src;
        a.contrib = g->contrib[it & 1];
        a.contrib_out = last ? nullptr : g->contrib[(it & 1) ^ 1];
        a.pr_out = last ? g->pr[0] : nullptr;
        if (timing) ktimer_begin(g, CGB_K_PR);
        ++g->stats.launches;
        // programmatic dependent launches: a kernel's CTAs are placed while the last
        // ones of the kernel before it run, and wait for its results there.  They
        // may be placed only once a CTA's own work is done: placed earlier, the
        // waiting CTAs of a grid that fits the machine at once crowd where there is
        // room, and the next iteration runs with some SMs full and others idle
        // (random graph, 2^17 vertices of 30 edges, 20 iterations: 0.60 ms placed
        // at the start of a kernel, 0.36 at its end, 0.41 without such launches;
        // RMAT-16 0.225, 0.194, 0.297; RMAT-24 13.64, 13.62; 4900^2 grid 6.5 each).
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.blockDim = dim3(kBlock);
        cfg.stream = g->stream;
        cfg.attrs = attr;
        cfg.numAttrs = timing ? 0 : 1;
        cfg.gridDim = dim3(grid_for((uint64_t)a.n_seg_slices + div_up(a.n_rows, 32), kBlock / 32,
                                    num_sms() * g->tune.pr_ctas_per_sm));
        CGB_CUDA_TRY(cudaLaunchKernelEx(&cfg, pull, a));
        if (g->n_pr_long) {
            ++g->stats.launches;
            cfg.gridDim = dim3(g->n_pr_hubs + div_up((uint64_t)g->n_pr_long * 8, kBlock));
            CGB_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_pr_combine, a, (const uint32_t*)g->pr_long_rows,
                                            (const uint32_t*)g->pr_seg_base, g->n_pr_long,
                                            (const uint32_t*)g->pr_hubs, g->n_pr_hubs));
        }
        if (timing) ktimer_end(g);
    }
    // the other pr buffer receives the result in the caller's ids
    ++g->stats.launches;
    k_pr_unpermute<<<grid_for(V, kBlock, num_sms() * 8), kBlock, 0, g->stream>>>(V, g->pr_rank, g->pr[0], g->pr[1]);
    CGB_CUDA_TRY(cudaEventRecord(g->ev_stop, g->stream));
    g->result = g->pr[1];
    g->stats.iterations = iters;
}

}  // namespace cgb
