// Multi-root BFS state and kernels shared by the batch path (msbfs.cu) and
// the request server (serve.cu).  See msbfs.cu for the algorithm.
#pragma once

#include "engine.cuh"
#include "push.cuh"

namespace cgb {

// Several arrays in one device allocation (a cudaMalloc each cost more than
// the first pass's kernels): sizes are added up by a first pass over the
// arrays, pointers set by a second one.
struct Carve {
    char* base = nullptr;
    size_t bytes = 0;
    template <class T>
    void take(T*& p, size_t n)
    {
        if (base) p = reinterpret_cast<T*>(base + bytes);
        bytes += ((n ? n : 1) * sizeof(T) + 255) / 256 * 256;
    }
};

struct MsBuffers {
    void* block = nullptr;                  // the allocation that holds the arrays
    unsigned long long* seen = nullptr;
    unsigned long long* front[2] = {nullptr, nullptr};
    unsigned long long* next = nullptr;     // top-down scratch; bottom-up partial masks; zero between levels
    uint32_t* heavy_w = nullptr;            // bottom-up: vertices finished by a warp (V)
    uint32_t* heavy_b = nullptr;            // ... in chunks (cap_b)
    uint2* hub_chunks = nullptr;            // their chunks: (vertex, chunk) (cap_c)
    uint32_t* heavy_len = nullptr;          // [3] lengths of the three lists
    uint32_t cap_b = 0, cap_c = 0;
};

MsBuffers* ms_buffers_alloc(uint32_t V, uint64_t E);
void ms_buffers_free(MsBuffers* b);

// One bottom-up level (four kernels, see msbfs.cu).
struct MsBuArgs {
    uint32_t V;
    const uint32_t* in_off;
    const uint32_t* in_src;
    const unsigned long long* front;  // current frontier masks
    unsigned long long* seen;
    unsigned long long* fnext;        // next frontier masks (zero on entry)
    unsigned long long* acc;          // partial masks (zero on entry and exit)
    unsigned long long full;          // roots that still have a frontier
    uint32_t* level_out;
    uint32_t lvl;
    uint32_t nz;
    uint32_t* qact;                   // next queue
    uint32_t* qact_len;
    uint32_t cap;
    DevCounters* ctr;
    const uint32_t* start;            // per-root start level (server) or NULL
    unsigned long long* alive;        // roots given new frontier vertices, or NULL
    uint32_t* heavy_w;
    uint32_t* heavy_b;
    uint32_t* heavy_len;
    uint32_t cap_b;
    uint2* hub_chunks;
    uint32_t cap_c;
};
void ms_bottom_up(const MsBuArgs& a, cudaStream_t st, uint64_t* launches);

struct MsTdOp {
    const uint32_t* __restrict__ off;
    const uint32_t* __restrict__ dst;
    const unsigned long long* __restrict__ front;
    const unsigned long long* seen;
    unsigned long long* next;
    uint32_t* qout;
    uint32_t* qlen;
    uint32_t cap;
    DevCounters* ctr;

    static constexpr bool kStaged = true;
    static constexpr int kBatch = 4;  // edge slots per lane visited together (push.cuh)

    __device__ __forceinline__ bool load(uint32_t v, uint32_t& s, uint32_t& d, uint32_t& m) const
    {
        s = off[v];
        d = off[v + 1] - s;
        m = v;
        return true;
    }
    template <int N>
    __device__ __forceinline__ void edges(const bool (&valid)[N], const uint32_t (&e)[N], const uint32_t (&v)[N]) const
    {
        uint32_t u[N];
        unsigned long long add[N], have[N];
        bool first[N];
#pragma unroll
        for (int i = 0; i < N; i++) u[i] = valid[i] ? __ldcs(dst + e[i]) : 0u;
#pragma unroll
        for (int i = 0; i < N; i++) add[i] = valid[i] ? front[v[i]] & ~seen[u[i]] : 0ull;
#pragma unroll
        for (int i = 0; i < N; i++) have[i] = add[i] ? next[u[i]] : 0ull;
#pragma unroll
        for (int i = 0; i < N; i++) first[i] = (add[i] & ~have[i]) && atomicOr(next + u[i], add[i]) == 0ull;
        stage_append_n<N>(first, u, qout, qlen, cap, &ctr->overflow);
    }
    __device__ __forceinline__ void edge(bool valid, uint32_t e, uint32_t v) const
    {
        const bool va[1] = {valid};
        const uint32_t ea[1] = {e}, ma[1] = {v};
        edges<1>(va, ea, ma);
    }
    __device__ __forceinline__ void block_begin() const { stage_begin(); }
    __device__ __forceinline__ void block_end() const { stage_end(qout, qlen, cap, &ctr->overflow); }
};

// n_ptr (optional) replaces n by a device-resident count; off (optional):
// the next frontier's out-edges are added to ctr->medges.
__global__ void k_ms_finalize(const uint32_t* __restrict__ q, uint32_t n, const uint32_t* n_ptr,
                              unsigned long long* seen,
                              unsigned long long* next, unsigned long long* fnext, uint32_t* level_out, uint32_t V,
                              uint32_t lvl, uint32_t nz, uint32_t* qact, uint32_t* qact_len, uint32_t cap,
                              DevCounters* ctr, const uint32_t* start, unsigned long long* alive,
                              const uint32_t* __restrict__ off);
__global__ void k_ms_clear(const uint32_t* __restrict__ q, uint32_t n, unsigned long long* f);
__global__ void k_ms_fill(uint64_t n, uint32_t* a, uint32_t value);
__global__ void k_ms_degree_sum(const uint32_t* __restrict__ q, uint32_t n, const uint32_t* n_ptr,
                                const uint32_t* __restrict__ off, DevCounters* ctr);

}  // namespace cgb
