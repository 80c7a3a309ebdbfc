// Kruskal stress-1 against hop distance, and the multi-source BFS it needs.
//
// Reference: crates/graph-cli/src/bench.rs:255-295 (`stress`): BFS from every
// max(n / SOURCES, 1)-th node, then over every reachable (source, target) pair
// with d = hops and e = |p_target - p_source| (the f32 difference per axis,
// widened to f64, then hypot): DE = sum d e, EE = sum e^2, DD = sum d^2 in FP64,
// stress = sqrt(max((DD - DE / EE * DE) / DD, 0)), or 1 when EE or DD is 0.
//
// The BFS runs 64 sources at a time as one level-synchronous pull: node v's
// 64-bit frontier word at level L is the OR of its neighbours' words at L - 1,
// minus the sources that reached v already; each new bit writes v's hop count
// for that source. Hop counts are integers, so the result is the reference's
// exactly. The sums are per-thread sequential over a fixed grid-stride, then
// block sums and one fold of the block partials in block order: the same value
// every run (the reference's own order differs, so they agree to FP64 rounding).
#pragma once

#include "common.cuh"

namespace gr {

constexpr int BFS_T = 256;
constexpr int STRESS_T = 256;
constexpr uint32_t HOP_NONE = 0xffffffffu;

// ---- the adjacency of the raw edges, both directions, self-loops dropped: rows
// counted, scanned (Scanner) and filled. A row's entries land in any order; a
// level ORs their words, so the hops do not depend on it. An endpoint out of range
// leaves the first such edge in *bad and is not counted.
__global__ void __launch_bounds__(BFS_T)
k_adj_count(uint32_t n, uint32_t m, const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst,
            uint32_t *__restrict__ deg, uint32_t *bad) {
    const uint32_t e = blockIdx.x * BFS_T + threadIdx.x;
    if (e >= m) return;
    const uint32_t a = src[e], b = dst[e];
    if (a >= n || b >= n) {
        atomicMin(bad, e);
    } else if (a != b) {
        atomicAdd(&deg[a], 1u);
        atomicAdd(&deg[b], 1u);
    }
}

// fill: each row's next free entry, its first one before this kernel.
__global__ void __launch_bounds__(BFS_T)
k_adj_fill(uint32_t n, uint32_t m, const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst,
           uint32_t *__restrict__ fill, uint32_t *__restrict__ col) {
    const uint32_t e = blockIdx.x * BFS_T + threadIdx.x;
    if (e >= m) return;
    const uint32_t a = src[e], b = dst[e];
    if (a >= n || b >= n || a == b) return;
    col[atomicAdd(&fill[a], 1u)] = b;
    col[atomicAdd(&fill[b], 1u)] = a;
}

// The batch's sources: bit b of node sources[k0 + b] in visited and frontier,
// hop 0 at that node.
__global__ void k_msbfs_seed(uint32_t n, uint32_t k0, uint32_t kb, const uint32_t *__restrict__ sources,
                             unsigned long long *visited, unsigned long long *frontier, uint32_t *__restrict__ hops) {
    const uint32_t b = threadIdx.x;
    if (b >= kb) return;
    const uint32_t v = sources[k0 + b];
    atomicOr(&visited[v], 1ull << b);
    atomicOr(&frontier[v], 1ull << b);
    hops[(size_t)(k0 + b) * n + v] = 0u;
}

// Rows of more entries are pulled by the warp, BFS_ROW_AHEAD entries a lane at a
// time: a hub of 10,000 neighbours in one lane's loop took 750 us a level.
constexpr uint32_t BFS_ROW = 64;
constexpr int BFS_ROW_AHEAD = 16;

// One level: node v takes the batch's sources that reached any neighbour at the
// previous level and not v yet. Reads frontier, writes next (ping-pong).
// changed[level] is set when any node took one; nothing is left to do once the
// level before changed nothing, so several levels may be launched at a time.
template <typename Offset>
__global__ void __launch_bounds__(BFS_T)
k_msbfs_level(uint32_t n, const Offset *__restrict__ rp, const uint32_t *__restrict__ col, unsigned long long all,
              const unsigned long long *__restrict__ frontier, unsigned long long *__restrict__ visited,
              unsigned long long *__restrict__ next, uint32_t *__restrict__ hops, uint32_t k0, uint32_t level,
              const uint32_t *before, uint32_t *changed) {
    if (*before == 0u) return;
    const uint32_t v = blockIdx.x * BFS_T + threadIdx.x, lane = threadIdx.x % GR_WARP;
    if ((v & ~(GR_WARP - 1u)) >= n) return;  // whole warps only
    const bool valid = v < n;
    const unsigned long long vis = valid ? visited[v] : all;
    unsigned long long acc = 0ull;
    Offset e0 = 0, e1 = 0;
    if ((vis & all) != all) {
        e0 = rp[v];
        e1 = rp[v + 1];
    }
    const bool longrow = e1 - e0 > BFS_ROW;
    if (!longrow)
        for (Offset e = e0; e < e1; e++) {
            acc |= frontier[col[e]];
            if (((acc | vis) & all) == all) break;  // nothing left to reach v
        }
    for (uint32_t rows = __ballot_sync(GR_FULL, longrow); rows; rows &= rows - 1) {
        const int src = __ffs(rows) - 1;
        const Offset r0 = __shfl_sync(GR_FULL, e0, src), r1 = __shfl_sync(GR_FULL, e1, src);
        const unsigned long long rv = __shfl_sync(GR_FULL, vis, src);
        unsigned long long got = 0ull;
        for (Offset e = r0; e < r1; e += GR_WARP * BFS_ROW_AHEAD) {
            unsigned long long f[BFS_ROW_AHEAD];
#pragma unroll
            for (int u = 0; u < BFS_ROW_AHEAD; u++) {
                const Offset q = e + u * GR_WARP + lane;
                f[u] = q < r1 ? frontier[col[q]] : 0ull;
            }
#pragma unroll
            for (int u = 0; u < BFS_ROW_AHEAD; u++) got |= f[u];
            const unsigned long long lo = __reduce_or_sync(GR_FULL, (uint32_t)got);
            const unsigned long long hi = __reduce_or_sync(GR_FULL, (uint32_t)(got >> 32));
            got = lo | (hi << 32);
            if (((got | rv) & all) == all) break;
        }
        if ((int)lane == src) acc = got;
    }
    if (!valid) return;
    acc &= ~vis & all;
    next[v] = acc;
    if (acc) {
        visited[v] = vis | acc;
        for (unsigned long long a = acc; a; a &= a - 1) hops[(size_t)(k0 + __ffsll((long long)a) - 1) * n + v] = level;
        *changed = 1u;
    }
}

// DE, EE, DD over every (source s, target v) pair of a k x n hop table; the last
// block folds the block partials in block order into out[0..3).
__global__ void __launch_bounds__(STRESS_T)
k_stress_sums(uint32_t n, uint32_t k, const uint32_t *__restrict__ sources, const uint32_t *__restrict__ hops,
              const float *__restrict__ x, const float *__restrict__ y, double *__restrict__ part, double *out,
              uint32_t *ticket) {
    __shared__ double s_red[STRESS_T / GR_WARP];
    __shared__ bool s_last;
    double de = 0.0, ee = 0.0, dd = 0.0;
    // pairs idx, idx + stride, ... of the k x n table, the quotient and remainder by n
    // carried along
    const uint64_t total = (uint64_t)k * n, stride = (uint64_t)gridDim.x * STRESS_T;
    const uint32_t step_s = (uint32_t)(stride / n), step_v = (uint32_t)(stride % n);
    uint64_t idx = (uint64_t)blockIdx.x * STRESS_T + threadIdx.x;
    uint32_t s = (uint32_t)(idx / n), v = (uint32_t)(idx % n);
    for (; idx < total; idx += stride, s += step_s + (v >= n - step_v ? 1u : 0u), v += v >= n - step_v ? step_v - n : step_v) {
        const uint32_t from = sources[s], h = hops[idx];
        if (v == from || h == HOP_NONE) continue;
        const double dist = (double)h;
        const double dx = (double)(x[v] - x[from]), dy = (double)(y[v] - y[from]);
        const double e = hypot(dx, dy);
        de += dist * e;
        ee += e * e;
        dd += dist * dist;
    }
    de = block_sum_d<STRESS_T>(de, s_red);
    ee = block_sum_d<STRESS_T>(ee, s_red);
    dd = block_sum_d<STRESS_T>(dd, s_red);
    const uint32_t G = gridDim.x;
    if (threadIdx.x == 0) {
        part[blockIdx.x] = de;
        part[G + blockIdx.x] = ee;
        part[2 * G + blockIdx.x] = dd;
    }
    if (!last_block_done(ticket, &s_last)) return;
    if (threadIdx.x < 3) {
        double t = 0.0;
        for (uint32_t b = 0; b < G; b++) t += part[threadIdx.x * G + b];
        out[threadIdx.x] = t;
    }
}

}  // namespace gr
