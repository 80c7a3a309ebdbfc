// Attraction, gravity, the FP64 swing/traction reductions, the speed controller
// and the position update.
//
// Reference: crates/graph-core/src/layout/forceatlas2/state.rs:152-162 (attraction),
// 208-251 (gravity), state/schedule.rs:16-77 (swing/traction, estimate_factor,
// apply_update); the options graph-core leaves at their defaults follow networkx
// 3.6 `forceatlas2_layout` (networkx/drawing/layout.py:1806-1872): linlog,
// distributed_action (dissuade hubs), strong_gravity, weighted adjacency.
//
// Attraction is a CSR gather: node i sums w_ij * (p_j - p_i) over its own row in
// a fixed order, so there is no scatter and no float atomic, and the sum is the
// same every run. Every reduction folds per-block partials in block order in the
// grid's last block.
#pragma once

#include "common.cuh"
#include "tree.cuh"

namespace gr {

constexpr int FRC_THREADS = 256;
// k_forces and k_update stride over the nodes with at most FRC_MAX_BLOCKS
// blocks (4 per SM): fewer per-block partials and last-block tickets.
constexpr uint32_t FRC_MAX_BLOCKS = 4 * 148;  // measured: 8 and 16 per SM slower (3 and 8 us at 1M nodes)

__host__ __device__ inline uint32_t frc_blocks(uint32_t n) {
    const uint32_t b = (n + FRC_THREADS - 1) / FRC_THREADS;
    return b < 1 ? 1 : (b > FRC_MAX_BLOCKS ? FRC_MAX_BLOCKS : b);
}
// Rows longer than LIGHT_MAX are summed in SEG-entry segments, one warp each,
// so a hub of 30k neighbours costs ~120 warps instead of one thread's 30k steps.
// (64: on the 1M-node power-law tick 3 us faster than 32, 16 slower by 9 us.)
constexpr uint32_t LIGHT_MAX = 64;
constexpr uint32_t SEG = 256;

// One edge's pull on node p from neighbour q: w * (q - p), or with linlog
// w * log(1 + d) / d * (q - p) (networkx layout.py:1806-1813).
template <int D>
__device__ __forceinline__ void attr_term(const float4 &p, const float4 &q, float w, int lin_log, float &a0,
                                          float &a1, float &a2) {
    const float d0 = q.x - p.x, d1 = q.y - p.y, d2 = (D == 3) ? q.z - p.z : 0.f;
    float c = w;
    if (lin_log) {
        const float dist = sqrtf(d0 * d0 + d1 * d1 + d2 * d2);
        c *= dist > 0.f ? log1pf(dist) / dist : 0.f;
    }
    a0 += d0 * c;
    a1 += d1 * c;
    if (D == 3) a2 += d2 * c;
}

// Heavy rows: warp s sums entries [seg_begin(s), seg_begin(s) + SEG) of row
// seg_row[s] (lanes stride by 32, then a fixed butterfly), writing D floats.
// A null wt means every weight is 1.
template <int D>
__global__ void __launch_bounds__(FRC_THREADS)
k_attract_seg(uint32_t nseg, int lin_log, const DevState *st, const float4 *__restrict__ pos,
              const uint32_t *__restrict__ rp, const uint32_t *__restrict__ col, const float *__restrict__ wt,
              const uint32_t *__restrict__ seg_row, const uint32_t *__restrict__ seg_first,
              float *__restrict__ seg_out) {
    if (st->converged) return;
    const uint32_t s = (blockIdx.x * FRC_THREADS + threadIdx.x) / GR_WARP;
    const uint32_t lane = threadIdx.x % GR_WARP;
    if (s >= nseg) return;
    const uint32_t row = seg_row[s];
    const uint32_t e0 = rp[row] + (s - seg_first[row]) * SEG;
    const uint32_t e1 = min(e0 + SEG, rp[row + 1]);
    const float4 p = pos[row];
    float a0 = 0.f, a1 = 0.f, a2 = 0.f;
    for (uint32_t e = e0 + lane; e < e1; e += GR_WARP)
        attr_term<D>(p, pos[col[e]], wt ? wt[e] : 1.f, lin_log, a0, a1, a2);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a0 += __shfl_xor_sync(GR_FULL, a0, o);
        a1 += __shfl_xor_sync(GR_FULL, a1, o);
        if (D == 3) a2 += __shfl_xor_sync(GR_FULL, a2, o);
    }
    if (lane == 0) {
        seg_out[(size_t)s * D] = a0;
        seg_out[(size_t)s * D + 1] = a1;
        if (D == 3) seg_out[(size_t)s * D + 2] = a2;
    }
}

struct ForceParams {
    uint32_t n;
    float gravity;
    int lin_log, strong_gravity, dissuade_hubs;
    double jitter_tolerance;
};

// schedule.rs:33-60 estimate_factor (networkx's helper), FP64.
__device__ __forceinline__ void estimate_factor(DevState *st, double n, double jt) {
    const double swing = st->swing, traction = st->traction;
    const double opt_jitter = 0.05 * sqrt(n);
    const double min_jitter = sqrt(opt_jitter);
    const double min_se = 0.05;
    const double other = fmin(10.0, opt_jitter * traction / (n * n));
    double jitter = jt * fmax(min_jitter, other);
    double se = st->speed_efficiency, speed = st->speed;
    if (swing / traction > 2.0) {
        if (se > min_se) se *= 0.5;
        jitter = fmax(jitter, jt);
    }
    const double target = swing == 0.0 ? INFINITY : jitter * se * traction / swing;
    if (swing > jitter * traction) {
        if (se > min_se) se *= 0.7;
    } else if (speed < 1000.0) {
        se *= 1.3;
    }
    speed += fmin(target - speed, 0.5 * speed);
    st->speed = speed;
    st->speed_efficiency = se;
}

// Node i's force accumulator given its attraction (a*) and repulsion (r*):
// u = attraction (/ mass with dissuade hubs) + repulsion - gravity, gravity the
// unit vector first (state.rs:223-251) or strong (layout.py:1830-1832); writes u
// and returns the node's FP64 swing and traction terms (schedule.rs:16-30).
template <int D>
__device__ __forceinline__ void node_force(const ForceParams &P, const float4 &p, float a0, float a1, float a2,
                                           float r0, float r1, float r2, const double *mean, float *u, double &sw,
                                           double &tr) {
    if (P.dissuade_hubs) {
        a0 /= p.w;
        a1 /= p.w;
        a2 /= p.w;
    }
    float u0 = a0 + r0;
    float u1 = a1 + r1;
    float u2 = (D == 3) ? a2 + r2 : 0.f;
    const float c0 = (float)((double)p.x - mean[0]);
    const float c1 = (float)((double)p.y - mean[1]);
    const float c2 = (D == 3) ? (float)((double)p.z - mean[2]) : 0.f;
    const float g = P.gravity * p.w;
    if (P.strong_gravity) {
        u0 -= g * c0;
        u1 -= g * c1;
        u2 -= g * c2;
    } else {
        const float nrm = sqrtf(c0 * c0 + c1 * c1 + c2 * c2);
        if (nrm > 0.f) {
            u0 -= g * (c0 / nrm);
            u1 -= g * (c1 / nrm);
            u2 -= g * (c2 / nrm);
        }
    }
    u[0] = u0;
    u[1] = u1;
    if (D == 3) u[2] = u2;
    const double m = (double)p.w;
    const double b0 = (double)p.x - u0, b1 = (double)p.y - u1, b2 = (D == 3) ? (double)p.z - u2 : 0.0;
    const double g0 = (double)p.x + u0, g1 = (double)p.y + u1, g2 = (D == 3) ? (double)p.z + u2 : 0.0;
    sw = m * sqrt(b0 * b0 + b1 * b1 + b2 * b2);
    tr = 0.5 * m * sqrt(g0 * g0 + g1 * g1 + g2 * g2);
}

// schedule.rs:62-77 apply_update for one node: factor = speed / (1 + sqrt(speed
// * m * |u|)), p += u * factor; returns |step| summed over the axes (FP64).
template <int D>
__device__ __forceinline__ double node_update(float4 &p, const float *__restrict__ u, double speed, bool &bad) {
    const double u0 = u[0], u1 = u[1], u2 = (D == 3) ? u[2] : 0.0;
    const double nrm = sqrt(u0 * u0 + u1 * u1 + u2 * u2);
    const double factor = speed / (1.0 + sqrt(speed * (double)p.w * nrm));
    const float d0 = (float)(u0 * factor), d1 = (float)(u1 * factor), d2 = (float)(u2 * factor);
    p.x += d0;
    p.y += d1;
    if (D == 3) p.z += d2;
    bad = !(isfinite(p.x) && isfinite(p.y) && isfinite(p.z));
    return fabs((double)d0) + fabs((double)d1) + ((D == 3) ? fabs((double)d2) : 0.0);
}

// Attraction of node i over its own CSR row (rows of <= LIGHT_MAX entries), or
// its segment sums in segment order (longer rows, when seg_first is given).
// A null wt means every weight is 1 (the same terms, without the weight reads).
template <int D>
__device__ __forceinline__ void node_attraction(uint32_t i, const float4 &p, int lin_log,
                                                const float4 *__restrict__ pos, const uint32_t *__restrict__ rp,
                                                const uint32_t *__restrict__ col, const float *__restrict__ wt,
                                                const uint32_t *__restrict__ seg_first,
                                                const float *__restrict__ seg_out, float &a0, float &a1, float &a2) {
    a0 = a1 = a2 = 0.f;
    const uint32_t e0 = rp[i], e1 = rp[i + 1];
    if (seg_first == nullptr || e1 - e0 <= LIGHT_MAX) {
        // four neighbours' gathers in flight at a time, their terms in order (one at a
        // time the linlog tick at 100,000 nodes took 151 us, so 149; unit weights the same)
        constexpr uint32_t U = 4;
        uint32_t e = e0;
        for (; e + U <= e1; e += U) {
            float4 q[U];
            float w[U];
#pragma unroll
            for (uint32_t j = 0; j < U; j++) {
                q[j] = pos[col[e + j]];
                w[j] = wt ? wt[e + j] : 1.f;
            }
#pragma unroll
            for (uint32_t j = 0; j < U; j++) attr_term<D>(p, q[j], w[j], lin_log, a0, a1, a2);
        }
        for (; e < e1; e++) attr_term<D>(p, pos[col[e]], wt ? wt[e] : 1.f, lin_log, a0, a1, a2);
    } else {  // the row's segment sums, in segment order
        const uint32_t s0 = seg_first[i], ns = (e1 - e0 + SEG - 1) / SEG;
        for (uint32_t s = s0; s < s0 + ns; s++) {
            a0 += seg_out[(size_t)s * D];
            a1 += seg_out[(size_t)s * D + 1];
            if (D == 3) a2 += seg_out[(size_t)s * D + 2];
        }
    }
}

// Every node's attraction (node_attraction) into att (n x D). It reads only the
// positions and the graph, so it can run beside the tree build and the walk.
template <int D>
__global__ void __launch_bounds__(FRC_THREADS)
k_attract(uint32_t n, int lin_log, const DevState *st, const float4 *__restrict__ pos,
          const uint32_t *__restrict__ rp, const uint32_t *__restrict__ col, const float *__restrict__ wt,
          const uint32_t *__restrict__ seg_first, const float *__restrict__ seg_out, float *__restrict__ att) {
    if (st->converged) return;
    const uint32_t i = blockIdx.x * FRC_THREADS + threadIdx.x;
    if (i >= n) return;
    float a0, a1, a2;
    node_attraction<D>(i, pos[i], lin_log, pos, rp, col, wt, seg_first, seg_out, a0, a1, a2);
    att[(size_t)i * D] = a0;
    att[(size_t)i * D + 1] = a1;
    if (D == 3) att[(size_t)i * D + 2] = a2;
}

// ---- sums over CSR rows whose terms cost a square root and a quotient. A warp
// takes 32 consecutive rows: its lanes compute the terms of all their entries side
// by side (consecutive entries, whatever the rows' lengths), ROWS_WIN at a time
// into shared memory, and each lane then adds its own row's in entry order, the
// sum a loop over the row gives. One lane a row, the lanes wait for the longest of
// 32 rows, each entry's loads and arithmetic in one serial chain: d3-force's link
// pass at 1M nodes and 3.1M entries took 79 us that way and 43 this way. FA2's
// attraction stays a lane a row: its linear term costs little beside its gather
// (unit weights over 8M entries: 56 us, spread 69), and the row sums run beside
// the walk, whose pipe the shared memory's traffic shares (a 1M-node tick 40 us
// longer).
constexpr int ROWS_WIN = 128;

template <int D>
struct RowsShared {  // one warp's
    float4 p[GR_WARP];
    uint32_t pre[GR_WARP], base[GR_WARP];
    float v[D + 1][ROWS_WIN];
};

// acc += the terms of this lane's row (row0 + lane): `len` entries from e0, p its
// record. term(p, row, e, q, d) gives the factor of entry e, whose neighbour's
// record is q, and its D components in d. The whole warp calls it.
template <int D, typename Col, typename Term>
__device__ __forceinline__ void warp_rows(RowsShared<D> &S, uint32_t row0, const float4 &p, uint32_t e0,
                                          uint32_t len, float *acc, const float4 *__restrict__ pos, Col col, Term term) {
    const uint32_t lane = threadIdx.x % GR_WARP;
    uint32_t inc = len;
#pragma unroll
    for (int o = 1; o < GR_WARP; o <<= 1) {
        const uint32_t y = __shfl_up_sync(GR_FULL, inc, o);
        if (lane >= (uint32_t)o) inc += y;
    }
    const uint32_t total = __shfl_sync(GR_FULL, inc, GR_WARP - 1), pre = inc - len;
    S.p[lane] = p;
    S.pre[lane] = pre;
    S.base[lane] = e0 - pre;
    __syncwarp();
    for (uint32_t w0 = 0; w0 < total; w0 += ROWS_WIN) {
#pragma unroll
        for (int u = 0; u < ROWS_WIN / GR_WARP; u++) {
            const uint32_t slot = u * GR_WARP + lane, t = w0 + slot;
            if (t < total) {
                uint32_t r = 0;  // the last row that begins at or before t
#pragma unroll
                for (uint32_t h = GR_WARP / 2; h >= 1; h >>= 1)
                    if (S.pre[r + h] <= t) r += h;
                float d[D];
                const uint32_t e = t + S.base[r];
                const float c = term(S.p[r], row0 + r, e, pos[col(e)], d);
#pragma unroll
                for (int a = 0; a < D; a++) S.v[a][slot] = d[a];
                S.v[D][slot] = c;
            }
        }
        __syncwarp();
        const uint32_t t1 = min(pre + len, w0 + ROWS_WIN);
        for (uint32_t t = max(pre, w0); t < t1; t++) {
            const float c = S.v[D][t - w0];
#pragma unroll
            for (int a = 0; a < D; a++) acc[a] = __fmaf_rn(S.v[a][t - w0], c, acc[a]);
        }
        __syncwarp();
    }
}

// Rows of more than LIGHT_MAX entries are summed in SEG-entry segments, one warp
// each (lanes stride by 32, then a fixed butterfly); the warp that finishes a
// row's last segment adds the segment sums in segment order. `done` counts a row's
// finished segments at the index of its first one, and is 0 again afterwards.
// Returns whether this lane holds the row's sum in acc (lane 0 of that warp).
template <int D, typename Col, typename Term>
__device__ __forceinline__ bool warp_segment(uint32_t s, uint32_t row, uint32_t first, uint32_t r0, uint32_t r1,
                                             float *seg_out, uint32_t *done, float *acc,
                                             const float4 *__restrict__ pos, Col col, Term term) {
    const uint32_t lane = threadIdx.x % GR_WARP;
    const uint32_t e0 = r0 + (s - first) * SEG, e1 = min(e0 + SEG, r1);
#pragma unroll
    for (int a = 0; a < D; a++) acc[a] = 0.f;
    const float4 p = pos[row];
    for (uint32_t e = e0 + lane; e < e1; e += GR_WARP) {
        float d[D];
        const float c = term(p, row, e, pos[col(e)], d);
#pragma unroll
        for (int a = 0; a < D; a++) acc[a] = __fmaf_rn(d[a], c, acc[a]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int a = 0; a < D; a++) acc[a] += __shfl_xor_sync(GR_FULL, acc[a], o);
    if (lane != 0) return false;
#pragma unroll
    for (int a = 0; a < D; a++) __stcg(&seg_out[(size_t)s * D + a], acc[a]);
    __threadfence();
    const uint32_t ns = (r1 - r0 + SEG - 1) / SEG;
    if (atomicAdd(&done[first], 1u) != ns - 1) return false;
    __threadfence();
    done[first] = 0u;
#pragma unroll
    for (int a = 0; a < D; a++) acc[a] = 0.f;
    for (uint32_t k = first; k < first + ns; k++)
#pragma unroll
        for (int a = 0; a < D; a++) acc[a] += __ldcg(&seg_out[(size_t)k * D + a]);
    return true;
}

// A graph's heavy rows, none when count is 0.
struct Segments {
    uint32_t count;
    const uint32_t *row, *first;  // segment -> row, row -> its first segment
    float *out;                   // D a segment
    uint32_t *done;               // zero
};

__host__ __device__ inline uint32_t seg_blocks(uint32_t count) {
    return (uint32_t)(((uint64_t)count * GR_WARP + FRC_THREADS - 1) / FRC_THREADS);
}
__host__ __device__ inline uint32_t rows_grid(uint32_t n, uint32_t segs) {
    return seg_blocks(segs) + (n + FRC_THREADS - 1) / FRC_THREADS;
}

// Every row's sum of term over its CSR entries, by blocks of FRC_THREADS threads:
// the segments' blocks first, then one lane a row with the warp's lanes
// sharing the terms. col(e) is entry e's neighbour; put(row, acc) takes each sum.
template <int D, typename Col, typename Term, typename Put>
__device__ __forceinline__ void block_rows(uint32_t n, const float4 *__restrict__ pos, const uint32_t *__restrict__ rp,
                                           const Segments &G, Col col, Term term, Put put) {
    const uint32_t sb = seg_blocks(G.count);
    float acc[D];
    if (blockIdx.x < sb) {
        const uint32_t s = (blockIdx.x * FRC_THREADS + threadIdx.x) / GR_WARP;
        if (s >= G.count) return;
        const uint32_t row = G.row[s];
        if (warp_segment<D>(s, row, G.first[row], rp[row], rp[row + 1], G.out, G.done, acc, pos, col, term)) put(row, acc);
        return;
    }
    const uint32_t i = (blockIdx.x - sb) * FRC_THREADS + threadIdx.x, row0 = i & ~(GR_WARP - 1u);
    if (row0 >= n) return;
    const bool valid = i < n;
    const uint32_t e0 = valid ? rp[i] : 0u;
    uint32_t len = valid ? rp[i + 1] - e0 : 0u;
    const bool heavy = G.count != 0u && len > LIGHT_MAX;
    if (heavy) len = 0u;
    const float4 p = valid ? pos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int a = 0; a < D; a++) acc[a] = 0.f;
    __shared__ RowsShared<D> s_rows[FRC_THREADS / GR_WARP];
    warp_rows<D>(s_rows[threadIdx.x / GR_WARP], row0, p, e0, len, acc, pos, col, term);
    if (valid && !heavy) put(i, acc);
}

// u_i for every node from its attraction (read from U, where k_attract put it;
// each thread reads and then overwrites only its own node's entries) and its
// repulsion; per-block FP64 swing and traction; the last block accumulates
// them into the state (cumulative, state.rs:141-143) and runs estimate_factor.
template <int D>
__global__ void __launch_bounds__(FRC_THREADS)
k_forces(ForceParams P, DevState *st, const float4 *__restrict__ pos, const float *__restrict__ rep, float *U,
         double *__restrict__ part, int speed_update) {
    gr_pdl_enter();
    if (st->converged) return;
    __shared__ double s_red[FRC_THREADS / GR_WARP][2];
    __shared__ bool s_last;
    double sum[2] = {0.0, 0.0};  // swing, traction
    const double mean[3] = {st->mean[0], st->mean[1], st->mean[2]};
    for (uint32_t i = blockIdx.x * FRC_THREADS + threadIdx.x; i < P.n; i += gridDim.x * FRC_THREADS) {
        const float4 p = pos[i];
        float *u = U + (size_t)i * D;
        const float a0 = u[0], a1 = u[1], a2 = D == 3 ? u[2] : 0.f;
        double s1, t1;
        node_force<D>(P, p, a0, a1, a2, rep[(size_t)i * D + 0], rep[(size_t)i * D + 1],
                      D == 3 ? rep[(size_t)i * D + 2] : 0.f, mean, u, s1, t1);
        sum[0] += s1;
        sum[1] += t1;
    }
    if (!speed_update) return;
    block_sums_d<FRC_THREADS, 2>(sum, s_red);
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = sum[0];
        part[2 * blockIdx.x + 1] = sum[1];
    }
    if (!last_block_done(&st->counters[1], &s_last)) return;
    sum[0] = strided_sum_cg<FRC_THREADS>(part, gridDim.x, 2, 0);
    sum[1] = strided_sum_cg<FRC_THREADS>(part, gridDim.x, 2, 1);
    block_sums_d<FRC_THREADS, 2>(sum, s_red);
    if (threadIdx.x == 0) {
        st->swing += sum[0];
        st->traction += sum[1];
        estimate_factor(st, (double)P.n, P.jitter_tolerance);
    }
}

// The update for every node; FP64 sum of |step| decides the 1e-10 early exit
// (state.rs:122-128). The same pass also takes the new positions'
// extent and FP64 sums (bounds_block / bounds_finish over k_bounds' grid and
// per-thread order, so the same bits k_bounds would get) into the root square
// and mean of the next tick, and stamps them valid for it.
// On a small grid both this pass and k_forces are the latency of their reductions:
// sums taken together, extents by warp shuffles, one fence a block and a root
// square that starts near its size took a 1,500-node tick from 70.4 to 63.3 us with
// the leaf prefix's shorter folds (100,000 nodes: 158 to 151; same bits).
static_assert(FRC_THREADS == BND_THREADS, "k_update and k_bounds share one grid shape");
template <int D>
__global__ void __launch_bounds__(FRC_THREADS)
k_update(uint32_t n, DevState *st, float4 *__restrict__ pos, const float *__restrict__ U,
         double *__restrict__ part, double *__restrict__ bpart) {
    gr_pdl_enter();
    if (st->converged) return;
    __shared__ double s_red[BND_W][D + 1], s_g[2 * D][BND_W];
    __shared__ float s_f[2 * D][BND_W];
    __shared__ bool s_last;
    double sum[D + 1];  // the new positions', then the steps'
    bool bad = false;
    const double speed = st->speed;
    float lo[D], hi[D];
    sum[D] = 0.0;
#pragma unroll
    for (int a = 0; a < D; a++) {
        lo[a] = INFINITY;
        hi[a] = -INFINITY;
        sum[a] = 0.0;
    }
    for (uint32_t i = blockIdx.x * FRC_THREADS + threadIdx.x; i < n; i += gridDim.x * FRC_THREADS) {
        float4 p = pos[i];
        bool b;
        sum[D] += node_update<D>(p, U + (size_t)i * D, speed, b);
        bad = bad || b;
        pos[i] = p;
        const float c[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int a = 0; a < D; a++) {
            lo[a] = fminf(lo[a], c[a]);
            hi[a] = fmaxf(hi[a], c[a]);
            sum[a] += (double)c[a];
        }
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(&st->error, (uint32_t)ERR_NONFINITE);
    bounds_block<D, D + 1>(lo, hi, sum, bpart, s_red, s_f);
    if (threadIdx.x == 0) part[blockIdx.x] = sum[D];
    if (!last_block_done(&st->counters[2], &s_last)) return;
    sum[D] = strided_sum_cg<FRC_THREADS>(part, gridDim.x, 1, 0);
    bounds_finish<D, D + 1>(bpart, n, st, sum, s_red, s_g);
    if (threadIdx.x == 0) {
        st->moved = sum[D];
        st->iter_no += 1;
        if (sum[D] < 1e-10 || st->error) st->converged = 1;
        st->bounds_stamp = st->iter_no + 1u;
    }
}

// Row-major n x D copy of the float4 positions (the per-tick buffer); with
// nonfinite, a non-finite coordinate sets it to 1.
template <int D>
__global__ void k_export(uint32_t n, const float4 *__restrict__ pos, float *__restrict__ out,
                         uint32_t *nonfinite = nullptr) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 p = pos[i];
    out[(size_t)i * D] = p.x;
    out[(size_t)i * D + 1] = p.y;
    if (D == 3) out[(size_t)i * D + 2] = p.z;
    if (nonfinite && !(isfinite(p.x) && isfinite(p.y) && (D == 2 || isfinite(p.z)))) *nonfinite = 1u;
}

template <int D>
__global__ void k_import(uint32_t n, float4 *__restrict__ pos, const float *__restrict__ in) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 p = pos[i];
    p.x = in[(size_t)i * D];
    p.y = in[(size_t)i * D + 1];
    p.z = (D == 3) ? in[(size_t)i * D + 2] : 0.f;
    pos[i] = p;
}

}  // namespace gr
