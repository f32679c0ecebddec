// Deterministic P2G (MPM_P2G_DETERMINISTIC): bitwise identical results from
// run to run.
//
// FP32 atomics make the order of a node's additions depend on scheduling.  This
// mode never adds floats atomically.  Every particle writes its P2G source
// record (stencil fractions, m v, m C, -dt V tau, m; a row of whole float4s) and
// counts itself at its base node; the particles of a base node become one run,
// ordered by creation index (k_det_starts, k_det_slots, k_det_order: a counting
// sort whose counters decide only where a run lies, then each particle's rank
// among its run's indices).  One thread per run sums, particle by particle in
// that order, the run's contributions to each of the 3^D nodes of its stencil
// (k_det_partials: a partial sum per (base node, offset)); then each grid node
// adds, in a fixed offset order, the partials of the 3^D base nodes whose
// stencils cover it (k_det_sum), and stores the sum.  Where a run lies and in
// which order runs and blocks are listed enters no sum.  Particles stay in
// creation order in this mode and the grid update visits the blocks the stencils
// touched, as in the binned path.
//
// Bound by the latency of dependent kernels and their random reads rather than
// by bytes.  A radix sort of 238k keys runs 27 CTAs, three passes of 13 us; the
// counting sort's three kernels take 13 us together, and G2P, update and source of
// a particle are one kernel.  Jello cube of 238k particles in a 101^3 grid: the
// substep takes 86 us instead of 171 (2.1M particles in 256^3: 474 instead of
// 712), bit for bit the radix sort's result.  Three threads per run, one per
// x-plane, were slower (35 us against 26 for the partials) and round differently.
#pragma once

#include "mpm_grid.cuh"
#include "mpm_kernels_binned.cuh"
#include "mpm_particle.cuh"

namespace mpm {

// P2G source record of a particle: [0, D) fx, [D, 2D) m v, [2D, 2D + D^2) m C,
// then A (D^2), then m, padded to whole float4s
template <int D>
struct SrcRow {
    static constexpr int FX = 0, MV = D, MC = 2 * D, A = 2 * D + D * D, M = 2 * D + 2 * D * D;
    static constexpr int COUNT = 2 * D + 2 * D * D + 1;
    static constexpr int N4 = (COUNT + 3) / 4;
};

// what the passes share: per base node, first (.x) and count (while records come
// in), then end (.y) of its run in the order; the key (base node) of each
// particle and its arrival number at it
struct DetCells {
    int2* cells;
    unsigned long long* keys;
    unsigned long long no_cell;  // key of a particle whose stencil left the grid: one past the last node
    unsigned* arrival;
};

// Source record, base node and block marks of particle i at x (its error bits
// when the stencil left the grid)
template <int D>
__device__ __forceinline__ unsigned det_record(long long i, const float* x, const float* v, const float* C,
                                               const float* F, float aux, const GroupParams& g, const SceneParams& sc,
                                               float4* __restrict__ rows, const DetCells& dc,
                                               unsigned* __restrict__ blk_flag, int* __restrict__ active,
                                               int* __restrict__ n_active) {
    using SR = SrcRow<D>;
    unsigned err = 0;
    Stencil<D> st;
    if (!make_stencil<D>(x, sc, st, err)) {
        dc.keys[i] = dc.no_cell;
        return err;
    }
    P2GSource<D> s;
    particle_stress_source<D>(v, C, F, aux, g, sc, s);
    float r[SR::N4 * 4];
#pragma unroll
    for (int k = 0; k < SR::N4 * 4; ++k) r[k] = 0.f;
#pragma unroll
    for (int a = 0; a < D; ++a) {
        r[SR::FX + a] = st.fx[a];
        r[SR::MV + a] = s.mv[a];
    }
#pragma unroll
    for (int k = 0; k < D * D; ++k) {
        r[SR::MC + k] = s.mC[k];
        r[SR::A + k] = s.A[k];
    }
    r[SR::M] = s.m;
#pragma unroll
    for (int q = 0; q < SR::N4; ++q)
        rows[i * SR::N4 + q] = make_float4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
    const long long node = node_index<D>(sc, st.base[0], st.base[1], D == 3 ? st.base[2] : 0);
    dc.keys[i] = (unsigned long long)node;
    dc.arrival[i] = (unsigned)atomicAdd(&dc.cells[node].y, 1);
    mark_stencil<D>(st.base, sc, blk_flag, active, n_active);
    return err;
}

// counters of the deterministic passes: runs listed, particles given a place
struct DetCounters {
    int* n_runs;
    int* placed;
};

// Source records of the state as it is (the first P2G of a state)
template <int D>
__global__ void __launch_bounds__(128) k_det_source(ParticleBuf pb, long long n, const GroupParams* __restrict__ groups,
                                                    const SceneParams* __restrict__ scenes, float4* __restrict__ rows,
                                                    DetCells dc, unsigned* __restrict__ blk_flag,
                                                    int* __restrict__ active, int* __restrict__ n_active,
                                                    DetCounters cnt, unsigned* err_word) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *cnt.n_runs = *cnt.placed = 0;
    if (i >= n) return;
    float x[D], v[D], C[D * D], F[D * D], aux;
    load_particle<D>(pb, i, x, v, C, F, aux);
    const GroupParams g = groups[pb.grp[i]];
    const unsigned err = det_record<D>(i, x, v, C, F, aux, g, scenes[g.scene], rows, dc, blk_flag, active, n_active);
    if (err) atomicOr(err_word, err);
}

// G2P, update and the next substep's source record of every particle
// (k_g2p_direct and k_det_source in one pass over the state); the epoch moves on.
// Ten CTAs of 64 threads an SM hold 20 warps at 96 registers; left alone, the
// compiler takes 124 (16 warps): the substep 98 us against 93.
constexpr int kDetStepThreads = 64;
template <int D>
__global__ void __launch_bounds__(kDetStepThreads, 10) k_det_step(ParticleBuf pb, long long n, const GroupParams* __restrict__ groups,
                                                  const SceneParams* __restrict__ scenes,
                                                  const float4* __restrict__ grid, float4* __restrict__ rows,
                                                  DetCells dc, unsigned* __restrict__ blk_flag,
                                                  int* __restrict__ active, int* __restrict__ n_active, DetCounters cnt,
                                                  int* __restrict__ epoch, unsigned* err_word) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        *cnt.n_runs = *cnt.placed = 0;
        *epoch += 1;
    }
    if (i >= n) return;
    const GroupParams g = groups[pb.grp[i]];
    const SceneParams& sc = scenes[g.scene];
    float x[D], v[D], C[D * D], F[D * D], aux;
    unsigned err = 0;
    if (g2p_update<D>(pb, i, g, sc, grid, x, v, C, F, aux, err))
        err |= det_record<D>(i, x, v, C, F, aux, g, sc, rows, dc, blk_flag, active, n_active);
    else dc.keys[i] = dc.no_cell;
    if (err) atomicOr(err_word, err);
}

// A place for the run of every base node of the touched blocks, and the list of
// the runs: four blocks per CTA turn, one counter add for both
__global__ void __launch_bounds__(256) k_det_starts(int2* __restrict__ cells, const int* __restrict__ blocks,
                                                    const int* __restrict__ n_blocks, int4* __restrict__ runs,
                                                    DetCounters cnt) {
    pdl_wait();
    pdl_trigger();
    __shared__ int2 warp_sum[8];  // particles, runs
    __shared__ int2 start;
    const int nb = *n_blocks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int e0 = blockIdx.x * 4; e0 < nb; e0 += gridDim.x * 4) {
        const int e = e0 + (threadIdx.x >> 6);
        const long long node = e < nb ? (long long)blocks[e] * 64 + (threadIdx.x & 63) : 0;
        const int c = e < nb ? cells[node].y : 0;
        int incl = c;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, k);
            if (lane >= k) incl += up;
        }
        const unsigned used = __ballot_sync(0xffffffffu, c > 0);
        if (lane == 31) warp_sum[warp] = make_int2(incl, __popc(used));
        __syncthreads();
        if (threadIdx.x == 0) {
            int2 sum = make_int2(0, 0);
            for (int w = 0; w < 8; ++w) {
                const int2 v = warp_sum[w];
                warp_sum[w] = sum;
                sum.x += v.x;
                sum.y += v.y;
            }
            start = sum.y ? make_int2(atomicAdd(cnt.placed, sum.x), atomicAdd(cnt.n_runs, sum.y)) : sum;
        }
        __syncthreads();
        if (c > 0) {
            const int j0 = start.x + warp_sum[warp].x + incl - c;
            cells[node] = make_int2(j0, j0 + c);
            runs[start.y + warp_sum[warp].y + __popc(used & ((1u << lane) - 1u))] =
                make_int4((int)(node >> 6), j0, j0 + c, 0);
        }
        __syncthreads();  // the sums are rewritten by the next turn
    }
}

// every particle into its run, in arrival order
__global__ void __launch_bounds__(256) k_det_slots(DetCells dc, long long n, unsigned* __restrict__ slots) {
    pdl_wait();
    pdl_trigger();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long k = dc.keys[i];
    if (k != dc.no_cell) slots[dc.cells[k].x + (int)dc.arrival[i]] = (unsigned)i;
}

// the runs in creation order: a particle's place is the number of smaller
// indices in its run
__global__ void __launch_bounds__(256) k_det_order(DetCells dc, long long n, const unsigned* __restrict__ slots,
                                                   const int* __restrict__ placed, unsigned* __restrict__ order) {
    pdl_wait();
    pdl_trigger();
    const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n || s >= *placed) return;
    const unsigned p = slots[s];
    const int2 run = dc.cells[dc.keys[p]];
    int less = 0;
    for (int j = run.x; j < run.y; ++j) less += slots[j] < p ? 1 : 0;
    order[run.x + less] = p;
}

// One thread per run (its block, first place j0 and end): the run's P2G
// contributions to each stencil node, summed particle by particle in creation
// order, stored as partial[j0 * 3^D + k] with k = (ox * 3 + oy) * 3 + oz (3D) or
// ox * 3 + oy (2D).
template <int D>
__global__ void __launch_bounds__(64, 4) k_det_partials(const float4* __restrict__ rows,
                                                        const unsigned* __restrict__ order,
                                                        const int4* __restrict__ runs, const int* __restrict__ n_runs,
                                                        const SceneParams* __restrict__ scenes, int n_scenes,
                                                        float4* __restrict__ partial) {
    pdl_wait();
    pdl_trigger();
    using SR = SrcRow<D>;
    constexpr int K = D == 3 ? 27 : 9;
    const int nr = *n_runs;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nr; r += gridDim.x * blockDim.x) {
        const int4 run = runs[r];
        const int j0 = run.y, j1 = run.z;
        const SceneParams& sc = scenes[scene_of_block(scenes, n_scenes, run.x)];
        float4 acc[K];
#pragma unroll
        for (int k = 0; k < K; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        // the next record is on its way while this one is summed
        float4 nxt[SR::N4];
        unsigned next = j0 + 1 < j1 ? order[j0 + 1] : 0;
#pragma unroll
        for (int q = 0; q < SR::N4; ++q) nxt[q] = rows[(long long)order[j0] * SR::N4 + q];
        for (int j = j0; j < j1; ++j) {
            float rec[SR::N4 * 4];
#pragma unroll
            for (int q = 0; q < SR::N4; ++q) {
                rec[4 * q] = nxt[q].x;
                rec[4 * q + 1] = nxt[q].y;
                rec[4 * q + 2] = nxt[q].z;
                rec[4 * q + 3] = nxt[q].w;
            }
            if (j + 1 < j1) {
#pragma unroll
                for (int q = 0; q < SR::N4; ++q) nxt[q] = rows[(long long)next * SR::N4 + q];
                if (j + 2 < j1) next = order[j + 2];
            }
            Stencil<D> st;
            P2GSource<D> s;
#pragma unroll
            for (int a = 0; a < D; ++a) {
                st.fx[a] = rec[SR::FX + a];
                s.mv[a] = rec[SR::MV + a];
            }
#pragma unroll
            for (int k = 0; k < D * D; ++k) {
                s.mC[k] = rec[SR::MC + k];
                s.A[k] = rec[SR::A + k];
            }
            s.m = rec[SR::M];
            p2g_scatter<D>(st, s, sc.h, sc.inv_h, [&](int ox, int oy, int oz, float4 c) {
                float4& t = acc[D == 3 ? (ox * 3 + oy) * 3 + oz : ox * 3 + oy];
                t.x += c.x;
                t.y += c.y;
                t.z += c.z;
                t.w += c.w;
            });
        }
#pragma unroll
        for (int k = 0; k < K; ++k) partial[(long long)j0 * K + k] = acc[k];
    }
}

// the cells of the touched blocks back to no particles
__global__ void __launch_bounds__(256) k_det_reset(int2* __restrict__ cells, const int* __restrict__ blocks,
                                                   const int* __restrict__ n_blocks) {
    pdl_wait();
    const int nb = *n_blocks;
    for (int e = blockIdx.x * 4 + (threadIdx.x >> 6); e < nb; e += gridDim.x * 4)
        cells[(long long)blocks[e] * 64 + (threadIdx.x & 63)] = make_int2(0, 0);
}

// Every node of the listed blocks adds, in the order of the stencil offset o,
// the partial sums of the base nodes node - o, o in {0,1,2}^D, and stores the
// total.  Nine loads in flight instead of one: the substep of 109 us takes 100,
// and 3 CTAs an SM, so that they stay in registers, 91 (with 64-thread
// k_det_step CTAs and the next record ahead in k_det_partials).
template <int D>
__global__ void __launch_bounds__(256, 3) k_det_sum(const float4* __restrict__ partial,
                                                 const int2* __restrict__ cells, const int* __restrict__ blocks,
                                                 const int* __restrict__ n_blocks,
                                                 const SceneParams* __restrict__ scenes, int n_scenes,
                                                 float4* __restrict__ grid_mom) {
    pdl_wait();
    pdl_trigger();
    constexpr int K = D == 3 ? 27 : 9;
    const int na = *n_blocks;
    const int lane = threadIdx.x & 63;
    for (int e = blockIdx.x * 4 + (threadIdx.x >> 6); e < na; e += gridDim.x * 4) {
        const int b = blocks[e];
        const SceneParams& sc = scenes[scene_of_block(scenes, n_scenes, b)];
        int id[3];
        block_node_coords<D>(sc, b - sc.block_off, lane, id[0], id[1], id[2]);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        const bool in_grid = id[0] < sc.n[0] && id[1] < sc.n[1] && (D == 2 || id[2] < sc.n[2]);
        if (in_grid) {
#pragma unroll
            for (int ox = 0; ox < 3; ++ox) {
                constexpr int P = D == 3 ? 9 : 3;
                // the runs of an x-plane of base nodes, then their partial sums: loads that do not wait on one another
                int j[P];
#pragma unroll
                for (int q = 0; q < P; ++q) {
                    const int bx = id[0] - ox, by = id[1] - (D == 3 ? q / 3 : q), bz = D == 3 ? id[2] - q % 3 : 0;
                    const int2 run = bx < 0 || by < 0 || bz < 0 ? make_int2(0, 0) : cells[node_index<D>(sc, bx, by, bz)];
                    j[q] = run.y > run.x ? run.x : -1;  // -1: no particle has this base node
                }
                float4 c[P];
#pragma unroll
                for (int q = 0; q < P; ++q)
                    c[q] = j[q] < 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : partial[(long long)j[q] * K + ox * P + q];
#pragma unroll
                for (int q = 0; q < P; ++q) {
                    if (j[q] < 0) continue;
                    acc.x += c[q].x;
                    acc.y += c[q].y;
                    acc.z += c[q].z;
                    acc.w += c[q].w;
                }
            }
        }
        grid_mom[(long long)b * 64 + lane] = acc;
    }
}

}  // namespace mpm
