// Launch configurations of the fused substep kernel (the autotuner's search
// space), shared by the kernels and the C-ABI layer.
#pragma once

namespace mpm {

// Instantiations of the fused kernel.  chunk: threads per CTA; min_ctas: the
// minimum resident CTAs per SM given to __launch_bounds__ (which caps
// registers at 65536 / (chunk * min_ctas)); scatter: how the P2G of the next
// substep reaches the grid -- SCATTER_DIRECT: every particle reduces its 3^D
// node values into global memory (red.global.add.v4.f32); SCATTER_RUNS: the
// particles of a chunk that share a stencil base are summed first and each
// sum is reduced once (mpm_kernels_runs.cuh; the chunk's source records in
// shared memory limit these kernels to fewer CTAs per SM).
enum : int { SCATTER_DIRECT = 0, SCATTER_RUNS = 1 };
struct FusedKernel {
    int chunk;
    int min_ctas;
    int scatter;
};
constexpr int kNumFusedKernels = 12;
constexpr FusedKernel kFusedKernels[kNumFusedKernels] = {
    {128, 4, 0}, {128, 5, 0}, {128, 6, 0}, {64, 8, 0}, {64, 10, 0}, {64, 12, 0}, {256, 2, 0}, {256, 3, 0},
    {128, 5, 1}, {128, 4, 1}, {64, 9, 1}, {64, 7, 1}};

// A launch configuration (the autotuner's search space): an instantiation,
// rounds -- particles each thread processes per chunk, one after the other,
// so a chunk holds chunk * rounds particles and one velocity window and one
// pair of CTA barriers serve them all -- and order: how the re-binning orders
// the particles of a (block, material) segment.  ORDER_RANK: rank-major
// (every cell's first particle, then every cell's second, ...), so a warp's
// 32 lanes sit in 32 different cells and every scatter instruction hits 32
// different nodes; ORDER_CELL: cell-major (a cell's particles together), so
// the lanes of one cell gather the same nodes (shared-memory broadcasts) and
// scatter into the same nodes.
enum : int { ORDER_RANK = 0, ORDER_CELL = 1 };
struct FusedCfg {
    int chunk;
    int min_ctas;
    int rounds;
    int kernel;
    int order;
    int scatter;
};
struct FusedCfgTable {
    static constexpr int N = 36;
    FusedCfg c[N];
    // 0..11 direct scatter, rank-major; 12..23 the same shapes cell-major;
    // 24..31 run sums (cell-major), one to three rounds: two rounds of the
    // 128-thread kernel are the fastest from 400k particles up (256 particles
    // a chunk: about five per run), one round below, where the chunks are too
    // few to fill the SMs; 32..35 the
    // 64-thread, 10-CTA direct kernel with three and four rounds, rank-major
    // and cell-major (fewer window loads and barrier pairs per particle; on
    // the 2M-particle scenes 3-4 % faster than two rounds)
    constexpr FusedCfgTable() : c{} {
        constexpr int kr[12][2] = {{0, 1}, {1, 1}, {2, 1}, {3, 1}, {4, 1}, {5, 1},
                                   {6, 1}, {7, 1}, {1, 2}, {2, 2}, {4, 2}, {7, 2}};
        constexpr int sr[8][2] = {{8, 1}, {8, 2}, {9, 1}, {9, 2}, {9, 3}, {10, 1}, {11, 1}, {11, 2}};
        for (int i = 0; i < 24; ++i) {
            const int k = kr[i % 12][0];
            c[i] = FusedCfg{kFusedKernels[k].chunk, kFusedKernels[k].min_ctas, kr[i % 12][1], k,
                            i < 12 ? ORDER_RANK : ORDER_CELL, SCATTER_DIRECT};
        }
        for (int i = 0; i < 8; ++i) {
            const int k = sr[i][0];
            c[24 + i] = FusedCfg{kFusedKernels[k].chunk, kFusedKernels[k].min_ctas, sr[i][1], k, ORDER_CELL,
                                 SCATTER_RUNS};
        }
        for (int i = 0; i < 4; ++i)
            c[32 + i] = FusedCfg{kFusedKernels[4].chunk, kFusedKernels[4].min_ctas, 3 + i % 2, 4,
                                 i < 2 ? ORDER_RANK : ORDER_CELL, SCATTER_DIRECT};
    }
    constexpr const FusedCfg& operator[](int i) const { return c[i]; }
};
constexpr FusedCfgTable kFusedCfgs{};
constexpr int kNumFusedCfgs = FusedCfgTable::N;
// fewest particles a chunk of any configuration holds (sizes the chunk lists)
constexpr int kMinChunkParticles = 64;

// Whether a configuration sums runs: those declared so, which address a dense
// grid; and in a paged grid the cell-major ones of 128 threads with registers
// to spare (at most 5 CTAs per SM), which declare the direct scatter
constexpr bool sums_runs(int cfg, bool paged) {
    const FusedCfg& c = kFusedCfgs[cfg];
    return paged ? c.scatter == SCATTER_DIRECT && c.order == ORDER_CELL && c.chunk == 128 && c.min_ctas <= 5
                 : c.scatter == SCATTER_RUNS;
}
// Material that sprays leaves chunks of a few particles, for which a CTA of a
// run-sum configuration with several particles per thread pays its window, its
// lists and its three barriers all the same, four or five CTAs an SM.  Such a
// state hands the chunks of at most 64 particles to launches of kSmallCfg, the
// per-particle scatter with ten CTAs an SM, behind (and into, pass_end) the main
// one.  1.9M particles of colliding snow, each from the same state (two particles
// a thread, 27): after 2500 / 3000 / 3500 / 4300 substeps 377 / 462 / 565 / 717 ->
// 328 / 384 / 453 / 559 us a substep, the best per-particle scatter alone (35)
// 360 / 409 / 476 / 582.  While the blocks are full it costs 3-20 %
// (jello 128^3 54.3 -> 66: the list loses its order by size), so it begins when
// the chunks are less than half as full as they were when the configuration was
// timed (autotune; kept with its choice for handles of the same shape) or, for
// one the caller set, when it first ran, and ends when they are fuller than 0.6
// of that.
constexpr bool may_split_small(int cfg, bool paged) { return sums_runs(cfg, paged) && kFusedCfgs[cfg].rounds >= 2; }
constexpr bool wants_split_small(bool now, float fill, float fill_at_first) {
    return fill < (now ? 0.6f : 0.5f) * fill_at_first;
}
constexpr int kSmallCfg = 16;
static_assert(kFusedCfgs[kSmallCfg].scatter == SCATTER_DIRECT && kFusedCfgs[kSmallCfg].rounds == 1 &&
                  kFusedCfgs[kSmallCfg].chunk == 64,
              "a particle per thread");
// SCATTER_RUNS: float4s of a particle's source record, and the dynamic shared
// memory of a chunk (a record and two run-list entries per particle)
constexpr int run_rec4(int dim) { return dim == 3 ? 6 : 4; }
constexpr int run_smem(int dim, int particles) { return particles * (run_rec4(dim) * 16 + 4); }
// dynamic shared memory of a launch configuration
constexpr int fused_dyn_smem(int dim, int cfg, bool paged) {
    return sums_runs(cfg, paged) ? run_smem(dim, kFusedCfgs[cfg].chunk * kFusedCfgs[cfg].rounds) : 0;
}
// the most any configuration of the same instantiation asks for
constexpr int fused_dyn_smem_max(int dim, int cfg, bool paged) {
    int most = 0;
    for (int i = 0; i < kNumFusedCfgs; ++i)
        if (kFusedCfgs[i].kernel == kFusedCfgs[cfg].kernel && fused_dyn_smem(dim, i, paged) > most)
            most = fused_dyn_smem(dim, i, paged);
    return most;
}

constexpr bool fused_cfgs_consistent() {
    for (int i = 0; i < kNumFusedCfgs; ++i) {
        const FusedCfg& c = kFusedCfgs[i];
        if (c.kernel < 0 || c.kernel >= kNumFusedKernels) return false;
        const FusedKernel& k = kFusedKernels[c.kernel];
        if (k.chunk != c.chunk || k.min_ctas != c.min_ctas || k.scatter != c.scatter ||
            (c.order != ORDER_RANK && c.order != ORDER_CELL) ||
            (c.scatter == SCATTER_RUNS && c.order != ORDER_CELL) ||
            c.chunk * c.rounds < kMinChunkParticles || c.chunk % 32 != 0)
            return false;
    }
    return true;
}
static_assert(fused_cfgs_consistent(), "each configuration names the instantiation of its launch shape");

}  // namespace mpm
