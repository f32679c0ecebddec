// Fused substep whose P2G sums the particles that share a stencil base before
// it reduces into the grid (SCATTER_RUNS).  Same pass as k_g2p2g, in two
// phases per chunk:
//   A. every thread: G2P, update and stress of its particles; each particle's
//      P2G source goes to a record in shared memory and onto the list of the
//      records with its base node (a run: one exchange on the base's head);
//   B. a thread per (run, x-plane of the stencil): walks the run's records,
//      sums its nine nodes in registers and reduces each once.
// k_g2p2g is bound by the L1 data pipe and the L1-to-L2 request path (66 % busy
// each on the 2M-particle jello scene): a float4 reduction instruction takes 26
// data wavefronts, and it issues 27 per particle.  Here a run's particles share
// its 27 reductions (39.3M -> 5.0M reduction requests' sectors per launch).  What
// bounds it now: the issue rate (60 % of the slots, 16 warps an SM), the data
// pipe (56 %: window gathers and records) and the waits at the three barriers of
// a chunk (1.6 stall cycles per issue).  Substep, the best configuration of the
// per-particle scatter with the decomposed stress against run sums with the
// polar one: jello 256^3 2M particles 320 -> 203 us, snow 256^3 331 -> 217, jello
// 128^3 450k 90 -> 54.7, water 149 x 122 x 83 600k 104 -> 64, 16 mixed scenes 376
// -> 216, 2D water 40k 12.5 -> 9.1, paged snow 152 -> 103.  By themselves the run
// sums took jello 256^3 from 320 to 260, snow to 300.
// The records stay in the order of the particles: linking them per base (one
// exchange each) needs no sort, and a drifted particle joins its new base's run.
// Ordering the runs by length (a counting sort over 16 lengths whose counts the
// insertions keep) keeps a warp's lanes on runs of about one length: fused pass
// 248 -> 239 us, jello 128^3 70.5 -> 67.7.  Letting a warp start on the next chunk
// before the others have summed their runs (the first barrier moved to the first
// record) was slower: the values live across it spill (213 -> 217 us).
#pragma once

#include "mpm_kernels_binned.cuh"

namespace mpm {

// bases a stencil inside the window can have, per axis and in all
template <int D>
struct RunShape {
    static constexpr int B = TileShape<D>::T - 2;
    static constexpr int N = D == 3 ? B * B * B : B * B;
    static constexpr int PLANES = D == 3 ? 3 : 1;  // threads per run
};
// run-list entry of a particle whose stencil left the window: this bit and its slot
constexpr unsigned kRunOutside = 0x8000u;
// runs are ordered by length, those of kRunBins or more together
constexpr int kRunBins = 16;

__device__ __forceinline__ float2 dup2(float s) { return make_float2(s, s); }

// A particle's source record: with alpha = m v - h (m C) f, beta = h m C and
// A' = A / h (p2g_scatter), columns of beta and the symmetric A' as
//   3D  (alpha, m) (beta_0, fx) (beta_1, fy) (beta_2, fz)
//       (A'00, A'01, A'01, A'11) (A'02, A'12, A'22, next)
//   2D  (alpha, m, next) (beta_0, beta_1) (A'00, A'01, A'01, A'11) (fx, fy)
template <int D>
__device__ __forceinline__ void write_record(float4* __restrict__ r, const Stencil<D>& st, const P2GSource<D>& src,
                                             float h, float inv_h, int next) {
    float alpha[D], beta[D][D], Ap[D][D];
#pragma unroll
    for (int c = 0; c < D; ++c) {
        float a0 = src.mv[c];
#pragma unroll
        for (int b = 0; b < D; ++b) {
            a0 = fmaf(-h * src.mC[c * D + b], st.fx[b], a0);
            beta[c][b] = h * src.mC[c * D + b];
            Ap[c][b] = inv_h * src.A[c * D + b];
        }
        alpha[c] = a0;
    }
    if constexpr (D == 3) {
        r[0] = make_float4(alpha[0], alpha[1], alpha[2], src.m);
        r[1] = make_float4(beta[0][0], beta[1][0], beta[2][0], st.fx[0]);
        r[2] = make_float4(beta[0][1], beta[1][1], beta[2][1], st.fx[1]);
        r[3] = make_float4(beta[0][2], beta[1][2], beta[2][2], st.fx[2]);
        r[4] = make_float4(Ap[0][0], Ap[0][1], Ap[0][1], Ap[1][1]);
        r[5] = make_float4(Ap[0][2], Ap[1][2], Ap[2][2], __int_as_float(next));
    } else {
        r[0] = make_float4(alpha[0], alpha[1], src.m, __int_as_float(next));
        r[1] = make_float4(beta[0][0], beta[1][0], beta[0][1], beta[1][1]);
        r[2] = make_float4(Ap[0][0], Ap[0][1], Ap[0][1], Ap[1][1]);
        r[3] = make_float4(st.fx[0], st.fx[1], 0.f, 0.f);
    }
}

// Sums of one run over the nine nodes (oy, oz) of stencil plane ox (3D; the
// nodes (ox, oy) in 2D).  With per-plane vectors
//   a = wx (alpha + ox beta_0) + dx A'_0, b = wx beta_1, c = wx beta_2,
//   e = wx A'_1, g = wx A'_2
// node (oy, oz) gets wz (U + oz V) + dz W, U = wy (a + oy b) + dy e,
// V = wy c, W = wy g: the contraction of p2g_scatter, x taken first.
struct PlaneSums {
    float2 xy[9];
    float z[9], m[9];
};

__device__ __forceinline__ void axis3(float f, float (&w)[3], float (&d)[3]) {
    const float t0 = 1.5f - f, t1 = f - 1.f, t2 = f - 0.5f;
    w[0] = 0.5f * t0 * t0;
    w[1] = 0.75f - t1 * t1;
    w[2] = 0.5f * t2 * t2;
    d[0] = -t0;
    d[1] = -2.f * t1;
    d[2] = t2;
}

__device__ __forceinline__ void sum_plane3(const float4* __restrict__ recs, int slot, int ox, PlaneSums& acc) {
    // wx(ox) = s t^2 + k, wx' = 2 s t, t = fx - c
    const float c = 1.5f - 0.5f * (float)ox, s = ox == 1 ? -1.f : 0.5f, k = ox == 1 ? 0.75f : 0.f;
    const float2 o2 = dup2((float)ox);
#pragma unroll
    for (int n = 0; n < 9; ++n) {
        acc.xy[n] = make_float2(0.f, 0.f);
        acc.z[n] = acc.m[n] = 0.f;
    }
    do {
        const float4* r = recs + slot * run_rec4(3);
        const float4 q5 = r[5], q0 = r[0], q1 = r[1], q2 = r[2], q3 = r[3], q4 = r[4];
        slot = __float_as_int(q5.w);
        const float t = q1.w - c, st = s * t, wx = fmaf(st, t, k), dx = st + st;
        const float2 wx2 = dup2(wx);
        const float2 a = __ffma2_rn(wx2, __ffma2_rn(o2, make_float2(q1.x, q1.y), make_float2(q0.x, q0.y)),
                                    __fmul2_rn(dup2(dx), make_float2(q4.x, q4.y)));
        const float a_z = fmaf(wx, fmaf(o2.x, q1.z, q0.z), dx * q5.x);
        const float2 b = __fmul2_rn(wx2, make_float2(q2.x, q2.y)), cc = __fmul2_rn(wx2, make_float2(q3.x, q3.y));
        const float2 e = __fmul2_rn(wx2, make_float2(q4.z, q4.w)), g = __fmul2_rn(wx2, make_float2(q5.x, q5.y));
        const float b_z = wx * q2.z, c_z = wx * q3.z, e_z = wx * q5.y, g_z = wx * q5.z, mw = wx * q0.w;
        float wy[3], dy[3], wz[3], dz[3];
        axis3(q2.w, wy, dy);
        axis3(q3.w, wz, dz);
#pragma unroll
        for (int oy = 0; oy < 3; ++oy) {
            const float2 wy2 = dup2(wy[oy]);
            float2 U = __ffma2_rn(wy2, a, __fmul2_rn(dup2(dy[oy]), e));
            float U_z = fmaf(wy[oy], a_z, dy[oy] * e_z);
            if (oy > 0) {
                const float wo = (float)oy * wy[oy];
                U = __ffma2_rn(dup2(wo), b, U);
                U_z = fmaf(wo, b_z, U_z);
            }
            const float2 V = __fmul2_rn(wy2, cc), W = __fmul2_rn(wy2, g);
            const float V_z = wy[oy] * c_z, W_z = wy[oy] * g_z, M = mw * wy[oy];
#pragma unroll
            for (int oz = 0; oz < 3; ++oz) {
                if (oz > 0) {
                    U = __fadd2_rn(U, V);
                    U_z += V_z;
                }
                const int n = oy * 3 + oz;
                acc.xy[n] = __ffma2_rn(dup2(wz[oz]), U, __ffma2_rn(dup2(dz[oz]), W, acc.xy[n]));
                acc.z[n] = fmaf(wz[oz], U_z, fmaf(dz[oz], W_z, acc.z[n]));
                acc.m[n] = fmaf(wz[oz], M, acc.m[n]);
            }
        }
    } while (slot >= 0);
}

__device__ __forceinline__ void sum_plane2(const float4* __restrict__ recs, int slot, PlaneSums& acc) {
#pragma unroll
    for (int n = 0; n < 9; ++n) {
        acc.xy[n] = make_float2(0.f, 0.f);
        acc.z[n] = acc.m[n] = 0.f;
    }
    do {
        const float4* r = recs + slot * run_rec4(2);
        const float4 q0 = r[0], q1 = r[1], q2 = r[2], q3 = r[3];
        slot = __float_as_int(q0.w);
        float wx[3], dx[3], wy[3], dy[3];
        axis3(q3.x, wx, dx);
        axis3(q3.y, wy, dy);
#pragma unroll
        for (int ox = 0; ox < 3; ++ox) {
            float2 a = make_float2(q0.x, q0.y);
            if (ox > 0) a = __ffma2_rn(dup2((float)ox), make_float2(q1.x, q1.y), a);
            a = __ffma2_rn(dup2(wx[ox]), a, __fmul2_rn(dup2(dx[ox]), make_float2(q2.x, q2.y)));
            const float2 b = __fmul2_rn(dup2(wx[ox]), make_float2(q1.z, q1.w));
            const float2 e = __fmul2_rn(dup2(wx[ox]), make_float2(q2.z, q2.w));
            const float mw = q0.z * wx[ox];
#pragma unroll
            for (int oy = 0; oy < 3; ++oy) {
                const int n = ox * 3 + oy;
                if (oy > 0) a = __fadd2_rn(a, b);
                acc.xy[n] = __ffma2_rn(dup2(wy[oy]), a, __ffma2_rn(dup2(dy[oy]), e, acc.xy[n]));
                acc.m[n] = fmaf(wy[oy], mw, acc.m[n]);
            }
        }
    } while (slot >= 0);
}

// Shared memory of a run-sum pass
template <int D>
struct __align__(128) RunShared {
    float4 tv[TileShape<D>::VN];      // the chunk's velocity window
    Chunk ch[2];                      // records of this and the next chunk
    int head[2][RunShape<D>::N];      // first record of each base's run, -1: none
    int cnt[RunShape<D>::N];          // its length, reset by its reader
    int level[2][kRunBins];           // runs longer than k
    int taken[kRunBins];              // runs of a length given a place so far
    int s27[2][27];                   // PAGED: the windows' physical blocks
    int n_runs[2];
    int list[2];                      // large and all chunks of the launch
    unsigned touched[2];              // 3^D neighbour-block bits
    int next[2];
    unsigned speed;                   // adaptive dt: this chunk's max signal speed
    unsigned long long bar;
};

// Puts particle li's P2G source on the list of its base node (phase A)
template <int D>
__device__ __forceinline__ void insert_record(RunShared<D>& sm, float4* recs, unsigned short* runs, int b, int li,
                                              const Stencil<D>& sn, const P2GSource<D>& src, const SceneParams& sc,
                                              const int* o, const FusedArgs& A) {
    using RS = RunShape<D>;
    int next = -1;
    if (in_window<D>(sn.base, o)) {
        const int l0 = sn.base[0] - o[0], l1 = sn.base[1] - o[1], l2 = D == 3 ? sn.base[2] - o[2] : 0;
        const int key = l0 + RS::B * (l1 + RS::B * l2);
        next = atomicExch(&sm.head[b][key], li);
        // the run now has more than `longer` records; one record of a run says so
        const int longer = atomicAdd(&sm.cnt[key], 1);
        if (longer < kRunBins) atomicAdd(&sm.level[b][longer], 1);
        if (next < 0) {
            runs[atomicAdd(&sm.n_runs[b], 1)] = (unsigned short)key;
            atomicOr(&sm.touched[b], touched_bits<D>(l0, l1, l2));
        }
    } else {
        atomicAdd(A.fallback, 1u);
        atomicAdd(&sm.level[b][0], 1);
        runs[atomicAdd(&sm.n_runs[b], 1)] = (unsigned short)(kRunOutside | (unsigned)li);
    }
    write_record<D>(recs + li * run_rec4(D), sn, src, sc.h, sc.inv_h, next);
}

template <int D>
__device__ __forceinline__ void load_position(const ParticleBuf& pb, long long i, float* x) {
#pragma unroll
    for (int a = 0; a < D; ++a) x[a] = pb.s[(Planes<D>::X + a) * pb.cap + i];
}

// The pass of a CTA over its chunks.  round(ch, sc, o, b, li, x, speed_bits) is
// phase A of one particle of every thread (li >= ch.count: none), at position x
// (the round may overwrite it); it puts the
// P2G source it computes on the lists of parity b with insert_record.
template <int D, int CHUNK, bool FIXED, bool PAGED, class Round>
__device__ __forceinline__ void run_chunks(const ParticleBuf& pb, const FusedArgs& A, RunShared<D>& sm, float4* recs,
                                           unsigned short* runs, Round round) {
    using P = Planes<D>;
    using RS = RunShape<D>;
    constexpr bool TMA = FIXED && !PAGED;
    unsigned short* sorted = runs + A.chunk_cap;
    for (int t = threadIdx.x; t < RS::N; t += CHUNK) {
        sm.head[0][t] = sm.head[1][t] = -1;
        sm.cnt[t] = 0;
    }
    if (threadIdx.x < kRunBins) sm.level[0][threadIdx.x] = sm.level[1][threadIdx.x] = sm.taken[threadIdx.x] = 0;
    if (threadIdx.x < 2) {
        sm.n_runs[threadIdx.x] = 0;
        sm.touched[threadIdx.x] = 0u;
    }
    if (threadIdx.x == 0) {
        sm.speed = 0u;
        if constexpr (TMA) {
            mbar_init(&sm.bar);
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        }
    }
    // The chunk list was last written before the grid update ahead of this launch
    // began: a CTA starts once that kernel's CTAs (or those of another material's
    // pass) have all passed their own wait, so its kernels' writes are in L2.  Its
    // length and the first chunk's record are fetched from there (an SM's L1 may
    // hold older lines until the wait) before this kernel's wait, the record ahead
    // of knowing whether it lies at the front; everything else after the wait.  By
    // two threads: read by all of them past L1, the length alone cost 1.4 us of
    // the 8.8 us of a 2D water substep.
    // the first chunk is the CTA's own index, later ones come from the cursor
    int cur = blockIdx.x;
    if (threadIdx.x < 2) {
        if (threadIdx.x == 0) pass_acquire(A);
        const int n_front = __ldcg(A.n_chunks), n_back = __ldcg(A.n_chunks + kMats);
        const int large = A.part == PART_SMALL ? 0 : n_front, all = large + (A.part == PART_LARGE ? 0 : n_back);
        const int4* front = reinterpret_cast<const int4*>(A.chunks + cur) + threadIdx.x;
        int4 half = A.part != PART_SMALL && cur < A.list_cap ? __ldcg(front) : make_int4(0, 0, 0, 0);
        if (cur >= large && cur < all)
            half = __ldcg(reinterpret_cast<const int4*>(A.chunks + (A.list_cap - 1 - (cur - large))) + threadIdx.x);
        reinterpret_cast<int4*>(&sm.ch[0])[threadIdx.x] = half;
        sm.list[threadIdx.x] = threadIdx.x ? all : large;
    }
    __syncthreads();  // the record, the barrier and the lists initialised
    const ChunkList list(sm.list[0], sm.list[1]);
    const int nch = list.all;
    pass_begin(A);  // the grid update ahead has finished
    if (cur < nch) load_window<D, CHUNK, FIXED, PAGED>(A, sm.ch[0], sm.tv, sm.s27[0], &sm.bar);
    cp_async_commit();
    SpeedFlush speed;
    for (int k = 0; cur < nch; ++k) {
        const int b = k & 1;
        int nxt = 0;
        if (threadIdx.x == 0) nxt = (int)gridDim.x + atomicAdd(A.cursor, 1);
        const Chunk ch = sm.ch[b];
        // the first round's positions, on their way while the window arrives
        float x[D];
        if ((int)threadIdx.x < ch.count) load_position<D>(pb, (long long)ch.start + threadIdx.x, x);
        cp_async_wait<0>();
        // (1) the window and the chunk's record are there; the last chunk's runs are summed
        if constexpr (TMA) {
            const bool ok = mbar_wait(&sm.bar, (unsigned)k & 1u);
            if (__syncthreads_or(!ok)) {  // a window that never arrived: report it and stop
                if (threadIdx.x == 0) atomicOr(A.err_word, ERR_TIMEOUT);
                break;
            }
        } else {
            __syncthreads();
        }
        const SceneParams& sc = chunk_scene<FIXED>(A, ch.scene);
        const int o[3] = {ch.o[0], ch.o[1], ch.o[2]};
        unsigned speed_bits = 0u;
#pragma unroll 1
        for (int r = 0; r * CHUNK < ch.count; ++r) {
            const int li = (int)threadIdx.x + r * CHUNK;
            if (r > 0 && li < ch.count) load_position<D>(pb, (long long)ch.start + li, x);
            round(ch, sc, o, b, li, x, speed_bits);
            // the next chunk's record, on its way while the rest of this phase runs
            if (r == 0 && threadIdx.x == 0 && nxt < nch) {
                const char* from = reinterpret_cast<const char*>(list.at(A, nxt));
                char* to = reinterpret_cast<char*>(&sm.ch[b ^ 1]);
                cp_async16(to, from, true);
                cp_async16(to + 16, from + 16, true);
            }
        }
        if (A.speed_max) speed_warp_reduce(speed_bits, &sm.speed);
        if (threadIdx.x == 0) {
            sm.next[b] = nxt;
            cp_async_commit();
            cp_async_wait<0>();
        }
        __syncthreads();  // (2) records, runs and the next chunk's record complete; the window is free
        const int next_chunk = sm.next[b];
        if (next_chunk < nch) load_window<D, CHUNK, FIXED, PAGED>(A, sm.ch[b ^ 1], sm.tv, sm.s27[b ^ 1], &sm.bar);
        cp_async_commit();
        mark_touched<D>(sm.touched[b], sc, o, A);
        speed.fold(ch.scene, &sm.speed, A.speed_max);
        // the other parity's lists were last read before barrier (1)
        for (int t = threadIdx.x; t < RS::N; t += CHUNK) sm.head[b ^ 1][t] = -1;
        if (threadIdx.x == 0) {
            sm.n_runs[b ^ 1] = 0;
            sm.touched[b ^ 1] = 0u;
        }
        // the runs by length, the longest first, so that the lanes of a warp
        // walk runs of about one length: a run's place is the number of longer
        // runs, counted as the records came in, plus its turn among those of its
        // length (those of kRunBins or more together)
        const int nr = sm.n_runs[b];
        if (threadIdx.x < kRunBins) sm.level[b ^ 1][threadIdx.x] = 0;
        for (int t = threadIdx.x; t < nr; t += CHUNK) {
            const unsigned e = runs[t];
            int len = 1;
            if (!(e & kRunOutside)) {
                len = sm.cnt[e];
                sm.cnt[e] = 0;
            }
            const int k = min(len, kRunBins) - 1;
            const int longer = k + 1 < kRunBins ? sm.level[b][k + 1] : 0;
            sorted[longer + atomicAdd(&sm.taken[k], 1)] = (unsigned short)e;
        }
        __syncthreads();  // (3)
        if (threadIdx.x < kRunBins) sm.taken[threadIdx.x] = 0;
        // ---- phase B
        const int items = nr * RS::PLANES;
        for (int it = threadIdx.x; it < items; it += CHUNK) {
            const int run = D == 3 ? it / 3 : it, ox = D == 3 ? it - 3 * run : 0;
            const unsigned e = sorted[run];
            int base[3] = {o[0], o[1], o[2]};
            int slot;
            if (e & kRunOutside) {
                // a particle that drifted out of the window: a run of its own,
                // its base from the position this CTA has just stored
                slot = (int)(e & (kRunOutside - 1u));
                float x[D];
#pragma unroll
                for (int a = 0; a < D; ++a) x[a] = pb.s[(P::X + a) * pb.cap + ch.start + slot];
                Stencil<D> sn;
                unsigned err = 0;
                make_stencil<D>(x, sc, sn, err);
#pragma unroll
                for (int a = 0; a < D; ++a) base[a] = sn.base[a];
                if (ox == 0) mark_stencil<D>(base, sc, A.blk_flag, A.active, A.n_active);
            } else {
                slot = sm.head[b][e];
                const int l12 = (int)e / RS::B;
                base[0] += (int)e - RS::B * l12;
                base[1] += D == 3 ? l12 % RS::B : l12;
                if (D == 3) base[2] += l12 / RS::B;
            }
            PlaneSums acc;
            if constexpr (D == 3) sum_plane3(recs, slot, ox, acc);
            else sum_plane2(recs, slot, acc);
            auto value = [&](int n) { return make_float4(acc.xy[n].x, acc.xy[n].y, acc.z[n], acc.m[n]); };
            if constexpr (PAGED) {
                // a block the stencil covers has no page: the pool ran out or
                // the particle moved more than a cell since the last grid update
                if (ox == 0 && !stencil_paged<D>(sc, A.pages, base)) atomicOr(A.err_word, ERR_POOL);
                if (e & kRunOutside) {
#pragma unroll
                    for (int n = 0; n < 9; ++n)
                        atomicAdd(&A.grid_mom[grid_node<D, true>(sc, A.pages, base[0] + (D == 3 ? ox : n / 3),
                                                                 base[1] + (D == 3 ? n / 3 : n % 3),
                                                                 D == 3 ? base[2] + n % 3 : 0)],
                                  value(n));
                } else {
                    const PagedStencilIndex<D> ix(base, o);
                    const int x = ox == 0 ? ix.x[0] : ox == 1 ? ix.x[1] : ix.x[2];
#pragma unroll
                    for (int n = 0; n < 9; ++n) {
                        const int p = D == 3 ? x + ix.y[n / 3] + ix.z[n % 3] : ix.x[n / 3] + ix.y[n % 3];
                        atomicAdd(&A.grid_mom[(long long)sm.s27[b][p & 255] * 64 + (p >> 8)], value(n));
                    }
                }
            } else {
                const StencilIndex<D> ix(sc, base);
                float4* gm = A.grid_mom + sc.node_off;
                const int x = ox == 0 ? ix.x[0] : ox == 1 ? ix.x[1] : ix.x[2];
#pragma unroll
                for (int n = 0; n < 9; ++n)
                    atomicAdd(&gm[D == 3 ? x + ix.y[n / 3] + ix.z[n % 3] : ix(n / 3, n % 3, 0)], value(n));
            }
        }
        cur = next_chunk;
    }
    speed.flush(A.speed_max);
    pass_end(A);
}

template <int D, int MAT, int CHUNK, int MINB, bool FIXED, bool PAGED>
__global__ void __launch_bounds__(CHUNK, MINB) k_g2p2g_runs(ParticleBuf pb, const __grid_constant__ FusedArgs A) {
    // What the registers allow, by measurement (substep, us; rolled gather / y
    // loop unrolled / rolled with F loaded ahead of the gather).  128 registers:
    // jello 256^3 214 / 212 / 206, snow 256^3 231 / 222 / 226, water tank 67.8 /
    // 65.2 / -; scene table, 16 mixed scenes 255 / 242 / -.  96 registers: jello
    // 211 / 228 / 224, snow 227 / 239 / 243, water 64.5 / 71.5 / -; scene table
    // 241 / 233 / 244.
    constexpr bool ROOMY = MINB <= 4;
    constexpr bool PRELOAD = D == 3 && FIXED && ROOMY && MAT == JELLO;
    constexpr bool UNROLL_Y = !FIXED || (ROOMY && MAT != JELLO);
    __shared__ RunShared<D> sm;
    extern __shared__ __align__(16) float4 recs[];
    unsigned short* runs = reinterpret_cast<unsigned short*>(recs + A.chunk_cap * run_rec4(D));
    run_chunks<D, CHUNK, FIXED, PAGED>(pb, A, sm, recs, runs,
                                       [&](const Chunk& ch, const SceneParams& sc, const int* o, int b, int li, float* x,
                                           unsigned& speed_bits) {
        if (li >= ch.count) return;
        const long long i = (long long)ch.start + li;
        float* S = pb.s;
        const long long cap = pb.cap;
        unsigned err = 0;
        Stencil<D> st;
        if (make_stencil<D>(x, sc, st, err)) {
            float F[D * D], aux;
            if constexpr (PRELOAD) {
#pragma unroll
                for (int k = 0; k < D * D; ++k) F[k] = S[(Planes<D>::F + k) * cap + i];
            }
            G2PAcc<D> acc;
            g2p_window<D, PAGED, FIXED && !PAGED, UNROLL_Y>(st, o, sm.tv, sc, A, acc);
            // loaded after the gather, its register peak
            const GroupParams g = particle_group<FIXED>(A, pb, i);
            float Cn[D * D], v[D];
            typename SnowKeep<D>::T esvd;  // snow: what the plasticity step found, reused by the stress
            err |= update_and_store<D, MAT>(acc, sc, g, S, cap, i, x, v, Cn, F, aux, MAT == SNOW ? &esvd : nullptr,
                                            A.defer_vc != 0, PRELOAD);
            if (A.speed_max) speed_bits = max(speed_bits, __float_as_uint(signal_speed<D, MAT>(v, g, aux)));
            Stencil<D> sn;
            if (make_stencil<D>(x, sc, sn, err)) {
                P2GSource<D> src;
                if (MAT == SNOW) snow_stress_source(v, Cn, F, esvd, aux, g, sc.dt_next, src);
                else particle_stress_source<D, MAT, true>(v, Cn, F, aux, g, sc.dt_next, src);
                insert_record<D>(sm, recs, runs, b, li, sn, src, sc, o, A);
            }
        }
        if (err) atomicOr(A.err_word, err);
    });
}

}  // namespace mpm
