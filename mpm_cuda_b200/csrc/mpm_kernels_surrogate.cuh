// Fused substep with the learned stress (MPM_STRESS_SURROGATE), 3D jello.
// (Snow's exact stress comes almost free with its plasticity clamp, which leaves
// the distance of F from its rotation behind, so snow keeps the plain kernel.)  Same pass as
// k_g2p2g_runs (G2P, particle update, stress, run sums of the next P2G) with
// the stress of eligible particles taken from the BF16 MLP (mpm_mlp.cuh)
// instead of the polar iteration of kirchhoff_polar3 (MPMCUDA.cu:229-264
// decomposes F):
//   1. every thread: G2P, update, store the new state (v and C deferred as in
//      k_g2p2g), keep x, v, C, F in its record's slot and write its network
//      input (X = F F^T - I, J - 1) to its network row;
//   2. every warp: forward pass of its 32 rows on the tensor cores, in place;
//   3. every thread: stress from the prediction when F is inside the training
//      envelope and the error estimate is below tolerance, else from the polar
//      iteration; the P2G source replaces the stash in the record's slot.
// The stash keeps the network's registers from adding to the G2P registers
// without a round trip of the state through L2; a stash and a source record
// both take 24 floats, so they share the slot, and the network rows hold BF16
// pairs, so 4 CTAs of 128 threads with 256 particles fit an SM.  Launched with
// programmatic dependent launch like k_g2p2g; FIXED: the scene from the kernel
// parameters.
#pragma once

#include "mpm_kernels_runs.cuh"
#include "mpm_mlp.cuh"

namespace mpm {

// row stride (floats) of the per-particle network rows in shared memory: 16
// BF16 features, then 9 outputs; odd, so the rows of a warp's 32 particles
// start in 32 different banks
constexpr int kSurRowStride = 9;
// dynamic shared memory of k_g2p2g_sur: the chunk's records and run list, a
// network row per thread
constexpr int sur_dyn_smem(int cta, int particles) {
    return run_smem(3, particles) + cta * kSurRowStride * (int)sizeof(float);
}
// the most any configuration asks for
constexpr int sur_dyn_smem_max(int cta) {
    int most = 0;
    for (int i = 0; i < kNumFusedCfgs; ++i)
        most = kFusedCfgs[i].chunk * kFusedCfgs[i].rounds > most ? kFusedCfgs[i].chunk * kFusedCfgs[i].rounds : most;
    return sur_dyn_smem(cta, most);
}

struct SurArgs {
    const mlp::Forward* weights;
    mlp::Meta meta;
    unsigned long long* counts;  // [0] stresses from the network, [1] exact ones in their place
};

template <int CHUNK, int MINB, bool FIXED, bool PAGED>
__global__ void __launch_bounds__(CHUNK, MINB) k_g2p2g_sur(ParticleBuf pb, const __grid_constant__ FusedArgs A,
                                                            SurArgs SA) {
    constexpr int D = 3;
    constexpr int MAT = JELLO;
    static_assert(CHUNK % 32 == 0, "whole warps");
    static_assert(run_rec4(3) * 4 == 24, "x, v, C and F of a particle fill its record's slot");
    constexpr int XS = kSurRowStride;
    __shared__ RunShared<D> sm;
    __shared__ __align__(16) mlp::Forward W;  // network weights
    extern __shared__ __align__(16) float4 recs[];
    float* rows = reinterpret_cast<float*>(recs + A.chunk_cap * run_rec4(D));
    unsigned short* runs = reinterpret_cast<unsigned short*>(rows + CHUNK * XS);

    {
        // the weights do not depend on the launches ahead; published by run_chunks' first barrier
        const int4* src = reinterpret_cast<const int4*>(SA.weights);
        int4* dst = reinterpret_cast<int4*>(&W);
        for (int k = threadIdx.x; k < (int)(sizeof(mlp::Forward) / 16); k += CHUNK) dst[k] = src[k];
    }
    const int lane = threadIdx.x & 31, w0 = threadIdx.x & ~31;
    float* row = rows + threadIdx.x * XS;
    unsigned n_net = 0, n_svd = 0;
    // every thread runs every round (the network step is warp-synchronous)
    run_chunks<D, CHUNK, FIXED, PAGED>(pb, A, sm, recs, runs,
                                       [&](const Chunk& ch, const SceneParams& sc, const int* o, int b, int li, float* x,
                                           unsigned& speed_bits) {
        unsigned err = 0;
        bool next = false;      // the particle scatters into the next substep
        bool eligible = false;  // its group takes the network's stress
        int gi = 0;             // its group (re-read after the network: fewer live registers)
        float4* stash = recs + li * run_rec4(D);
        if (li < ch.count) {
            const long long i = (long long)ch.start + li;
            float* S = pb.s;
            const long long cap = pb.cap;
            gi = pb.grp[i];
            Stencil<D> st;
            if (make_stencil<D>(x, sc, st, err)) {
                G2PAcc<D> acc;
                g2p_window<D, PAGED, FIXED && !PAGED>(st, o, sm.tv, sc, A, acc);
                const GroupParams g = A.groups[gi];
                float F[D * D], Cn[D * D], v[D], aux;
                err |= update_and_store<D, MAT>(acc, sc, g, S, cap, i, x, v, Cn, F, aux, nullptr, A.defer_vc != 0);
                if (A.speed_max) speed_bits = max(speed_bits, __float_as_uint(signal_speed<D, MAT>(v, g, aux)));
                Stencil<D> sn;
                next = make_stencil<D>(x, sc, sn, err);
                if (next) {
                    stash[0] = make_float4(x[0], x[1], x[2], v[0]);
                    stash[1] = make_float4(v[1], v[2], Cn[0], Cn[1]);
                    stash[2] = make_float4(Cn[2], Cn[3], Cn[4], Cn[5]);
                    stash[3] = make_float4(Cn[6], Cn[7], Cn[8], F[0]);
                    stash[4] = make_float4(F[1], F[2], F[3], F[4]);
                    stash[5] = make_float4(F[5], F[6], F[7], F[8]);
                }
                eligible = next && g.surrogate != 0;
                if (eligible) {
                    float f[mlp::IN_PAD];
                    mlp::features(F, det<3>(F), SA.meta, f);
#pragma unroll
                    for (int k = 0; k < mlp::IN_PAD / 2; ++k)
                        row[k] = __uint_as_float(mlp::pack_bf16(f[2 * k], f[2 * k + 1]));
                }
            }
        }
        if (!eligible) {
#pragma unroll
            for (int k = 0; k < mlp::IN_PAD / 2; ++k) row[k] = 0.f;
        }
        __syncwarp();
        // ---- network: 32 rows per warp, two 16-row tiles, in place
        if (__any_sync(0xffffffffu, eligible)) {
            mlp::forward_tile<XS, true>(W, rows + w0 * XS, rows + w0 * XS, lane);
            mlp::forward_tile<XS, true>(W, rows + (w0 + 16) * XS, rows + (w0 + 16) * XS, lane);
        }
        __syncwarp();
        if (next) {
            const float4 q0 = stash[0], q1 = stash[1], q2 = stash[2], q3 = stash[3], q4 = stash[4], q5 = stash[5];
            const float xn[D] = {q0.x, q0.y, q0.z};
            float v[D] = {q0.w, q1.x, q1.y};
            float Cn[9] = {q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, q3.x, q3.y, q3.z};
            float F[9] = {q3.w, q4.x, q4.y, q4.z, q4.w, q5.x, q5.y, q5.z, q5.w};
            const GroupParams g = A.groups[gi];
            Stencil<D> sn;
            make_stencil<D>(xn, sc, sn, err);  // the stencil found above
            float tau[D * D];
            bool use = false;
            if (eligible) {
                const float J = det<3>(F);
                use = mlp::in_envelope(F, J, SA.meta) && mlp::tau_from_prediction(row, F, J, g.mu, g.lambda, SA.meta, tau);
            }
            P2GSource<D> src;
            if (use) {
                source_from_tau<D>(v, Cn, tau, g, sc.dt_next, src);
                ++n_net;
            } else {
                particle_stress_source<D, MAT, true>(v, Cn, F, 1.f, g, sc.dt_next, src);
                ++n_svd;
            }
            insert_record<D>(sm, recs, runs, b, li, sn, src, sc, o, A);
        }
        if (err) atomicOr(A.err_word, err);
        __syncwarp();  // the rows are rewritten by the next round
    });
    n_net = __reduce_add_sync(0xffffffffu, n_net);
    n_svd = __reduce_add_sync(0xffffffffu, n_svd);
    if (lane == 0 && (n_net | n_svd)) {
        atomicAdd(&SA.counts[0], (unsigned long long)n_net);
        atomicAdd(&SA.counts[1], (unsigned long long)n_svd);
    }
}

}  // namespace mpm
