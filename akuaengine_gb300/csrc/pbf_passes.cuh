// The launches of a step's walk and pair kernels in one math mode; pbf_fast.cu and pbf_exact.cu
// instantiate them once each, pbf_shapes.cu the walk's other tile shapes.
#pragma once

#include "pbf_handle.cuh"

namespace akua::mlp {
int enqueue_forward(const akua_mlp* m, const float* feat, int n, float* out, float* out2,
                    float* out4, cudaStream_t st);
}

namespace akua {

// The walk at one tile shape (BLOCK threads, a pool of 32 x STAGE words per warp).  It starts when the
// table build has ended, so that its lookups too are read-only loads: 255 us at 1M particles against 260
// set up early and waiting; steps of 1,000 and 27,000 take the same either way.
template <bool EXACT, int BLOCK, int STAGE>
void launch_search_shape(akua_pbf* s, cudaStream_t st, int density, float* feat) {
    constexpr size_t smem = search_smem(BLOCK, STAGE);
    static_assert(smem <= 48 * 1024, "above the default limit of dynamic shared memory");
    const int per_warp = search_per_warp(s->n, s->sms, EXACT);
    auto go = [&](auto kernel) {
        radix::launch(false, kernel, grid_for(s->n, per_warp * (BLOCK / 32)), BLOCK, smem, st, 1,
                      s->d_params, s->ps0, s->table, s->r2i, s->nbr, s->cnt, s->rho, s->lam, s->flags,
                      density, s->speed, s->lprev, s->lacc, feat, s->psl, per_warp);
    };
    if (EXACT && per_warp <= kFewPerWarp) go(k_search<EXACT, BLOCK, STAGE, EXACT>);
    else go(k_search<EXACT, BLOCK, STAGE, false>);
}

// The default tile shape's kernels are in the math mode's own device image, the others' in that of
// pbf_shapes.cu.
template <bool EXACT>
void launch_search(akua_pbf* s, cudaStream_t st, int density, float* feat) {
    if (s->search_block == kSearchBlock && s->search_stage == kListStage)
        launch_search_shape<EXACT, kSearchBlock, kListStage>(s, st, density, feat);
    else
        launch_search_other(s, st, EXACT, density, feat);
}

template <bool EXACT, int LANES>
void enqueue_pairs(akua_pbf* s, cudaStream_t st, Marker& mark) {
    const int n = s->n;
    const int* pb = s->pair_block;  // per kernel: density, delta, last delta, vort., conf., XSPH
    auto gp = [&](int k) { return grid_for(n, pb[k] / LANES); };
    const int iters = s->cfg.solverIterations;
    float4* ps[2] = {s->ps0, s->ps1};
    const uint4* nbr4 = reinterpret_cast<const uint4*>(s->nbr);
    const int learn = learn_mode(s);
    launch_search<EXACT>(s, st, iters > 0 ? 1 : 0, learn ? s->feat : nullptr);
    mark("k_search");
    if (learn == 2) {
        mlp::enqueue_forward(s->warm, s->feat, n, s->lam, s->lacc, &s->psl->w, st);
        mark("k_mlp_forward");
    }
    for (int it = 0; it < iters; ++it) {
        float4* cur = ps[it & 1];
        float4* nxt = ps[(it + 1) & 1];
        if (it > 0) {
            step_kernel(s, st, k_density_lambda<EXACT, LANES>, gp(0), pb[0], 0,
                        s->d_params, cur, nbr4, s->cnt, s->rho, s->lam,
                        learn == 1 ? s->lacc : nullptr, s->psl);  // warm: the network's estimate is the sum
            mark("k_density_lambda");
        }
        if (it + 1 < iters) {
            step_kernel(s, st, k_delta_correct<EXACT, LANES>, gp(1), pb[1], 0,
                        s->d_params, cur, s->lam, nbr4, s->cnt, nxt, s->dp4, s->psl, s->mass_bits);
            mark("k_delta_correct");
        } else {
            step_kernel(s, st, k_delta_final<EXACT, LANES>, gp(2), pb[2], 0,
                        s->d_params, cur, s->lam, nbr4, s->cnt, s->x4g, s->x4, s->v4, s->vstar4, s->dp4,
                        s->origing, s->origin, s->rrefg, s->rref, s->rhog, s->lamg, s->dpg,
                        s->rho, nullptr, 1, s->psl, s->mass_bits, s->xv8);  // lam_out: zero iterations only
            mark("k_delta_final");
        }
    }
    if (iters == 0) {
        step_kernel(s, st, k_delta_final<EXACT, LANES>, gp(2), pb[2], 0,
                    s->d_params, s->ps0, nullptr, nbr4, s->cnt, s->x4g, s->x4, s->v4, s->vstar4, s->dp4,
                    s->origing, s->origin, s->rrefg, s->rref, s->rhog, s->lamg, s->dpg,
                    s->rho, s->lam, 0, s->psl, s->mass_bits, s->xv8);  // no delta: lambda is not read
        mark("k_delta_final");
    }
    // psl is free after the last delta: it carries (x, |omega|) to confinement
    step_kernel(s, st, k_vorticity<EXACT, LANES>, gp(3), pb[3], 0,
                s->d_params, s->x4, s->v4, s->xv8, nbr4, s->cnt, s->om4, s->psl);
    mark("k_vorticity");
    step_kernel(s, st, k_confine<EXACT, LANES>, gp(4), pb[4], 0,
                s->d_params, s->x4, s->v4, s->om4, s->rho, nbr4, s->cnt, s->xv8, s->psl, s->mass_bits);
    mark("k_confine");
    step_kernel(s, st, k_xsph<EXACT, LANES>, gp(5), pb[5], 0,
                s->d_params, s->xv8, nbr4, s->cnt, s->v4, s->kr, s->table);
    mark("k_xsph");
}

template <bool EXACT>
void enqueue_pairs(akua_pbf* s, cudaStream_t st, Marker& mark) {
    switch (pair_lanes(s->n, s->sms, EXACT)) {
        case 8: return enqueue_pairs<EXACT, 8>(s, st, mark);
        case 4: return enqueue_pairs<EXACT, 4>(s, st, mark);
        case 2: return enqueue_pairs<EXACT, 2>(s, st, mark);
        default: return enqueue_pairs<EXACT, 1>(s, st, mark);
    }
}

}  // namespace akua
