// The solver's handle and what the translation units that enqueue a step's kernels share: pbf_solver.cu
// (memory, sorts, graph, C ABI), pbf_fast.cu and pbf_exact.cu (the walk and the pair kernels of one
// math mode each), pbf_shapes.cu (the walk's other tile shapes).
#pragma once

#include <cstdint>
#include <vector>

#include "akua_pbf.h"
#include "mlp_handle.h"
#include "pbf_pairs.cuh"
#include "pbf_search.cuh"
#include "radix_sort.cuh"

struct akua_pbf {
    int device = 0;
    int sms = 1;  // multiprocessors of the device
    bool cluster_sort = false;  // a sort pass is one cluster
    int n = 0;
    akua_pbf_config cfg{};
    akua_lambda_corr_params corr{};
    uint32_t table_size = 0;
    uint32_t table_alloc = 0;
    float restitution = 0.0f;
    float friction = 0.95f;
    uint32_t options = 0;
    cudaStream_t stream = nullptr;          // caller's stream (nullptr = legacy default stream)
    cudaStream_t capture_stream = nullptr;  // private stream used only for graph capture
    char* attached = nullptr;
    size_t stride = 0;
    bool state_valid = false;  // device state holds the particles (resident mode)
    bool stepped = false;      // the reference-order tables describe the current state

    akua::StepParams* d_params = nullptr;
    // state, internal order
    float4 *x4 = nullptr, *v4 = nullptr, *col4 = nullptr;
    float* size = nullptr;
    uint32_t* rref = nullptr;
    float *rho = nullptr, *lam = nullptr;
    float4* dp4 = nullptr;
    // gathered copies and per-step arrays
    float4 *x4g = nullptr, *ps0 = nullptr, *ps1 = nullptr;
    uint32_t *origin = nullptr, *origing = nullptr;  // a slot's colour and size: their import index
    float4 *vstar4 = nullptr, *om4 = nullptr, *xv8 = nullptr, *dpg = nullptr;
    float *rhog = nullptr, *lamg = nullptr;
    uint32_t *rrefg = nullptr, *rank_of_import = nullptr, *r2i = nullptr, *order = nullptr;
    // sorts: reference order (A) and Morton order (B)
    uint32_t *ka0 = nullptr, *va0 = nullptr, *ka1 = nullptr, *va1 = nullptr;
    uint32_t *kb0 = nullptr, *vb0 = nullptr, *kb1 = nullptr, *vb1 = nullptr;
    uint32_t* sort_scratch = nullptr;
    uint32_t* sort_scratch_b = nullptr;  // the Morton sort's, which runs beside the hash sort
    cudaStream_t side_stream = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    uint2* table = nullptr;
    uint32_t *nbr = nullptr, *cnt = nullptr, *flags = nullptr;
    float4* psl = nullptr;          // (x*, lambda) of the current iteration, for uniform masses
    akua::SdfShape* shapes = nullptr;  // SDF obstacles (device), AKUA_SDF_MAX_SHAPES
    int num_shapes = 0;
    float sdf_min_dist = 0.025f, sdf_stiffness = 0.5f;
    uint32_t* mass_bits = nullptr;  // {another mass seen, record 0's mass bits} of this step
    char* staging = nullptr;
    size_t staging_bytes = 0;

    akua::radix::Plan plan_ref, plan_sp;
    int sp_bits = 0;
    uint32_t *kr = nullptr, *refperm = nullptr, *spperm = nullptr;  // sort results (set at enqueue)

    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    bool graph_ok = false;
    uint32_t graph_options = 0;
    const char* graph_aos = nullptr;
    size_t graph_stride = 0;
    int graph_sp_bits = -1;
    int graph_captures = 0;
    int body_launches = 0;
    bool chain = false;  // the body's kernels are set up while the previous one ends

    // learned warm start (allocated on first use): features, predicted velocity (.w = density),
    // the step's accumulated lambda, the previous step's (internal order) and the export copy
    // (reference order, read back at import)
    akua_mlp* warm = nullptr;
    bool track = false;  // accumulate lambda and compute features every step
    float* cap_feat = nullptr;
    float* cap_target = nullptr;
    float *feat = nullptr, *lacc = nullptr, *lprev = nullptr, *lacc_ref = nullptr;
    float* speed = nullptr;
    uint32_t* err_max = nullptr;
    double* err_sum = nullptr;
    int graph_learn = 0;

    // batches of independent scenes (akua_pbf_create_batch); empty for a single scene
    std::vector<akua_scene_desc> scenes;
    std::vector<uint32_t> scene_first;  // first particle of each scene
    uint16_t* scene_of = nullptr;       // device: the scene of every particle
    int scene_bits = 0;                 // bits of the scene index in the Morton sort key

    // block sizes of the neighbour-pair kernels (akua_pbf_set_pair_blocks / akua_pbf_autotune)
    int pair_block[AKUA_PBF_PAIR_KERNELS] = {128, 128, 128, 128, 128, 128};
    // the walk's tile shape (akua_pbf_set_search_shape / akua_pbf_autotune)
    int search_block = akua::kSearchBlock;
    int search_stage = akua::kListStage;

    int64_t steps = 0;
    uint64_t device_bytes = 0;

    // profiling (akua_pbf_profile_begin/end): one event after every kernel of a step
    bool prof_active = false;
    int prof_steps_left = 0;
    std::vector<cudaEvent_t> prof_events;
    std::vector<const char*> prof_names;  // nullptr marks the start of a step
    size_t prof_next = 0;
};

namespace akua {

inline int grid_for(int n, int block) { return (n + block - 1) / block; }

// 0: plain step; 1: features and accumulated lambda are tracked (training capture); 2: and the
// network's prediction replaces iteration 1's lambda.
inline int learn_mode(const akua_pbf* s) { return s->warm ? 2 : ((s->track || s->cap_feat) ? 1 : 0); }

// Counts launches and, while profiling (never during capture), records an event after each.
struct Marker {
    akua_pbf* s;
    cudaStream_t st;
    bool record;
    int launches = 0;
    void operator()(const char* name) {
        ++launches;
        if (record && s->prof_next < s->prof_events.size()) {
            cudaEventRecord(s->prof_events[s->prof_next], st);
            s->prof_names[s->prof_next] = name;
            ++s->prof_next;
        }
    }
};

// A kernel of the body's chain.
template <class... Params, class... Args>
inline void step_kernel(const akua_pbf* s, cudaStream_t st, void (*kernel)(Params...), int grid,
                        int block, size_t smem, Args... args) {
    radix::launch(s->chain, kernel, grid, block, smem, st, 1, args...);
}

// The walk and the pair kernels of a step (pbf_passes.cuh).  A process loads the device image of a
// translation unit when it first uses a kernel of it, so a math mode's kernels have one of their own,
// and the walk's tile shapes other than the default another (a process's creation and first step of 1,000
// particles: 3.1 ms with all of them in one image, 2.4 by math mode, 2.3 like this).
void enqueue_pairs_fast(akua_pbf* s, cudaStream_t st, Marker& mark);
void enqueue_pairs_exact(akua_pbf* s, cudaStream_t st, Marker& mark);
void launch_search_other(akua_pbf* s, cudaStream_t st, bool exact, int density, float* feat);

}  // namespace akua
